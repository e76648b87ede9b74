"""Row kernels of the .bed path at the sizes where their forms change.

Counts are integers and the GRM diagonal is compared in FP64: against the oracle's
statistics and a NumPy restatement."""
import numpy as np
import pytest
import torch

import csaige_b200 as cs
import mixed_model as MM
import oracle_ffi as O

pytestmark = pytest.mark.gpu


def _bed(n, m, seed):
    bpm = (n + 3) // 4
    bed = np.random.default_rng(seed).integers(0, 256, 3 + m * bpm, dtype=np.uint8)
    bed[:3] = (0x6C, 0x1B, 0x01)
    return bed


def _stats_at(bed, shift, n, m, sidx):
    """Statistics with the .bed `shift` bytes into a device allocation."""
    buf = torch.zeros(bed.size + shift, dtype=torch.uint8, device="cuda")
    buf[shift:] = torch.from_numpy(bed)
    torch.cuda.synchronize()
    return cs.api.bed_marker_stats_dev(buf.data_ptr() + shift, bed.size, n, m, sidx)


# a warp per row up to 2,048 bytes, the block beyond; rows of every length modulo 4, which
# with the shifts puts their starts and ends at every alignment
@pytest.mark.parametrize("n", [1, 15, 17, 33, 4093, 8190, 8192, 8197, 30011])
@pytest.mark.parametrize("m", [1, 9, 35])
def test_counts_of_all_samples(n, m):
    bed = _bed(n, m, n + m)
    want = O.marker_stats(bed, n, m, None)
    for shift in range(4):
        got = _stats_at(bed, shift, n, m, None)
        assert all(np.array_equal(a, b) for a, b in zip(got, want)), shift


@pytest.mark.parametrize("n", [8197, 70001])
def test_counts_of_many_long_rows(n):
    # enough rows for a warp each (2,368 and more) although they are long
    bed = _bed(n, 2370, n)
    want = O.marker_stats(bed, n, 2370, None)
    got = _stats_at(bed, 1, n, 2370, None)
    assert all(np.array_equal(a, b) for a, b in zip(got, want))


# rows staged per block: 4 (short rows), 3, 2, 1 (half and whole SM), 0 (read in place)
@pytest.mark.parametrize("n_fam", [50, 20003, 120001, 150001, 200003, 300001, 500003, 830003])
@pytest.mark.parametrize("m", [1, 6])
def test_counts_of_a_subset(n_fam, m):
    rng = np.random.default_rng(n_fam)
    bed = _bed(n_fam, m, n_fam + m)
    for sidx in (rng.permutation(n_fam)[: n_fam // 3 + 1], np.arange(n_fam)[::2].copy()):
        want = O.marker_stats(bed, n_fam, m, sidx)
        got = _stats_at(bed, n_fam % 4, n_fam, m, sidx)
        assert all(np.array_equal(a, b) for a, b in zip(got, want))


@pytest.mark.parametrize("n,m", [(1, 1), (500, 64), (4096, 65), (4100, 700), (70001, 130)])
def test_diagonal(n, m):
    # the sums are FP64 in another order than NumPy's: m terms of about 1
    spec = cs.CohortSpec(n=n, m=m, seed=n + m, missing_rate=0.03)
    bed = cs.gen_bed(spec)
    af, _, _ = O.marker_stats(bed, n, m, None)
    keep = np.nonzero((af > 0.0) & (af < 1.0))[0]
    if keep.size == 0:
        pytest.skip("no polymorphic marker")
    grm = cs.OnTheFlyGrm.from_bed(bed, n, m, keep, af[keep])
    codes, p = MM.codes(bed, n, keep), af[keep][:, None]
    dose = np.choose(codes, [2.0, np.nan, 1.0, 0.0])
    z = np.nan_to_num((dose - 2 * p) / np.sqrt(2 * p * (1 - p)))
    want = (z * z).sum(0) / keep.size
    np.testing.assert_allclose(grm.diag(), want, rtol=1e-15 * (m + 8), atol=0)
