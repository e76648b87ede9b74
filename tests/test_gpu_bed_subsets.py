"""Sample subsets of a .bed: counts against a mask, rows of ascending subsets by compression.

Counts are integers, and products of the packed rows are compared to the bit with the CPU model
on the subset's codes."""
import numpy as np
import pytest
import torch

import csaige_b200 as cs
import mixed_model as MM
import oracle_ffi as O

pytestmark = pytest.mark.gpu


def _on_device(bed, shift):
    buf = torch.zeros(bed.size + shift + 16, dtype=torch.uint8, device="cuda")
    buf[shift:shift + bed.size] = torch.from_numpy(bed)
    torch.cuda.synchronize()
    return buf, buf.data_ptr() + shift


def _subsets(n_fam, rng):
    perm = rng.permutation(n_fam)
    some = np.sort(perm[: max(1, int(0.4 * n_fam))])
    yield "ascending", some
    yield "few", np.sort(perm[: max(1, n_fam // 100)])   # below the compression's line
    yield "nearly all", np.sort(perm[: max(1, n_fam - 1)])
    yield "one swapped", np.concatenate([some[1:2], some[:1], some[2:]])
    yield "one twice", np.sort(np.concatenate([some, some[-1:]]))
    yield "tail", np.arange(n_fam // 2, n_fam)


# rows of every length modulo 4 and words of 16 samples cut anywhere; 830,003: rows that are
# not staged; with 2,400 markers a warp per row
@pytest.mark.parametrize("n_fam,m", [(19, 40), (64, 40), (1001, 33), (4097, 70), (20003, 9),
                                     (150001, 5), (830003, 2), (9001, 2400)])
def test_counts_and_rows_of_subsets(n_fam, m):
    rng = np.random.default_rng(n_fam)
    spec = cs.CohortSpec(n=n_fam, m=m, seed=n_fam, missing_rate=0.03, maf_lo=0.1)
    bed = cs.gen_bed(spec)
    for k, (name, sidx) in enumerate(_subsets(n_fam, rng)):
        buf, ptr = _on_device(bed, k % 4)
        n = sidx.size
        want = O.marker_stats(bed, n_fam, m, sidx)
        af, mac, nv = cs.api.bed_marker_stats_dev(ptr, bed.size, n_fam, m, sidx)
        for a, b in zip((af, mac, nv), want):
            assert np.array_equal(a, b), name
        keep = np.nonzero((af > 0.0) & (af < 1.0))[0][:60]
        if keep.size == 0 or m > 100:
            continue
        grm = cs.OnTheFlyGrm.from_bed_dev(ptr, bed.size, n_fam, m, keep, af[keep],
                                          sample_idx=sidx, precision=cs.PREC_MIXED)
        v = rng.standard_normal(n)
        want = MM.kv(MM.codes(bed, n_fam, keep, sidx), af[keep], v[:, None])[:, 0]
        assert np.array_equal(grm.mat_vec(v), want), name
        grm.close()
