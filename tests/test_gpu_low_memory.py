"""Calls with little device memory left: workspaces that only make a call faster are done
without, and the results are the same bits.

Each case runs once with memory to spare (which also loads the kernels), then on a new handle
with all but `leave` bytes taken: more than what the call cannot do without, and less than that
and the workspace in question together."""
import numpy as np
import pytest

import csaige_b200 as cs
from csaige_b200._lib import LIB, check

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")

MB = 1 << 20


def _grm(n, m, precision):
    """A handle, with no blocks left over from building it."""
    spec = cs.CohortSpec(n=n, m=m, seed=n, missing_rate=0.01)
    bed = cs.gen_bed(spec)
    af, _, _ = cs.bed_marker_stats(bed, n, m)
    keep = np.nonzero((af >= 0.02) & (af <= 0.98))[0]
    return cs.OnTheFlyGrm.from_bed(bed, n, m, keep, af[keep], precision=precision)


class _Taken:
    """All device memory but `leave` bytes."""

    def __init__(self, leave):
        torch.cuda.empty_cache()
        check(LIB.saige_release_cached_memory())
        free, _ = torch.cuda.mem_get_info()
        self.block = torch.empty(free - leave, dtype=torch.uint8, device="cuda")

    def __enter__(self):
        return self

    def __exit__(self, *_):
        self.block = None
        torch.cuda.empty_cache()


def _same_when_short(make, call, leave):
    ready = make()
    want = call(ready)
    ready.close()
    short = make()
    with _Taken(leave):
        got = call(short)
    short.close()
    assert np.array_equal(got, want)


def test_mixed_block_without_room_for_shared_tiles():
    # 64 columns: 21 MB of vectors and 9 MB of operands; the shared tiles' sums take 19 MB
    n, m = 20000, 5000
    v = np.random.default_rng(1).standard_normal((64, n))

    def make():
        g = _grm(n, m, cs.PREC_MIXED)
        g.mat_vec(v[0])  # the tiles
        return g

    _same_when_short(make, lambda g: g.mat_vec(v), 44 * MB)


def test_mixed_column_without_room_for_divided_passes():
    # the divided passes' sums take 6.4 MB; the rest is there since the two-column product
    n, m = 400000, 600
    v = np.random.default_rng(2).standard_normal((2, n))

    def make():
        g = _grm(n, m, cs.PREC_MIXED)
        g.mat_vec(v)
        return g

    _same_when_short(make, lambda g: g.mat_vec(v[0]), 4 * MB)


def test_fp32_columns_without_room_for_a_shared_decode():
    # 13 MB of vectors; scratch of 7 MB for a column, 31 MB for eight
    n, m = 100000, 2000
    v = np.random.default_rng(3).standard_normal((8, n))
    _same_when_short(lambda: _grm(n, m, cs.PREC_FP32), lambda g: g.mat_vec(v), 30 * MB)


def test_diagonal_without_room_for_all_ranges():
    # 23 MB for the sums of all 47 ranges of markers
    n, m = 60000, 6000
    _same_when_short(lambda: _grm(n, m, cs.PREC_FP32), lambda g: g.diag(), 8 * MB)


def test_explicit_grm_without_room_for_shared_tiles():
    # 528 tiles on 148 SMs: two launches, between which 148 tiles' sums take 19 MB
    n, m = 4001, 600
    bed = cs.gen_bed(cs.CohortSpec(n=n, m=m, seed=4, missing_rate=0.01))
    want, used = cs.compute_sparse_grm(bed, n, m)
    with _Taken(12 * MB):
        got, used_short = cs.compute_sparse_grm(bed, n, m)
    assert used_short == used
    for a, b in ((got.rows, want.rows), (got.cols, want.cols), (got.vals, want.vals)):
        assert np.array_equal(a, b)
