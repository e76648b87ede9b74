"""The page-locked blocks of closed handles: kept for the next handles, as many as were in use
at once (a block handed back to the driver waits for the device, and so for other fits)."""
import ctypes as C
import os

import numpy as np
import pytest

import csaige_b200 as cs
from csaige_b200._lib import LIB, check


def _blocks():
    kept, most = C.c_int32(), C.c_int32()
    check(LIB.saige_pinned_blocks(C.byref(kept), C.byref(most)))
    return kept.value, most.value


def test_a_block_for_every_concurrent_fit():
    # the sub-cohort call runs a fit on every second hardware thread
    assert _blocks()[1] >= max(2, len(os.sched_getaffinity(0)) // 2)


@pytest.mark.gpu
def test_blocks_of_closed_handles_are_kept():
    check(LIB.saige_release_cached_memory())
    assert _blocks()[0] == 0
    n, m = 300, 200
    bed = cs.gen_bed(cs.CohortSpec(n=n, m=m, seed=2))
    af, _, _ = cs.bed_marker_stats(bed, n, m)
    keep = np.nonzero((af >= 0.05) & (af <= 0.95))[0]
    v = np.random.default_rng(1).standard_normal(n)
    for handles in (24, 7):
        grms = [cs.OnTheFlyGrm.from_bed(bed, n, m, keep, af[keep], precision=cs.PREC_MIXED)
                for _ in range(handles)]
        first = [g.mat_vec(v) for g in grms]
        assert all(np.array_equal(first[0], k) for k in first)
        assert _blocks()[0] == 24 - handles
        for g in grms:
            g.close()
        assert _blocks()[0] == 24
    check(LIB.saige_release_cached_memory())
    assert _blocks()[0] == 0
