"""Errors of products whose error word is read later: inside a solve the word arrives with
the columns' state, one wait per iteration."""
import numpy as np
import pytest

import csaige_b200 as cs
from csaige_b200 import _lib

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("q", [3, 40])
@pytest.mark.parametrize("warm", [False, True])
def test_timed_out_product_inside_a_solve(q, warm):
    n, m = 4096, 2048
    bed = cs.gen_bed(cs.CohortSpec(n=n, m=m, seed=17, missing_rate=0.02))
    af, mac, nv = cs.bed_marker_stats(bed, n, m)
    keep = np.nonzero((af >= 0.01) & (af <= 0.99))[0]
    grm = cs.OnTheFlyGrm.from_bed(bed, n, m, keep, af[keep], precision=cs.PREC_MIXED)
    rng = np.random.default_rng(5)
    w, b = rng.uniform(0.05, 0.25, n), rng.standard_normal((q, n))
    x0 = 0.01 * b if warm else None
    solve = lambda: cs.PcgSolver(1e-6, 100).solve(grm, w, [1.0, 0.4], b, x0=x0,
                                                  precision=cs.PREC_MIXED)
    want = solve()
    try:
        _lib.LIB.saige_tc_set_wait_budget(0)
        with pytest.raises(cs.SaigeError) as e:
            solve()
        assert e.value.code == _lib.TIMEOUT
    finally:
        _lib.LIB.saige_tc_set_wait_budget(-1)
    for a, b_ in zip(want, solve()):
        assert a.iterations == b_.iterations and np.array_equal(a.x, b_.x)
