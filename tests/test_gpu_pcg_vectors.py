"""The PCG's vector kernels at the edges of their row blocks and batches.

A row block has up to 4,096 rows, a thread takes every 256th of them, four at a time; columns
of up to eight row blocks (32,768 rows) take one launch per iteration.  The
solves are compared with a numpy PCG over the same products; MIXED products differ by their
quantisation (about 1e-7 of the largest entry) when the search directions differ by rounding,
far below the solves' tolerance of 1e-5."""
import numpy as np
import pytest

import csaige_b200 as cs

pytestmark = pytest.mark.gpu


def _grm(n, m=200):
    bed = cs.gen_bed(cs.CohortSpec(n=n, m=m, seed=n, missing_rate=0.02))
    af, mac, nv = cs.bed_marker_stats(bed, n, m)
    keep = np.nonzero((af >= 0.01) & (af <= 0.99))[0]
    return cs.OnTheFlyGrm.from_bed(bed, n, m, keep, af[keep], precision=cs.PREC_MIXED)


def _pcg(grm, w, tau, b, x0, tol):
    d = tau[0] / w + tau[1]
    sigma = lambda v: tau[0] * v / w + tau[1] * grm.mat_vec(v)
    x = np.zeros_like(b) if x0 is None else x0.copy()
    r = b if x0 is None else b - sigma(x)
    z = r / d
    p, rz = z, r @ z
    for it in range(1, 500):
        ap = sigma(p)
        alpha = rz / (p @ ap)
        x, r = x + alpha * p, r - alpha * ap
        if np.sqrt(r @ r) < tol * max(np.sqrt(b @ b), 1.0):
            return x, it
        z = r / d
        rz, old = r @ z, rz
        p = z + (rz / old) * p
    raise AssertionError("no convergence")


@pytest.mark.parametrize("n", [33, 255, 257, 1023, 1025, 4096, 4097, 9001, 13000, 16385, 32768, 32769])
@pytest.mark.parametrize("warm", [False, True])
def test_pcg_over_row_blocks(n, warm):
    grm = _grm(n)
    rng = np.random.default_rng(n)
    w = rng.uniform(0.05, 0.25, n)
    tau = [1.0, 0.4]
    b = rng.standard_normal((5, n)) * np.array([1.0, 10.0, 0.1, 3.0, 1.0])[:, None]
    x0 = rng.standard_normal((5, n)) * 0.01 if warm else None
    res = cs.PcgSolver(1e-5, 500).solve(grm, w, tau, b, x0=x0, precision=cs.PREC_MIXED)
    for c in range(5):
        x, it = _pcg(grm, w, tau, b[c], None if x0 is None else x0[c], 1e-5)
        assert res[c].converged and abs(res[c].iterations - it) <= 1
        ax = tau[0] * res[c].x / w + tau[1] * grm.mat_vec(res[c].x)
        assert np.linalg.norm(b[c] - ax) <= 2e-5 * max(np.linalg.norm(b[c]), 1.0)


def test_columns_stop_converge_and_run_out_side_by_side():
    n = 5000
    grm = _grm(n)
    rng = np.random.default_rng(1)
    w = rng.uniform(0.05, 0.25, n)
    b = rng.standard_normal((4, n))
    b[1] = 0.0     # p'Ap below 1e-30: stops in its first step, with x as it was
    b[2] *= 1e-20  # the same, from a right-hand side that is not zero
    res = cs.PcgSolver(0.0, 3).solve(grm, w, [1.0, 0.4], b, precision=cs.PREC_MIXED)
    assert [r.iterations for r in (res[0], res[2], res[3])] == [3, 0, 3]
    assert not any(r.converged for r in (res[0], res[2], res[3]))
    assert not res[1].x.any() and not res[2].x.any()
    one = cs.PcgSolver(0.0, 3).solve(grm, w, [1.0, 0.4], b[3:], precision=cs.PREC_MIXED)
    assert np.allclose(res[3].x, one[0].x, rtol=1e-6, atol=1e-9)
