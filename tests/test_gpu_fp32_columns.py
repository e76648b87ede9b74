"""FP32 products of several columns: each column's f32 operations and their order are those
of a product of its own, so a block equals its columns' products bit for bit; and the
product is the FP64 oracle's within the f32 rounding of its sums."""
import numpy as np
import pytest

import csaige_b200 as cs
import oracle_ffi as O

pytestmark = pytest.mark.gpu


# samples: one word, a ragged word, below and above a pass-B window; markers: below, at and
# above a pass-A group, a table chunk and a split
@pytest.mark.parametrize("n,m", [(3, 5), (511, 127), (513, 129), (2000, 5000), (4100, 640),
                                 (70001, 300), (20011, 3001)])
def test_block_equals_single_columns(n, m):
    spec = cs.CohortSpec(n=n, m=m, seed=n + m, missing_rate=0.02)
    bed = cs.gen_bed(spec)
    af, _, _ = O.marker_stats(bed, n, m)
    keep = np.nonzero((af > 0.0) & (af < 1.0))[0]
    grm = cs.OnTheFlyGrm.from_bed(bed, n, m, keep, af[keep], precision=cs.PREC_FP32)
    v = np.random.default_rng(n).standard_normal((11, n))
    v[2] *= 1e-30
    one = np.stack([grm.mat_vec(x) for x in v])
    for q in (2, 3, 4, 5, 6, 7, 8, 11):
        assert np.array_equal(grm.mat_vec(v[:q]), one[:q]), q
    if n * m < 12_000_000:
        z = O.standardize(O.dosages(bed, n, keep), af[keep], 0)
        for c in (0, 2, 6):
            want = O.grm_matvec(z, v[c], 0)
            # two f32 passes of up to m and n terms: 24-bit rounding, error growing like the
            # square root of the length of a chain
            assert np.abs(one[c] - want).max() < 2e-5 * np.abs(want).max()


@pytest.mark.parametrize("warm", [cs.WARM_ZERO, cs.WARM_PREVIOUS])
@pytest.mark.parametrize("precision", [cs.PREC_FP32, cs.PREC_MIXED])
def test_single_solves_run_side_by_side_with_the_same_bits(precision, warm):
    # SOLVE_SINGLE runs its right-hand sides as the columns of block solves: each column is
    # a PCG of its own, as PcgSolver solves them one by one
    n, m = 1200, 900
    spec = cs.CohortSpec(n=n, m=m, seed=5)
    bed = cs.gen_bed(spec)
    y, x = cs.gen_pheno(spec)
    af, mac, nv = cs.bed_marker_stats(bed, n, m)
    g, _ = cs.select_grm_markers(af, mac, nv, n)
    grm = cs.OnTheFlyGrm.from_bed(bed, n, m, g, af[g], precision=precision)
    b = np.random.default_rng(1).standard_normal((5, n))
    w, tau = np.full(n, 0.2), np.array([1.0, 0.4])
    solver = cs.PcgSolver()
    block = solver.solve(grm, w, tau, b)
    for c in range(5):
        one = solver.solve(grm, w, tau, b[c])
        assert np.array_equal(one.x, block[c].x) and one.iterations == block[c].iterations
    # and the fit agrees with the block strategy's to the bit, with its own launch count
    fits = [cs.fit_ai_reml(y, x, grm, cs.TraitType.Binary,
                           cs.AiRemlConfig(precision=precision, solve=s, warm_start=warm))
            for s in (cs.SOLVE_SINGLE, cs.SOLVE_BLOCK)]
    assert np.array_equal(fits[0].tau, fits[1].tau) and np.array_equal(fits[0].mu, fits[1].mu)
    assert fits[0].n_kv == fits[1].n_kv and fits[0].pcg_iters == fits[1].pcg_iters
    assert fits[0].n_kv_launches > fits[1].n_kv_launches
