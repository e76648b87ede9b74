"""The Galerkin start's Gram products at the edges of their tiles and row chunks.

A start only changes where the PCG begins; wrong sums would give a poor start or none at
all.  So with every basis width the recycled fit must keep the zero-start fit's tau (both
solve to the PCG tolerance) and need fewer PCG iterations."""
import numpy as np
import pytest

import csaige_b200 as cs

pytestmark = pytest.mark.gpu


# rows: one partial stage, a ragged last pair of rows, several chunks; columns: bases that
# end inside and at the edge of the 16- and 32-column tiles
@pytest.mark.parametrize("n,covar,probes", [(1003, 1, 6), (2049, 2, 13), (4095, 4, 27),
                                            (6150, 8, 30), (9001, 15, 32)])
def test_recycled_start_keeps_tau_and_saves_iterations(n, covar, probes):
    spec = cs.CohortSpec(n=n, m=3000, seed=n, trait=int(cs.TraitType.Quantitative), h2=0.3,
                         n_covar=covar)
    bed = cs.gen_bed(spec)
    y, x = cs.gen_pheno(spec)
    af, mac, nv = cs.bed_marker_stats(bed, n, spec.m)
    g, _ = cs.select_grm_markers(af, mac, nv, n)
    grm = cs.OnTheFlyGrm.from_bed(bed, n, spec.m, g, af[g], precision=cs.PREC_MIXED)
    fits = [cs.fit_ai_reml(y, x, grm, cs.TraitType.Quantitative,
                           cs.AiRemlConfig(tol=1e-5, precision=cs.PREC_MIXED, solve=cs.SOLVE_BLOCK,
                                           n_random_vectors=probes, warm_start=w))
            for w in (cs.WARM_ZERO, cs.WARM_RECYCLED)]
    zero, rec = fits
    assert np.all(np.abs(rec.tau - zero.tau) <= 1e-4 * np.abs(zero.tau))
    assert rec.pcg_iters < zero.pcg_iters
