"""The P-projection's coefficients: on the device up to 16 covariates, on the host beyond.

Fits are compared with the oracle's at the tolerance of the other fits' comparisons."""
import numpy as np
import pytest

import csaige_b200 as cs
import oracle_ffi as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("p", [1, 2, 15, 16, 17, 24])
def test_fits_with_many_covariates_match_the_oracle(p):
    n, m, trait = 800, 600, O.QUANTITATIVE
    spec = cs.CohortSpec(n=n, m=m, seed=21, missing_rate=0.01, trait=trait, n_covar=2, h2=0.4)
    bed = cs.gen_bed(spec)
    y, _ = cs.gen_pheno(spec)
    rng = np.random.default_rng(p)
    x = np.vstack([np.ones(n), rng.standard_normal((p - 1, n))]).T
    af, mac, nv = O.marker_stats(bed, n, m)
    g, _ = O.select_markers(af, mac, nv, n)
    grm = cs.OnTheFlyGrm.from_bed(bed, n, m, g, af[g])
    r = cs.fit_ai_reml(y, x, grm, cs.TraitType(trait), cs.AiRemlConfig(max_iter=6, tol=1e-5))
    k = O.grm_explicit(O.standardize(O.dosages(bed, n, g), af[g], 0))
    o = O.fit_ai_reml(y, x, trait, O.K_EXPLICIT, k, max_iter=6, tol=1e-5)
    assert r.iterations == o["iterations"]
    assert np.all(np.abs(r.tau - o["tau"]) <= 1e-4 * np.abs(o["tau"]))
    assert np.abs(r.alpha - o["alpha"]).max() <= 1e-4 * np.abs(o["alpha"]).max()
