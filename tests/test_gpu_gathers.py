"""Gathers that replaced copies: the variance-ratio candidates' packed rows."""
import numpy as np
import pytest

import csaige_b200 as cs
import oracle_ffi as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1021, 2047, 8193])  # rows of 256, 512 and 2,049 bytes
def test_variance_ratio_rows_of_any_length(n):
    m = 1200
    spec = cs.CohortSpec(n=n, m=m, seed=n, missing_rate=0.01, prevalence=0.2, h2=0.3, n_covar=2)
    bed = cs.gen_bed(spec)
    y, x = cs.gen_pheno(spec)
    cfg = cs.AiRemlConfig(max_iter=3)
    fr = cs.fit_null_from_bed(bed, n, m, y, x, cs.TraitType.Binary, cfg, variance_ratio=True)
    af, mac, nv = cs.bed_marker_stats(bed, n, m)
    gidx, vidx = cs.select_grm_markers(af, mac, nv, n, 0.01, 0.15, 12345)
    grm = cs.OnTheFlyGrm.from_bed(bed, n, m, gidx, af[gidx])
    fit = cs.fit_ai_reml(y, x, grm, cs.TraitType.Binary, cfg)
    vr = cs.estimate_variance_ratio(grm, O.dosages(bed, n, vidx), mac[vidx], fit.mu,
                                    fit.working_weights, fit.tau, cs.TraitType.Binary, x)
    assert vr.n_markers_used == fr.variance_ratio.n_markers_used
    assert vr.variance_ratio == fr.variance_ratio.variance_ratio
