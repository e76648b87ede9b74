"""Which handles sum over lists of their missing calls by themselves: small ones only, since the
dense flag sums are faster."""
import numpy as np
import pytest

import csaige_b200 as cs

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,m,miss,listed", [
    (2000, 1000, 0.01, True),    # up to 2^22 entries
    (3000, 4000, 0.001, True),   # up to 2^24 with few calls missing
    (3000, 4000, 0.01, False),
    (5000, 5000, 0.001, False),  # above 2^24
    (9001, 4003, 0.0, False),
])
def test_second_fit_lists_the_missing_calls_of_small_handles(monkeypatch, n, m, miss, listed):
    monkeypatch.delenv("SAIGE_SR_LISTS", raising=False)
    spec = cs.CohortSpec(n=n, m=m, seed=6, missing_rate=miss)
    bed = cs.gen_bed(spec)
    y, x = cs.gen_pheno(spec)
    af, mac, nv = cs.bed_marker_stats(bed, n, m)
    keep = np.nonzero((af >= 0.01) & (af <= 0.99))[0]
    grm = cs.OnTheFlyGrm.from_bed(bed, n, m, keep, af[keep], precision=cs.PREC_MIXED)
    cfg = cs.AiRemlConfig(max_iter=3, precision=cs.PREC_MIXED, solve=cs.SOLVE_BLOCK,
                          warm_start=cs.WARM_RECYCLED)
    v = np.random.default_rng(7).standard_normal(n)
    a = grm.mat_vec(v)
    r = [cs.fit_ai_reml(y, x, grm, cs.TraitType.Binary, cfg) for _ in range(2)]
    b = grm.mat_vec(v)
    st = grm.stats()
    assert (st["missing_listed"] >= 0, st["sc_list_launches"] > 0) == (listed, listed)
    assert np.array_equal(r[0].tau, r[1].tau) and np.array_equal(a, b)
