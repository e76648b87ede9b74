"""One-column MIXED products at the edges of their tiles, row blocks and list chunks.

The sums are integers: products are compared to the bit with the CPU model and with the
block path (SAIGE_SC=0), dense and with the missing-call lists."""
import numpy as np
import pytest

import csaige_b200 as cs
import mixed_model as MM
import oracle_ffi as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("lists", ["0", "2"])
@pytest.mark.parametrize("n,m", [
    (5, 3),         # one tile each way, most of it padding
    (129, 64),      # up to a block of markers, two sample tiles
    (1025, 75),     # a few markers in a second block
    (4097, 140),    # one sample past a chunk of the lists, a second marker tile
    (300, 1100),    # markers past a chunk of the lists
    (9001, 2100),   # pass B divided, chunks falling to different blocks
    (70, 9000),     # pass A undivided, pass B over many marker tiles of one row block
])
def test_one_column_products_at_the_edges(monkeypatch, n, m, lists):
    monkeypatch.setenv("SAIGE_SR_LISTS", lists)
    bed = cs.gen_bed(cs.CohortSpec(n=n, m=m, seed=n + m, missing_rate=0.02))
    af, mac, nv = O.marker_stats(bed, n, m, None)
    keep = np.nonzero((af >= 0.01) & (af <= 0.99))[0]
    grm = cs.OnTheFlyGrm.from_bed(bed, n, m, keep, af[keep], precision=cs.PREC_MIXED)
    v = np.random.default_rng(n).standard_normal((2, n))
    v[1] = np.where(np.arange(n) == n - 1, 1.0, 0.0)  # one entry, the last sample's
    want = MM.kv(MM.codes(bed, n, keep), af[keep], v.T).T
    for _ in range(2):  # sums and tickets are zero again
        for x, y in zip(v, want):
            assert np.array_equal(grm.mat_vec(x), y)
    monkeypatch.setenv("SAIGE_SC", "0")
    assert np.array_equal(grm.mat_vec(v[0]), want[0])


def test_lists_are_left_where_the_flags_are_cheaper(monkeypatch):
    # a handle above 2^22 entries: the second fit lists its missing calls up to 0.3 %
    monkeypatch.delenv("SAIGE_SR_LISTS", raising=False)
    for miss, listed in ((0.001, True), (0.01, False)):
        spec = cs.CohortSpec(n=3000, m=4000, seed=5, missing_rate=miss)
        bed = cs.gen_bed(spec)
        y, x = cs.gen_pheno(spec)
        af, mac, nv = cs.bed_marker_stats(bed, spec.n, spec.m)
        g, _ = cs.select_grm_markers(af, mac, nv, spec.n)
        grm = cs.OnTheFlyGrm.from_bed(bed, spec.n, spec.m, g, af[g], precision=cs.PREC_MIXED)
        cfg = cs.AiRemlConfig(max_iter=30, tol=1e-5, precision=cs.PREC_MIXED,
                              solve=cs.SOLVE_BLOCK, warm_start=cs.WARM_RECYCLED)
        r = [cs.fit_ai_reml(y, x, grm, cs.TraitType.Binary, cfg) for _ in range(2)]
        assert np.array_equal(r[0].tau, r[1].tau)
        v = np.random.default_rng(1).standard_normal(spec.n)
        a = grm.mat_vec(v)  # (the fits may have had no one-column product)
        assert (grm.stats()["missing_listed"] > 0) == listed
        # asked for, they are built after all
        monkeypatch.setenv("SAIGE_SR_LISTS", "2")
        assert np.array_equal(a, grm.mat_vec(v))
        assert grm.stats()["missing_listed"] > 0
        monkeypatch.setenv("SAIGE_SR_LISTS", "0")
        assert np.array_equal(a, grm.mat_vec(v))
        monkeypatch.delenv("SAIGE_SR_LISTS")
