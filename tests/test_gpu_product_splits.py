"""The one-column MIXED product's division of the markers over thread blocks (pass B).

The partial sums are integers, so every division gives the same product: it is compared
to the bit with the CPU model and with the tensor-core passes, which do not divide."""
import numpy as np
import pytest

import csaige_b200 as cs
import mixed_model as MM
import oracle_ffi as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("lists", ["2", "0"])
@pytest.mark.parametrize("n,m", [
    (300, 100),      # one pair of sample tiles, one marker tile: nothing to divide
    (520, 2300),     # few samples: chunks divided down to single tiles, ragged last chunk
    (2000, 5000),    # the CPU-scale cohort
    (40000, 500),    # many sample tiles, one partial chunk
    (30000, 4200),   # whole chunks, the last one of one tile
])
def test_one_column_marker_splits_give_the_same_product(monkeypatch, n, m, lists):
    monkeypatch.setenv("SAIGE_SR_LISTS", lists)
    spec = cs.CohortSpec(n=n, m=m, seed=n + m, missing_rate=0.02)
    bed = cs.gen_bed(spec)
    af, mac, nv = O.marker_stats(bed, n, m, None)
    keep = np.nonzero((af >= 0.01) & (af <= 0.99))[0]
    grm = cs.OnTheFlyGrm.from_bed(bed, n, m, keep, af[keep], precision=cs.PREC_MIXED)
    v = np.random.default_rng(n).standard_normal((2, n))
    first = [grm.mat_vec(x) for x in v]
    again = [grm.mat_vec(x) for x in v]  # the kept sums are zero again after each product
    assert all(np.array_equal(a, b) for a, b in zip(first, again))
    monkeypatch.setenv("SAIGE_SC", "0")
    for x, got in zip(v, first):
        assert np.array_equal(got, grm.mat_vec(x))
    if n * m < 20_000_000:
        want = MM.kv(MM.codes(bed, n, keep), af[keep], v[:1].T).T
        assert np.array_equal(first[0], want[0])


@pytest.mark.parametrize("n,m", [
    (4000, 3000),    # pass A: tiles shared by several CTAs; pass B: a CTA per tile
    (3000, 20000),   # pass B: each tile shared by six CTAs; pass A: whole tiles and one more
    (20000, 20100),  # both: a wave of whole tiles, the rest shared
])
@pytest.mark.parametrize("q", [2, 42, 43, 64])  # four operand slots, four, three, two
def test_block_products_with_shared_tiles_equal_one_column_products(n, m, q):
    spec = cs.CohortSpec(n=n, m=m, seed=n + m + q, missing_rate=0.02)
    bed = cs.gen_bed(spec)
    af, mac, nv = cs.bed_marker_stats(bed, n, m)
    keep = np.nonzero((af >= 0.01) & (af <= 0.99))[0]
    grm = cs.OnTheFlyGrm.from_bed(bed, n, m, keep, af[keep], precision=cs.PREC_MIXED)
    v = np.random.default_rng(q).standard_normal((q, n))
    got = grm.mat_vec(v)
    assert np.array_equal(got, grm.mat_vec(v))  # the shared tiles' sums are zero again
    for c in sorted({0, 1, q // 2, q - 1}):
        assert np.array_equal(got[c], grm.mat_vec(v[c]))
