"""The scales of a MIXED product's operands: block maxima and operand images.

The integer arithmetic is compared to the bit with the CPU model, for columns whose largest
entry lies at the edges of the blocks that look for it."""
import numpy as np
import pytest

import csaige_b200 as cs
import mixed_model as MM
import oracle_ffi as O

pytestmark = pytest.mark.gpu


def _case(n, m):
    bed = cs.gen_bed(cs.CohortSpec(n=n, m=m, seed=n + m, missing_rate=0.02))
    af, mac, nv = O.marker_stats(bed, n, m, None)
    keep = np.nonzero((af >= 0.01) & (af <= 0.99))[0]
    grm = cs.OnTheFlyGrm.from_bed(bed, n, m, keep, af[keep], precision=cs.PREC_MIXED)
    return grm, MM.codes(bed, n, keep), af[keep]


@pytest.mark.parametrize("n,m", [(4097, 300), (260, 4200), (2048, 129)])
def test_largest_entry_at_block_edges(n, m):
    grm, codes, af = _case(n, m)
    rows = sorted({r for r in (0, 31, 255, 256, 2047, 2048, 4096, n - 1) if r < n})
    v = np.random.default_rng(n).standard_normal((len(rows) + 1, n))
    for c, r in enumerate(rows):
        v[c, r] = -1000.0 - c
    v[-1] = 0.0  # no largest entry: the product is 0
    want = MM.kv(codes, af, v.T).T
    assert np.array_equal(grm.mat_vec(v), want)
    for c in (0, len(rows) - 1, len(rows)):
        assert np.array_equal(grm.mat_vec(v[c]), want[c])


def test_images_hold_nothing_of_an_earlier_wider_product():
    grm, codes, af = _case(700, 300)
    v = np.random.default_rng(3).standard_normal((70, 700))
    grm.mat_vec(v)  # 64 + 6 columns
    want = MM.kv(codes, af, v.T).T
    for q in (3, 5, 6, 21, 64, 65, 70):  # 9, 15, 18, 63, 192 limb rows of 16, 16, 32, 64, 192
        assert np.array_equal(grm.mat_vec(v[:q]), want[:q])
