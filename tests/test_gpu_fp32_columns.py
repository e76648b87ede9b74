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
