"""Explicit GRMs whose last wave of tiles is shared between two launches.

Every entry's sum keeps its order across the launches, so the matrix equals the oracle's bit
for bit.  With 148 SMs, n = 2,300 (18 x 18 tiles) shares its tiles in halves, n = 2,700 in
thirds, n = 3,000 fills its second wave and takes one launch, as do few markers."""
import numpy as np
import pytest

import csaige_b200 as cs
import oracle_ffi as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,m", [(2300, 300), (2300, 100), (2700, 700), (3000, 300)])
def test_shared_tiles_are_bit_identical_to_oracle(n, m):
    bed = cs.gen_bed(cs.CohortSpec(n=n, m=m, seed=n, missing_rate=0.01, sib_frac=0.2,
                                   cousin_frac=0.1, maf_lo=0.005, maf_hi=0.5))
    want, used_o = O.dense_grm_bed(bed, n, m)
    k, used = cs.compute_dense_grm(bed, n, m)
    assert used == used_o and np.array_equal(k, want)
    for cutoff in (0.125, -1.0):  # -1: more entries than the first guess, launched again
        g, _ = cs.compute_sparse_grm(bed, n, m, relatedness_cutoff=cutoff)
        r, c, v = O.sparse_from_dense(want, cutoff)
        assert np.array_equal(g.rows, r) and np.array_equal(g.cols, c)
        assert np.array_equal(g.vals, v)
