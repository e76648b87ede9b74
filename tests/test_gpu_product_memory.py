"""Device memory that MIXED products of a few columns take."""
import numpy as np
import pytest

import csaige_b200 as cs
import mixed_model as MM
from csaige_b200._lib import LIB, check

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")


def test_sums_of_shared_tiles_are_sized_by_the_columns():
    # 19 MB for 64 columns whatever the product had; two columns need 0.6 MB
    n, m = 3000, 900
    bed = cs.gen_bed(cs.CohortSpec(n=n, m=m, seed=8, missing_rate=0.02))
    af, _, _ = cs.bed_marker_stats(bed, n, m)
    keep = np.nonzero((af >= 0.05) & (af <= 0.95))[0]
    v = np.random.default_rng(3).standard_normal((40, n))
    want = MM.kv(MM.codes(bed, n, keep), af[keep], v.T).T
    for _ in range(2):  # (the first handle loads the kernels)
        grm = cs.OnTheFlyGrm.from_bed(bed, n, m, keep, af[keep], precision=cs.PREC_MIXED)
        grm.mat_vec(v[0])  # builds the tiles
        check(LIB.saige_release_cached_memory())
        before, _ = torch.cuda.mem_get_info()
        got = grm.mat_vec(v[:2])
        after, _ = torch.cuda.mem_get_info()
        assert np.array_equal(got, want[:2])
        # more columns: the room grows, its counts and sums zero again; fewer use it as it is
        for k in (40, 3, 17, 40):
            assert np.array_equal(grm.mat_vec(v[:k]), want[:k]), k
        grm.close()
    assert before - after <= 8 << 20  # (allocations come in steps of 2 MB)
