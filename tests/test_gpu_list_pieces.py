"""Missing-call lists whose segments are longer than the piece that is staged in shared memory
(4,096 entries): the rest is read from global memory, for the same integers."""
import numpy as np
import pytest

import csaige_b200 as cs
import mixed_model as MM
import oracle_ffi as O

pytestmark = pytest.mark.gpu


def _missing(bed, n, markers, samples):
    """Sets the calls of these markers and samples to missing (code 01)."""
    rows = bed[3:].reshape(-1, (n + 3) // 4)
    for s in samples:
        at, shift = s // 4, 2 * (s % 4)
        rows[markers, at] = (rows[markers, at] & (0xFF ^ (3 << shift))) | (1 << shift)


# pass A: 64 markers x 4,096 samples per segment; pass B: 256 samples x 1,024 markers
@pytest.mark.parametrize("case", ["markers", "samples", "both"])
def test_segments_longer_than_a_piece(monkeypatch, case):
    n, m = 9001, 1300
    monkeypatch.setenv("SAIGE_SR_LISTS", "2")
    bed = cs.gen_bed(cs.CohortSpec(n=n, m=m, seed=12, missing_rate=0.002)).copy()
    rng = np.random.default_rng(5)
    if case != "samples":  # six neighbouring markers, 60 % of their calls: 14,700 in a segment
        _missing(bed, n, np.arange(130, 136), rng.permutation(n)[: int(0.6 * n)])
    if case != "markers":  # nine samples of one row block, 95 % of their calls: 9,200
        _missing(bed, n, rng.permutation(m)[: int(0.95 * m)], range(5130, 5139))
    af, _, _ = O.marker_stats(bed, n, m, None)
    keep = np.nonzero((af >= 0.01) & (af <= 0.99))[0]
    codes = MM.codes(bed, n, keep)
    assert 0 < (codes == 1).mean() < 0.03
    segments_a = [(codes[i:i + 64, j:j + 4096] == 1).sum() for i in range(0, len(keep), 64)
                  for j in range(0, n, 4096)]
    segments_b = [(codes[j:j + 1024, i:i + 256] == 1).sum() for i in range(0, n, 256)
                  for j in range(0, len(keep), 1024)]
    assert (max(segments_a) > 2 * 4096) == (case != "samples")
    assert (max(segments_b) > 2 * 4096) == (case != "markers")
    grm = cs.OnTheFlyGrm.from_bed(bed, n, m, keep, af[keep], precision=cs.PREC_MIXED)
    v = rng.standard_normal((2, n))
    want = MM.kv(codes, af[keep], v.T).T
    for x, y in zip(v, want):
        assert np.array_equal(grm.mat_vec(x), y)
    assert grm.stats()["missing_listed"] == (codes == 1).sum()
    assert grm.stats()["sc_list_launches"] == 2
