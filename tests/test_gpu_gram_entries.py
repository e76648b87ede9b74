"""The Gram products of the recycled starts, entry by entry, with both tile sizes.

Integer entries: every partial sum is an integer below 2^53, so the products are exact in any
order.  For other entries the two tiles run the same chains and give the same bits."""
import ctypes as C

import numpy as np
import pytest

import csaige_b200 as cs  # noqa: F401  (loads the library)
from csaige_b200._lib import LIB, check

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")


def _gram(a, b, n, tile):
    out = torch.full((a.shape[0], b.shape[0]), float("nan"), dtype=torch.float64, device="cuda")
    torch.cuda.synchronize()
    check(LIB.saige_gram_dev(C.c_void_p(a.data_ptr()), a.shape[0], C.c_void_p(b.data_ptr()),
                             b.shape[0], n, a.shape[1], tile, C.c_void_p(out.data_ptr()), -1))
    return out.cpu().numpy()


def _columns(rng, k, n, ld, integers):
    x = np.full((k, ld), np.nan)  # rows from n on are not read
    x[:, :n] = rng.integers(-8, 9, (k, n)) if integers else rng.standard_normal((k, n))
    return x


# a, b: inside, at and past the edges of 16 and 32 columns; n: one row, a ragged pair, a ragged
# chunk, and enough rows (and tiles) for the rule to take the 32-column tile
@pytest.mark.parametrize("a,b", [(1, 1), (16, 17), (31, 33), (32, 32), (63, 64), (97, 146)])
@pytest.mark.parametrize("n", [1, 33, 2049, 9001, 200001])
def test_gram_entries_are_exact_and_tiles_agree(a, b, n):
    rng = np.random.default_rng(1000 * a + n)
    ld = (n + 511) // 512 * 512
    for integers in (True, False):
        x, y = _columns(rng, a, n, ld, integers), _columns(rng, b, n, ld, integers)
        dx, dy = torch.from_numpy(x).cuda(), torch.from_numpy(y).cuda()
        got = [_gram(dx, dy, n, tile) for tile in (0, 16, 32)]
        assert np.array_equal(got[1], got[2])
        assert np.array_equal(got[0], got[1])
        if integers:
            assert np.array_equal(got[0], x[:, :n] @ y[:, :n].T)


def test_misaligned_columns_are_refused():
    x = torch.zeros(3, 64, dtype=torch.float64, device="cuda")
    out = torch.zeros(1, dtype=torch.float64, device="cuda")
    p = C.c_void_p(x.data_ptr())
    odd = C.c_void_p(x.data_ptr() + 8)
    call = lambda a, b, ld: LIB.saige_gram_dev(a, 1, b, 1, 30, ld, 0, C.c_void_p(out.data_ptr()), -1)
    assert call(p, p, 64) == 0
    for a, b, ld in ((odd, p, 64), (p, odd, 64), (p, p, 63), (p, p, 28)):
        assert call(a, b, ld) == 1  # EINVAL
