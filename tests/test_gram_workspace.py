"""Partial sums of the recycled starts' Gram products (no GPU): the workspace that a fit
reserves for its widest basis holds the products of every narrower one, which are cut into
more row chunks (n = 200,000, 10 covariates and 30 probes: 592,800 doubles for a basis of 95
columns, 473,352 for the widest, 130)."""
import ctypes as C

import pytest

from csaige_b200._lib import LIB, check

PROBES = 30


def _workspace(n, a, b):
    needed, reserved = C.c_int64(), C.c_int64()
    check(LIB.saige_gram_workspace(n, a, b, C.byref(needed), C.byref(reserved)))
    return needed.value, reserved.value


def _widest(p, probes, learned):
    """ai_reml.cu's recycle_init: basis columns and right-hand sides."""
    q = 1 + p + probes
    return (3 if learned else 2) * q + 1 + min(3 * (1 + p), 48), q


@pytest.mark.parametrize("n", [1, 500, 2048, 2049, 20000, 100000, 200000, 300000, 2000000])
@pytest.mark.parametrize("p", [1, 3, 7, 11, 16, 40])
@pytest.mark.parametrize("learned", [False, True])
def test_widest_basis_reserves_for_every_narrower_one(n, p, learned):
    widest, q = _widest(p, PROBES, learned)
    _, reserved = _workspace(n, widest, widest + q)
    for a in range(1, widest + 1):
        for b in (a + 1, a + q):  # an AI solve's start, a block start
            assert _workspace(n, a, b)[0] <= reserved, (a, b)
    # no more than the larger of one chunk of the widest product and 592 tiles of 32 x 32
    assert reserved <= max(widest * (widest + q), 592 * 1024)


def test_sizes_of_the_reported_overflow():
    assert _workspace(200000, 62, 100)[0] == 458800
    assert _workspace(200000, 101, 139)[0] == 407131 < 458800 <= _workspace(200000, 101, 139)[1]
