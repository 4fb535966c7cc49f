"""The plain engine's shared-reciprocal quotients (quotient.cuh) against the
oracle's IEEE divisions (GPU tests): the same bits, on inputs at the edges of
what the fast forms take and beyond them.
"""
import ctypes as C

import numpy as np
import pytest

import pyoracle as O
from rt_b200 import engine as E
from rt_b200 import ffi
from test_gpu_parity import same_bits

pytestmark = pytest.mark.gpu

SPECIAL = np.array([0.0, -0.0, 1.0, -1.0, np.inf, -np.inf, np.nan, 5e-324, -5e-324, 1e-310, 1e308, 2.0 ** -899,
                    2.0 ** -901, -(2.0 ** -900), 2.0 ** -450, 2.0 ** -1022, 1 - 2.0 ** -53, 1 + 2.0 ** -52, 0.6, 0.8])


def directions(kind, n=200_003):
    rng = np.random.default_rng(71)
    v = rng.uniform(-1, 1, (3, n))
    if kind == "special":                                # every triple of them
        return np.stack(np.meshgrid(SPECIAL, SPECIAL, SPECIAL, indexing="ij")).reshape(3, -1).copy()
    if kind == "any":                                    # any bits at all
        return rng.integers(0, 2 ** 64, (3, n), dtype=np.uint64).view(np.float64)
    if kind == "small":                                  # one component down to 2^-1100
        i = rng.integers(0, 3, n)
        v[i, np.arange(n)] *= 2.0 ** -(rng.integers(0, 1075, n).astype(float))
    v /= np.sqrt((v * v).sum(0))
    if kind == "ulps":                                   # unit vectors a few last places off
        v.view(np.int64)[:] += rng.integers(-40, 41, v.shape)
    if kind == "off":                                    # |c| - 1 from 2^-53 to 2^-20, the limit 2^-28 among them
        v *= 1 + rng.choice([-1, 1], n) * 2.0 ** -rng.uniform(20, 53, n)
    if kind == "ties":                                   # few-bit components beside one next to 1
        v = rng.integers(-31, 32, (3, n)) * 2.0 ** -rng.integers(5, 60, (3, n)).astype(float)
        v[rng.integers(0, 3, n), np.arange(n)] = 1 + rng.integers(-4, 5, n) * 2.0 ** -53
    return v


@pytest.mark.parametrize("kind", ["unit", "ulps", "off", "ties", "small", "special", "any"])
def test_normalize_has_the_bits_of_ieee_divisions(kind):
    v = directions(kind)
    got, want = [x.copy() for x in v], [x.copy() for x in v]
    n = C.c_size_t(v.shape[1])
    ffi.check(E.lib().rtb_normalize(n, *map(ffi.vptr, got)), "rtb_normalize")
    assert O.load().oracle_normalize(n, *map(ffi.vptr, want)) == 0
    for g, w in zip(got, want):
        assert same_bits(g, w)
