"""rtb_rearrange around the number of lost rays up to which library vectors are
swapped in place (GPU test): the reordering of ordinary arrays.
"""
import ctypes as C

import numpy as np
import pytest

from rt_b200 import engine as E
from rt_b200 import ffi
from test_gpu_vectors import FIELDS, Vectors, rays

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [2049, 30_000])
@pytest.mark.parametrize("lost", [1, 2047, 2048, 2049])
@pytest.mark.parametrize("where", ["front", "back", "anywhere"])
@pytest.mark.parametrize("flags", ["vector", "array"])
def test_rearrange_around_the_line(n, lost, where, flags):
    plain = rays(n, 0.0)
    pick = {"front": np.arange(lost), "back": np.arange(n - lost, n),
            "anywhere": np.random.default_rng(lost).permutation(n)[:lost]}[where]
    plain["flag"][pick] = 0
    vec = Vectors(plain, 0)
    try:
        mixed = dict(vec.a, flag=plain["flag"].copy()) if flags == "array" else vec.a
        for a in (mixed, plain):
            good = C.c_size_t(n)
            ffi.check(E.lib().rtb_rearrange(C.byref(good), *(ffi.vptr(a[k]) for k in FIELDS + ("flag",))), "rearrange")
            assert good.value == n - lost
            assert a["flag"][:good.value].all() and not a["flag"][good.value:].any()
        for k in plain:
            assert np.array_equal(mixed[k], plain[k]), k
    finally:
        vec.free()
