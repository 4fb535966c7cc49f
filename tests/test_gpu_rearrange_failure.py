"""rtb_rearrange when one of its device allocations fails (GPU test; the
failure is made on the host, by the library's fault hook): the caller's count
and arrays stay as they were, and the next call reorders them.
"""
import ctypes as C

import numpy as np
import pytest

from rt_b200 import engine as E
from rt_b200 import ffi

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("vectors", [False, True])
def test_failed_rearrange_changes_nothing(vectors):
    L = E.lib()
    L.rtb_fail_allocations.argtypes = [C.c_uint32, C.c_uint32]
    n = 10_000
    rng = np.random.default_rng(5)
    source = [rng.normal(size=n) for _ in range(7)]
    lost = rng.random(n) < 0.4
    ptrs = [L.rtb_alocate_vector(n) for _ in range(8)] if vectors else []
    try:
        words = [np.ctypeslib.as_array(p, shape=(n,)) for p in ptrs] if vectors else [np.zeros(n) for _ in range(8)]
        a, flag = words[:7], words[7].view(np.int8)[:n]

        def reset():
            for x, s in zip(a, source):
                x[:] = s
            flag[:] = ~lost

        def call(n_good):
            return L.rtb_rearrange(C.byref(n_good), *map(ffi.vptr, a), ffi.vptr(flag))

        reset()
        good = C.c_size_t(n)
        assert call(good) == ffi.OK and good.value == int((~lost).sum())
        want = [x.copy() for x in a] + [flag.copy()]
        assert set(a[0][:good.value]) == set(source[0][~lost]) and flag[:good.value].all()
        failed = 0
        for after in range(6):
            reset()
            good = C.c_size_t(n)
            L.rtb_fail_allocations(after, 1)
            st = call(good)
            L.rtb_fail_allocations(0, 0)
            assert st in (ffi.OK, ffi.BAD_ALLOC)
            if st == ffi.BAD_ALLOC:
                failed += 1
                assert good.value == n, after
                assert all(np.array_equal(x, s) for x, s in zip(a, source)) and np.array_equal(flag, (~lost).astype(np.int8))
                assert call(good) == ffi.OK
            assert good.value == int((~lost).sum())
            assert all(np.array_equal(x, w) for x, w in zip(a + [flag], want))
        assert failed >= 3
    finally:
        L.rtb_fail_allocations(0, 0)
        for p in ptrs:
            L.rtb_free_vector(p)
