"""Drop-in calls that only read library vectors beside ordinary arrays, around
the size from which the vectors are copied too (GPU tests): the results of
ordinary arrays.
"""
import ctypes as C

import numpy as np
import pytest

from rt_b200 import engine as E
from rt_b200 import ffi, schemes as S
from test_gpu_vectors import Vectors, rays

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [65_535, 65_536, 131_071, 131_072])
def test_positions_in_vectors_and_ordinary_flags(n):
    plain = rays(n, 0.1)
    vec = Vectors({k: plain[k] for k in ("X", "Y", "lam")}, 0)
    qe = ffi.TableHolder(*S.qe_table())
    qe.y2[:] = E.spline_init(qe.x, qe.y)
    size, centre = (C.c_double * 2)(4.0, 0.0), (C.c_double * 2)(0.3, -0.2)
    try:
        results = []
        for a in (plain, vec.a):
            flag, spec, bad = plain["flag"].copy(), np.linspace(0, 1, n), C.c_size_t(3)
            ffi.check(E.lib().rtb_apply_constrains(0, ffi.CIRCLE, size, centre, C.c_size_t(n), ffi.vptr(a["X"]),
                                                   ffi.vptr(a["Y"]), ffi.vptr(flag), C.byref(bad)), "rtb_apply_constrains")
            ffi.check(E.lib().rtb_surface_QE(C.c_size_t(n), ffi.vptr(a["lam"]), ffi.vptr(spec), C.byref(qe.table)),
                      "rtb_surface_QE")
            results.append((flag, spec, bad.value))
        (f0, s0, b0), (f1, s1, b1) = results
        assert np.array_equal(f0, f1) and np.array_equal(s0, s1) and b0 == b1
        inside = np.hypot(plain["X"] - 0.3, plain["Y"] + 0.2) <= 4.0
        assert np.array_equal(f0 == 1, inside & (plain["flag"] == 1)) and b0 == 3 + int((~inside).sum())
        assert all(np.array_equal(vec.a[k], plain[k]) for k in vec.a)
    finally:
        vec.free()
