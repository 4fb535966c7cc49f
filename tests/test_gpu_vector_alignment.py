"""Arrays inside library vectors that do not start at a multiple of their
elements' size (GPU tests): the calls copy them, as they copy any other
array, and give the results of ordinary arrays.
"""
import ctypes as C

import numpy as np
import pytest

from rt_b200 import engine as E
from rt_b200 import ffi, schemes as S
from test_gpu_vectors import PlainRays, rays, stages

pytestmark = pytest.mark.gpu


class Unaligned:
    """A copy of an array `offset` bytes into a library vector."""

    def __init__(self, values, offset):
        self.ptr = E.lib().rtb_alocate_vector(len(values) + 8)
        words = np.ctypeslib.as_array(self.ptr, shape=(len(values) + 8,)).view(np.uint8)
        self.a = words[offset:offset + values.nbytes].view(values.dtype)
        self.a[:] = values

    def free(self):
        E.lib().rtb_free_vector(self.ptr)


@pytest.mark.parametrize("n", [1, 12_289])
@pytest.mark.parametrize("offset", [1, 4])
def test_drop_in_calls(n, offset):
    plain = rays(n, 0.01)
    held = {k: Unaligned(v, offset) for k, v in plain.items()}
    pixels = [Unaligned(np.zeros(n, np.uint32), offset) for _ in range(2)]
    try:
        a = {k: h.a for k, h in held.items()}
        status = stages(plain, n)
        assert status[:7] == [ffi.OK] * 7 and stages(a, n) == status
        for k, v in plain.items():
            assert np.array_equal(np.frombuffer(a[k].tobytes(), np.uint8), v.view(np.uint8)), k
        want = [np.zeros(n, np.uint32) for _ in range(2)]
        for pos, out in (([plain["X"], plain["Y"]], want), ([a["X"], a["Y"]], [p.a for p in pixels])):
            ffi.check(E.lib().rtb_ccd_coordinates(C.c_size_t(n), *map(ffi.vptr, pos), *map(C.c_double, (30, 30, .015, .015)),
                                                  *map(ffi.vptr, out)), "rtb_ccd_coordinates")
        assert all(np.array_equal(p.a, w) for p, w in zip(pixels, want))
    finally:
        for h in list(held.values()) + pixels:
            h.free()


@pytest.mark.parametrize("precision", [ffi.FP64, ffi.MIXED])
@pytest.mark.parametrize("offset", [1, 4])
def test_host_trace(precision, offset):
    n = 4099
    surf = S.to_c(S.echelle(), E.spline_init).surfaces
    beams = [S.make_beam(0, n, 1, S.C1_RADIUS, (0.6, 0.6), 3, orders=(45, 1))]
    source = E.generate(beams, n)
    results = []
    for unaligned in (False, True):
        h = PlainRays(n)
        for f in E.FIELDS + ("flag", "lost_stage"):
            getattr(h, f)[:] = getattr(source, f).cpu().numpy()
        held = [Unaligned(getattr(h, f), offset) for f in E.FIELDS + ("flag", "lost_stage")] if unaligned else []
        try:
            for f, u in zip(E.FIELDS + ("flag", "lost_stage"), held):
                setattr(h, f, u.a)
            st, stats = E.trace_host(surf, beams, h, E.opts(precision=precision, fixes=3, state_out=1))
            ffi.check(st, "rtb_trace_host")
            results.append([getattr(h, f).tobytes() for f in E.FIELDS + ("flag", "lost_stage")])
        finally:
            for u in held:
                u.free()
    assert results[0] == results[1]
