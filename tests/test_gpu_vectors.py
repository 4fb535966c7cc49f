"""The drop-in calls on the library's page-locked vectors, which the kernels
read and write in place, against the same calls on ordinary arrays (GPU
tests): the same bits, whatever arrays are mixed, shared or offset.
"""
import ctypes as C

import numpy as np
import pytest

from rt_b200 import engine as E
from rt_b200 import ffi, schemes as S

pytestmark = pytest.mark.gpu

FIELDS = ("X", "Y", "Z", "cX", "cY", "cZ", "lam")


class Vectors:
    """Arrays of doubles in library vectors, `offset` elements into them."""

    def __init__(self, arrays, offset):
        self.ptrs, self.a = [], {}
        for k, v in arrays.items():
            p = E.lib().rtb_alocate_vector(len(v) + offset + 8)
            self.ptrs.append(p)
            words = np.ctypeslib.as_array(p, shape=(len(v) + offset + 8,))
            if k == "flag":
                self.a[k] = words.view(np.int8)[offset:offset + len(v)]
            else:
                self.a[k] = words[offset:offset + len(v)]
            self.a[k][:] = v

    def free(self):
        for p in self.ptrs:
            E.lib().rtb_free_vector(p)


def rays(n, lost):
    rng = np.random.default_rng(n)
    a = {k: rng.uniform(-5, 5, n) for k in ("X", "Y", "Z")}
    c = rng.uniform(-0.1, 0.1, (2, n))
    a.update(cX=c[0], cY=c[1], cZ=np.sqrt(1 - (c * c).sum(0)), lam=rng.uniform(0.4, 0.7, n))
    a["Z"] -= 60.0
    a["flag"] = (rng.random(n) >= lost).astype(np.int8)
    return a


def stages(a, n):
    """One surface's calls and a reordering; the arrays change in place."""
    L, P = E.lib(), {k: ffi.vptr(v) for k, v in a.items()}
    pos, cos, N = [P[k] for k in FIELDS[:3]], [P[k] for k in FIELDS[3:6]], C.c_size_t(n)
    par = (C.c_double * 16)(-1 / 300.0, -0.2)
    angles, dist = (C.c_double * 3)(0.02, -0.01, 0.3), (C.c_double * 3)(0.1, 0.2, -3.0)
    size, centre, bad = (C.c_double * 2)(6.0, 0.0), (C.c_double * 2)(0.3, -0.2), C.c_size_t(7)
    glass, air = ffi.TableHolder(*S.glass_table()), ffi.TableHolder(value=1.0)
    glass.y2[:] = E.spline_init(glass.x, glass.y)
    good = C.c_size_t(n)
    out = [L.rtb_beam_transform(N, angles, dist, *pos, *cos), L.rtb_normalize(N, *cos),
           L.rtb_surface_intersection(ffi.CONIC, par, N, *pos, *cos, C.byref(bad), P["flag"]),
           L.rtb_apply_constrains(0, ffi.CIRCLE, size, centre, N, *pos[:2], P["flag"], C.byref(bad)),
           L.rtb_surface_reflection(ffi.CONIC, par, N, *pos, *cos),
           L.rtb_surface_refraction(ffi.PLANE, par, N, *pos, *cos, P["lam"], C.byref(air.table), C.byref(glass.table),
                                    C.byref(bad), P["flag"]),
           L.rtb_rearrange(C.byref(good), *pos, *cos, P["lam"], P["flag"])]
    return out + [bad.value, good.value]


@pytest.mark.parametrize("n,lost", [(1, 0.0), (255, 0.5), (12_288, 0.002), (40_001, 0.0), (40_001, 0.01), (40_001, 0.9)])
@pytest.mark.parametrize("offset", [0, 1, 3])
def test_library_vectors_give_the_same_bits(n, lost, offset):
    plain = rays(n, lost)
    want = {k: v.copy() for k, v in plain.items()}
    # the aperture loses many rays; a wide one leaves the few that `flag` marks
    status = stages(want, n)
    vec = Vectors(plain, offset)
    mixed = {k: (vec.a[k] if i % 2 else v.copy()) for i, (k, v) in enumerate(plain.items())}
    try:
        for a in (mixed, vec.a):
            for k, v in plain.items():
                a[k][:] = v
            assert stages(a, n) == status
            for k in plain:
                assert np.array_equal(a[k].view(np.uint8), want[k].view(np.uint8)), k
    finally:
        vec.free()


@pytest.mark.parametrize("n,lost", [(50_000, 0.001), (50_000, 0.0), (50_000, 0.3), (64, 1 / 64), (63, 0.5)])
def test_rearrange_in_place_and_in_copies(n, lost):
    plain = rays(n, lost)
    want = {k: v.copy() for k, v in plain.items()}
    vec = Vectors(plain, 0)
    try:
        for a in (want, vec.a):
            good = C.c_size_t(n)
            ffi.check(E.lib().rtb_rearrange(C.byref(good), *(ffi.vptr(a[k]) for k in FIELDS + ("flag",))), "rearrange")
            assert good.value == int(plain["flag"].sum())
        for k in plain:
            assert np.array_equal(vec.a[k].view(np.uint8), want[k].view(np.uint8)), k
        # an array given twice
        for a in (want, vec.a):
            for k, v in plain.items():
                a[k][:] = v
            good = C.c_size_t(n)
            args = [ffi.vptr(a[k]) for k in FIELDS[:6]] + [ffi.vptr(a["cZ"]), ffi.vptr(a["flag"])]
            ffi.check(E.lib().rtb_rearrange(C.byref(good), *args), "rearrange")
        for k in plain:
            assert np.array_equal(vec.a[k].view(np.uint8), want[k].view(np.uint8)), k
    finally:
        vec.free()


def test_shared_arrays_are_read_as_they_were():
    """An output that is also an input, in a vector and outside one."""
    n = 5000
    lam = np.linspace(0.4, 0.7, n)
    t = ffi.TableHolder(*S.qe_table())
    t.y2[:] = E.spline_init(t.x, t.y)
    vec = Vectors({"lam": lam}, 0)
    try:
        results = []
        for a in (lam.copy(), vec.a["lam"]):
            ffi.check(E.lib().rtb_surface_QE(n, ffi.vptr(a), ffi.vptr(a), C.byref(t.table)), "rtb_surface_QE")
            results.append(a.copy())
        assert np.array_equal(*results)
    finally:
        vec.free()


class PlainRays:
    """Ordinary host arrays with the fields rtb_trace_host takes."""

    def __init__(self, n):
        self.n = n
        for f in E.FIELDS:
            setattr(self, f, np.zeros(n))
        self.flag, self.lost_stage = np.ones(n, np.int8), np.zeros(n, np.uint8)

    def struct(self):
        return ffi.Rays(*(ffi.vptr(getattr(self, f)) for f in E.FIELDS), ffi.vptr(self.flag),
                        ffi.vptr(self.lost_stage), self.n)


@pytest.mark.parametrize("n", [1, 4097, 65_536, 65_537, 700_001])
@pytest.mark.parametrize("precision", [ffi.FP64, ffi.MIXED, ffi.MIXED32])
@pytest.mark.parametrize("state_out", [0, 1])
def test_host_trace_of_library_vectors(n, precision, state_out):
    """Rays traced in place have the results of copied arrays; rays that are not
    traced and survivors' lost stages stay as they were."""
    surf = S.to_c(S.echelle(), E.spline_init).surfaces
    k = n // 3
    beams = [S.make_beam(0, k, 1, S.C1_RADIUS, (0.6, 0.6), 3, orders=(45, 1)),
             S.make_beam(k, n - k, 1, S.C1_RADIUS, (0.62, 0.62), 4, orders=(46, 1))]
    if k == 0:
        beams = beams[1:]
    source = E.generate(beams, n)
    rng = np.random.default_rng(n)
    flag, stage = (rng.random(n) < 0.95).astype(np.int8), rng.integers(0, 255, n).astype(np.uint8)
    results = []
    for rays in (PlainRays(n), E.PinnedRays(n)):
        for f in E.FIELDS:
            getattr(rays, f)[:] = getattr(source, f).cpu().numpy()
        rays.flag[:], rays.lost_stage[:] = flag, stage
        st, stats = E.trace_host(surf, beams, rays, E.opts(precision=precision, fixes=3, state_out=state_out))
        results.append([st, stats.ray_surfaces, stats.n_good] +
                       [getattr(rays, f).copy() for f in E.FIELDS + ("flag", "lost_stage")])
    for a, b in zip(*results):
        if isinstance(a, np.ndarray):
            assert np.array_equal(a.view(np.uint8), b.view(np.uint8))
        else:
            assert a == b


@pytest.mark.parametrize("precision", [ffi.FP64, ffi.MIXED, ffi.MIXED32])
@pytest.mark.parametrize("n", [33, 40_001])
def test_host_trace_is_the_same_after_a_plan_of_its_scheme(n, precision):
    """A plan compiles its scheme's kernel, which later calls of the scheme may take."""
    surf = S.to_c(S.echelle(), E.spline_init).surfaces
    beams = [S.make_beam(0, n, 1, S.C1_RADIUS, (0.61, 0.61), 5, orders=(45, 1))]
    source = E.generate(beams, n)
    o = E.opts(precision=precision, fixes=3, state_out=1)
    results = []
    for plan_first in (False, True):
        if plan_first:
            plan = E.Plan(surf, beams, o)
        rays = E.PinnedRays(n)
        for f in E.FIELDS + ("flag", "lost_stage"):
            getattr(rays, f)[:] = getattr(source, f).cpu().numpy()
        st, stats = E.trace_host(surf, beams, rays, o)
        results.append([np.array([st, stats.ray_surfaces, stats.n_good])] +
                       [getattr(rays, f).copy() for f in E.FIELDS + ("flag", "lost_stage")])
    del plan
    for a, b in zip(*results):
        assert np.array_equal(a.view(np.uint8), b.view(np.uint8))
