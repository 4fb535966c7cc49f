"""Calls on library vectors, their statuses and results by themselves (GPU
tests): host traces against the CPU oracle, the arrays that are not traced in
place, and the drop-in calls' return codes and losses.
"""
import numpy as np
import pytest

import pyoracle as O
from rt_b200 import engine as E
from rt_b200 import ffi, schemes as S
from test_gpu_parity import assert_rays_equal
from test_gpu_vectors import PlainRays, Vectors, rays, stages

pytestmark = pytest.mark.gpu

ALL = E.FIELDS + ("flag", "lost_stage")


def fill(host, source):
    for f in ALL:
        getattr(host, f)[:] = getattr(source, f)
    return host


def test_host_trace_in_place_equals_the_oracle():
    beams = S.c1_beams(n_per_lambda=40)[:6]
    n = S.total_rays(beams)
    ora = O.generate(beams, n)
    mine = fill(E.PinnedRays(n), ora)
    st_o, stats_o, _ = O.trace(S.to_c(S.echelle(), O.spline_init).surfaces, beams, ora, fixes=3)
    st, stats = E.trace_host(S.to_c(S.echelle(), E.spline_init).surfaces, beams, mine, E.opts(fixes=3))
    assert st == st_o == ffi.OK
    assert (stats.ray_surfaces, stats.n_good) == (stats_o.ray_surfaces, stats_o.n_good) and 0 < stats.n_good < n
    assert_rays_equal(mine, ora)


@pytest.mark.parametrize("precision", [ffi.FP64, ffi.MIXED])
@pytest.mark.parametrize("why", ["gap", "no_lost_stage", "shared"])
def test_library_vectors_that_are_not_traced_in_place(precision, why):
    """Rays between the beams, no lost stages, two arrays in one: as ordinary arrays."""
    n, gap = 6000, 1000 if why == "gap" else 0
    surf = S.to_c(S.echelle(), E.spline_init).surfaces
    beams = [S.make_beam(0, n // 2 - gap, 1, S.C1_RADIUS, (0.6, 0.6), 3, orders=(45, 1)),
             S.make_beam(n // 2, n // 2, 1, S.C1_RADIUS, (0.62, 0.62), 4, orders=(46, 1))]
    source = E.generate(beams, n).to_host(PlainRays)
    if gap:
        for k, f in enumerate(E.FIELDS):
            getattr(source, f)[n // 2 - gap:n // 2] = 0.25 + k
    source.flag[:] = np.random.default_rng(1).random(n) < 0.9
    source.lost_stage[:] = 77
    results = []
    for h in (PlainRays(n), E.PinnedRays(n)):
        fill(h, source)
        if why == "shared":
            h.lost_stage = h.flag
        if why == "no_lost_stage":
            h.lost_stage = None
        st, stats = E.trace_host(surf, beams, h, E.opts(precision=precision, fixes=3, state_out=1))
        assert st == ffi.OK and 0 < stats.n_good <= int(source.flag.sum())
        results.append([stats.n_good] + [None if a is None else a.tobytes() for a in (getattr(h, f) for f in ALL)])
    assert results[0] == results[1]


@pytest.mark.parametrize("lost", [0.0, 0.01, 0.9])
def test_drop_in_calls_succeed_and_lose_the_rays_they_should(lost):
    n = 20_000
    plain = rays(n, lost)
    vec = Vectors(plain, 0)
    try:
        out = stages(vec.a, n)
        assert out[:7] == [ffi.OK] * 7
        marked = int((plain["flag"] == 0).sum())
        good = out[8]
        assert 0 < good <= n - marked and out[7] > 7                  # the aperture lost rays too
        assert vec.a["flag"][:good].all() and not vec.a["flag"][good:].any()
    finally:
        vec.free()
