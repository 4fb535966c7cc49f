"""The replay of Rearrange over a whole trace (rtb_reference_order) against
the reference's two pointers, and the wavelength reductions where the number
of distinct values decides the path (GPU tests).
"""
import numpy as np
import pytest
import torch

import pyoracle as O
from rt_b200 import engine as E
from rt_b200 import ffi, schemes as S

pytestmark = pytest.mark.gpu


def rearranged(stage, n_stages):
    """Beam::Rearrange after each stage (beam.cpp:574-598), literally."""
    order, good = np.arange(len(stage)), len(stage)
    for s in range(n_stages):
        lost = stage[order[:good]] == s
        i, j = 0, good - 1
        while True:
            while i < good and not lost[i]:
                i += 1
            while j >= 0 and lost[j]:
                j -= 1
            if i >= j:
                break
            order[i], order[j] = order[j], order[i]
            lost[i], lost[j] = lost[j], lost[i]
            i, j = i + 1, j - 1
        good -= int(lost.sum())
    return order


SIZES = [[1], [2], [15, 16, 17], [4095, 4096, 4097], [0, 5, 0, 8193], [40_000], [700] * 33, [9000, 1, 30_001, 0]]


@pytest.mark.parametrize("sizes", SIZES, ids=str)
@pytest.mark.parametrize("losses", ["none", "few", "most", "all", "back", "front"])
@pytest.mark.parametrize("gap", [0, 3])
def test_order_equals_two_pointers(sizes, losses, gap):
    rng = np.random.default_rng(len(sizes) + 7)
    n_stages = 96
    first, beams = gap, []
    for k in sizes:
        beams.append(S.make_beam(first, k, 1, 1.0, (0.5, 0.5), 1))
        first += k + gap
    n = first + gap
    stage = np.full(n, ffi.NOT_LOST, np.uint8)
    for b, k in zip(beams, sizes):
        p = {"none": 0.0, "few": 0.02, "most": 0.97, "all": 1.0, "back": 0.5, "front": 0.5}[losses]
        hit = rng.random(k) < p
        if losses == "back":
            hit[: k // 2] = False
        if losses == "front":
            hit[k // 2:] = False
        s = np.where(hit, rng.choice([0, 1, 7, 31, 32, 64, 95], k), ffi.NOT_LOST)
        stage[b.first_ray:b.first_ray + k] = s
    rays = E.DeviceRays(n)
    rays.lost_stage.copy_(torch.from_numpy(stage))
    order = E.reference_order(beams, n_stages, rays).cpu().numpy()
    seen = np.zeros(n, bool)
    for b, k in zip(beams, sizes):
        a = int(b.first_ray)
        assert np.array_equal(order[a:a + k], rearranged(stage[a:a + k], n_stages))
        seen[a:a + k] = True
    starts = np.array([b.first_ray for b in beams])
    for i in np.flatnonzero(~seen):      # between the beams: relative to the beam before
        base = starts[max(0, np.searchsorted(starts, i, side="right") - 1)]
        assert np.uint32(order[i]) == np.uint32((int(i) - int(base)) % 2 ** 32)


def bits_equal(a, b):
    a, b = np.asarray(a, np.float64), np.asarray(b, np.float64)
    return len(a) == len(b) and bool(np.all((a.view(np.int64) == b.view(np.int64)) | (np.isnan(a) & np.isnan(b))))


@pytest.mark.parametrize("values", [1, 2, 64, 300, 1023, 1024, 1025, 3000])
@pytest.mark.parametrize("n", [3001, 100_003])
def test_reductions_around_the_limit_of_distinct_values(values, n):
    rng = np.random.default_rng(values)
    pool = rng.uniform(-0.9, 0.9, values)
    lam = np.concatenate([pool, rng.choice(pool, n - values)]) if n >= values else pool
    rng.shuffle(lam)
    dev = torch.as_tensor(lam, device="cuda")
    for n_good in (0, 1, n // 3, n):
        assert bits_equal(E.unique_lambdas(dev, n_good, 4000), O.unique_lambdas(lam, n_good, 0)[:4000] if n_good else [])
        assert bits_equal(E.unique_lambdas(dev, n_good, 5), O.unique_lambdas(lam, n_good, 0)[:5] if n_good else [])
        for n_lambda in (1, values, 2 * n):
            got, want = E.loss_ratios(dev, n_good, n_lambda), O.loss_ratios(lam, n_good, n_lambda)
            assert bits_equal(got[0], want[0]) and bits_equal(got[1], want[1]), (n_good, n_lambda)


def test_reductions_with_zeros_nans_and_infinities():
    lam = np.array([0.5, -0.0, 0.0, np.inf, 0.5, -np.inf, 0.25, np.inf, -0.5, 0.0] * 50)
    for a in (lam, np.where(lam == 0, 0.75, lam)):
        dev = torch.as_tensor(a, device="cuda")
        got, want = E.loss_ratios(dev, 300, 6), O.loss_ratios(a, 300, 6)
        assert np.array_equal(got[0], want[0]) and bits_equal(got[1], want[1])    # of equal zeros either may come first
        assert bits_equal(E.unique_lambdas(dev, 300, 50), O.unique_lambdas(a, 300, 0)[:50])
    a[7] = np.nan
    assert bits_equal(E.unique_lambdas(torch.as_tensor(a, device="cuda"), 300, 50), O.unique_lambdas(a, 300, 0)[:50])
