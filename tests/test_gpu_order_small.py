"""rtb_reference_order where the size of a beam decides how it is replayed, and
with very many beams (GPU tests): the two-pointer order, and scratch in
proportion to the rays whatever the beams' sizes.
"""
import numpy as np
import pytest
import torch

from rt_b200 import engine as E
from rt_b200 import ffi, schemes as S
from test_gpu_order import rearranged

pytestmark = pytest.mark.gpu

LOSSY = [0, 1, 7, 31, 32, 64, 95]


def beams_of(sizes, gap=0):
    beams, first = [], gap
    for k in sizes:
        beams.append(S.make_beam(first, int(k), 1, 1.0, (0.5, 0.5), 1))
        first += int(k) + gap
    return beams, first


@pytest.mark.parametrize("sizes", [[511], [512], [513], [31, 32, 33, 64, 511, 512, 513, 4096],
                                   [512, 20_000, 1, 0, 513, 512], [3] * 700 + [600] * 9 + [511] * 40, [0, 0, 5]], ids=len)
@pytest.mark.parametrize("lost", [0.0, 0.03, 0.5, 0.97, 1.0])
@pytest.mark.parametrize("gap", [0, 2])
def test_order_equals_two_pointers_around_the_line(sizes, lost, gap):
    rng = np.random.default_rng(int(100 * lost) + len(sizes))
    beams, n = beams_of(sizes, gap)
    # stages beyond the scheme's lose no ray
    stage = np.where(rng.random(n) < lost, rng.choice(LOSSY, n), rng.choice([96, ffi.NOT_LOST], n)).astype(np.uint8)
    rays = E.DeviceRays(n)
    rays.lost_stage.copy_(torch.from_numpy(stage))
    order = E.reference_order(beams, 96, rays).cpu().numpy().view(np.uint32)
    inside = np.zeros(n, bool)
    for b, k in zip(beams, sizes):
        a = int(b.first_ray)
        assert np.array_equal(order[a:a + k], rearranged(stage[a:a + k], 96)), k
        inside[a:a + k] = True
    starts = np.array([b.first_ray for b in beams], np.int64)
    for i in np.flatnonzero(~inside):
        assert order[i] == np.uint32((i - starts[max(0, np.searchsorted(starts, i, side="right") - 1)]) % 2 ** 32)


def test_scratch_follows_the_rays():
    """3e5 beams of three rays: their scratch is megabytes, not a tile per beam."""
    k, count = 3, 300_000
    beams, n = beams_of([k] * count)
    rng = np.random.default_rng(2)
    stage = np.where(rng.random(n) < 0.5, rng.choice([2, 5], n), ffi.NOT_LOST).astype(np.uint8)
    rays = E.DeviceRays(n)
    rays.lost_stage.copy_(torch.from_numpy(stage))
    torch.cuda.synchronize()
    free = torch.cuda.mem_get_info()[0]
    order = E.reference_order(beams, 21, rays).cpu().numpy()
    assert free - torch.cuda.mem_get_info()[0] < 200 << 20
    s = stage.reshape(count, k)
    for c in rng.integers(0, count, 2000):
        assert np.array_equal(order[3 * c:3 * c + 3], rearranged(s[c], 21))
