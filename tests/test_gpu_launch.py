"""The launch configuration a trace takes by itself (GPU tests): the same
results as an explicit one, at the ray counts where the default changes and
at ragged ones.
"""
import numpy as np
import pytest
import torch

from rt_b200 import engine as E
from rt_b200 import ffi, schemes as S

pytestmark = pytest.mark.gpu

ROWS = 148 * 32     # rows of 32 rays, one per resident warp


@pytest.mark.parametrize("precision", [ffi.FP64, ffi.MIXED, ffi.MIXED32])
@pytest.mark.parametrize("n", [1, 31, 33, 32 * 2 * ROWS - 1, 32 * 2 * ROWS, 32 * 8 * ROWS - 7, 32 * 8 * ROWS + 1])
def test_default_configuration_traces_every_ray_once(precision, n):
    surf = S.to_c(S.littrow_free_asphere(), E.spline_init).surfaces
    beams = [S.make_beam(0, n, 1, S.C0_RADIUS, (0.55, 0.55), 5)]
    ccd = S.ccd(S.C0_CCD)
    results = []
    for block, rpt in ((0, 0), (128, 8)):
        counts = torch.zeros(int(ccd.xdim) * int(ccd.ydim), dtype=torch.int32, device="cuda")
        outside = torch.zeros(1, dtype=torch.int64, device="cuda")
        torch.cuda.synchronize()
        rays = E.generate(beams, n)
        st, stats = E.trace(surf, beams, rays, E.opts(precision=precision, block=block, rpt=rpt, ccd=ccd,
                                                      counts=counts, n_outside=outside))
        ffi.check(st, "rtb_trace")
        good = int((rays.flag == 1).sum())
        assert stats.n_good == good and int(counts.sum()) + int(outside) == good
        results.append([getattr(rays, f).cpu().numpy() for f in E.FIELDS[:6] + ("flag", "lost_stage")] +
                       [counts.cpu().numpy()])
    for a, b in zip(*results):
        assert np.array_equal(a, b, equal_nan=a.dtype.kind == "f")
