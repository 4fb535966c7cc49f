"""The launch configuration a mixed trace takes by itself where the number of
surfaces decides it (GPU test): every ray traced once, with the results of an
explicit configuration.
"""
import numpy as np
import pytest
import torch

from rt_b200 import engine as E
from rt_b200 import ffi, schemes as S

pytestmark = pytest.mark.gpu

ROWS = 148 * 32     # rows of 32 rays, one per resident warp


@pytest.mark.parametrize("precision", [ffi.MIXED, ffi.MIXED32])
@pytest.mark.parametrize("surfaces", [9, 10, 32])
@pytest.mark.parametrize("n", [32 * 2 * ROWS - 1, 32 * 2 * ROWS, 32 * 8 * ROWS - 7, 32 * 8 * ROWS + 33])
def test_default_configuration_traces_every_ray_once(precision, surfaces, n):
    idle = S.SurfaceSpec(ffi.AUX_CLASS, ffi.AUX_TYPE, distance=(0.0, 0.0, 0.0))
    specs = S.littrow_free()
    surf = S.to_c([idle] * (surfaces - len(specs)) + specs, E.spline_init).surfaces
    beams = [S.make_beam(0, n, 1, S.C0_RADIUS, (0.55, 0.55), 5)]
    results = []
    for block, rpt in ((0, 0), (128, 7)):
        plan = E.Plan(surf, beams, E.opts(precision=precision, block=block, rpt=rpt, state_out=0))
        plan.run()
        st, stats = plan.result()
        assert st == ffi.OK
        out = E.device_view(plan.rays()[1])
        assert stats.n_good == int((out["flag"] == 1).sum()) > 0
        if not rpt:
            assert plan.config()[1] == (1 if n < 64 * ROWS else 2 if n < 256 * ROWS or surfaces >= 10 else 4)
        results.append([out[f].clone() for f in ("flag", "lost_stage", "X", "Y")])
        torch.cuda.synchronize()
        plan.destroy()
    for a, b in zip(*results):
        assert np.array_equal(a.cpu().numpy(), b.cpu().numpy(), equal_nan=a.dtype == torch.float64)
