"""The arrays rtb_adjoint_forward returns positions and flags in (GPU test):
aligned device arrays, device arrays at odd addresses, page-locked host arrays
and none get the same values.
"""
import ctypes as C

import pytest
import torch

from rt_b200 import engine as E
from rt_b200 import ffi, schemes as S

pytestmark = pytest.mark.gpu


def array(kind, n, dtype, offset):
    bytes_ = n * dtype.itemsize
    if kind == "host":
        return torch.zeros(bytes_, dtype=torch.uint8).pin_memory()
    return torch.zeros(bytes_ + 8, dtype=torch.uint8, device="cuda")[offset:offset + bytes_]


@pytest.mark.parametrize("n_per_lambda", [1, 33])
def test_forward_outputs_wherever_they_lie(n_per_lambda):
    beams = S.c4_beams(n_per_lambda=n_per_lambda)
    n = S.total_rays(beams)
    surf = S.to_c(S.littrow_free_asphere(), E.spline_init).surfaces
    adj = E.Adjoint(surf, S.c4_params(), beams, n, fixes=ffi.FIX_ASPHERE_ROOT)
    rays = E.generate(beams, n)
    results = []
    for kinds in (("device",) * 3, ("odd",) * 3, ("host",) * 3, ("device", "odd", "none")):
        out = [None if k == "none" else array(k, n, t, 1 if k == "odd" else 0)
               for k, t in zip(kinds, (torch.float64, torch.float64, torch.int8))]
        torch.cuda.synchronize()
        stats = ffi.TraceStats()
        st = E.lib().rtb_adjoint_forward(adj.h, None, C.byref(rays.struct()), *map(ffi.vptr, out), C.byref(stats), None)
        assert st == ffi.OK and 0 < stats.n_good <= n
        results.append([None if o is None else bytes(o.cpu().numpy()) for o in out])
    assert any(results[0][0]) and sum(results[0][2]) == stats.n_good
    for r in results[1:]:
        assert all(x is None or x == want for x, want in zip(r, results[0]))
