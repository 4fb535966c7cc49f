"""The fused kernels for any scheme, for a scheme's structure and for a scheme
with its values (GPU tests), whose tables lie at different places in shared
memory, on schemes of the fewest to the most surfaces: the same rays.
"""
import numpy as np
import pytest

from rt_b200 import engine as E
from rt_b200 import ffi, schemes as S

pytestmark = pytest.mark.gpu

# FP64: the same operations.  Mixed: the same operations but for contractions,
# a few units in the last place of 64 or 32 bits at 1e2 mm through 7 surfaces;
# a table read from another place shifts rays by far more.
TOLERANCE_MM = {ffi.FP64: 0.0, ffi.MIXED: 1e-9, ffi.MIXED32: 1e-3}


def scheme(n):
    """C1 behind Aux surfaces that do nothing, or its last surfaces."""
    specs = S.echelle()
    idle = [S.SurfaceSpec(ffi.AUX_CLASS, ffi.AUX_TYPE, distance=(0.0, 0.0, 0.0)) for _ in range(max(0, n - len(specs)))]
    return idle + specs if idle else specs[len(specs) - n:]


@pytest.mark.parametrize("precision", list(TOLERANCE_MM))
@pytest.mark.parametrize("surfaces", [1, 2, 7, 31, 32])
@pytest.mark.parametrize("order", [ffi.ORDER_INDEX, ffi.ORDER_COHERENT])
def test_kernels_agree_whatever_the_number_of_surfaces(monkeypatch, precision, surfaces, order):
    surf = S.to_c(scheme(surfaces), E.spline_init).surfaces
    n = 5000
    beams = [S.make_beam(0, n, 4, 2.0, (0.55, 0.60), 3, orders=(45, 1) if surfaces >= 7 else ())]
    n = S.total_rays(beams)
    results = []
    for how in ("0", "structure", "1"):
        monkeypatch.setenv("RTB_SPECIALIZE", how)
        o = E.opts(precision=precision, fixes=3, state_out=1)
        o.ray_order = order
        plan = E.Plan(surf, beams, o)
        plan.run()
        st, stats = plan.result()
        assert st == ffi.OK and stats.n_good > 0 and plan.specialized()[0] == (how != "0")
        out = E.device_view(plan.rays()[1])
        results.append([out[f].cpu().numpy() for f in ("flag", "X", "Y")])
        plan.destroy()
    rays = E.generate(beams, n)
    monkeypatch.setenv("RTB_SPECIALIZE", "0")
    st, stats = E.trace(surf, beams, rays, E.opts(precision=precision, fixes=3))
    assert st == ffi.OK
    results.append([rays.flag.cpu().numpy(), rays.X.cpu().numpy(), rays.Y.cpu().numpy()])
    flag, X, Y = results[0]
    for r in results[1:]:
        assert np.array_equal(r[0], flag)
        for a, b in zip(r[1:], (X, Y)):
            assert np.abs(a - b)[flag == 1].max() <= TOLERANCE_MM[precision]
