"""Performance cases: the calls a user of rt_b200 makes, over the sizes they
are made at.

  * trace    rays generated on the device and traced in place by one call, as
             rt_trace does for every wavelength range
  * plan     one run of a prepared plan: the ray sets traced again and again
             (instrument simulation, the benchmark's timed step)
  * host     a one-shot trace of arrays in host memory
  * dropin   the reference's engine calls, one per stage of one surface, on
             host arrays, as its Beam and Surface classes make them
  * adjoint  one design step: forward, merit and its seeds, gradient
  * results  what is made of traced rays: frame, file order, transmission and
             the list of wavelengths

Schemes, beams, cameras, parameters and quirk fixes are those of
rt_b200/schemes.py and bench.py (C0 the Littrow-free spectrograph, C1 the
echelle, C3 its batch of uneven beams, C4 the field-flattener design).

exact() traces the same rays with plain torch operations in 64 bits.
"""
import ctypes as C
import math

import numpy as np
import torch

from rt_b200 import engine as E
from rt_b200 import ffi
from rt_b200 import schemes as S

PRECISION = {"fp64": ffi.FP64, "mixed": ffi.MIXED, "mixed32": ffi.MIXED32}
TORIC_FIXES = ffi.FIX_TORIC_SIGN | ffi.FIX_TORIC_STEP    # as bench.py and the mixed engines
DESIGN_FIXES = TORIC_FIXES | ffi.FIX_ASPHERE_ROOT        # the converged model, for gradients
TARGET_WEIGHT = 10.0                                     # of the spot merit's centroid term, as bench.py
EXACT_RAYS = 30_000_000                                  # exact() declines beyond this


def listed():
    return [
        # The smallest call: C0 at the size of the smoke test and the golden
        # files; launches, allocations and copies of a one-shot trace.
        dict(name="trace_c0_small", kind="trace", scheme="c0", precision="fp64", orders=1, n_lambda=5,
             n_per_lambda=2000, frame=False, state_out=1),
        # An ordinary one-shot trace with the default engine: all echelle
        # orders, every ray's full state kept (the .dat files' content).
        dict(name="trace_c1_fp64", kind="trace", scheme="c1", precision="fp64", orders=31, n_lambda=64,
             n_per_lambda=1009, frame=False, state_out=1),
        # A one-shot trace for a picture only: mixed engine, detector frame.
        dict(name="trace_c4_mixed", kind="trace", scheme="c4", precision="mixed", orders=1, n_lambda=64,
             n_per_lambda=31250, frame=True, state_out=0),
        # The headline: 1e8 echelle rays a run, outputs at the tracing slots.
        dict(name="plan_c1_mixed", kind="plan", scheme="c1", precision="mixed", orders=31, n_lambda=64,
             n_per_lambda=50404, frame=True, out="slot"),
        # The bit-exact engine on the same instrument, outputs at the rays.
        dict(name="plan_c1_fp64", kind="plan", scheme="c1", precision="fp64", orders=31, n_lambda=64,
             n_per_lambda=10081, frame=True, out="index"),
        # A batch of 512 beams of uneven, odd sizes, fields and orders.
        dict(name="plan_c3_mixed", kind="plan", scheme="c3", precision="mixed", orders=512, n_lambda=1,
             n_per_lambda=250, frame=True, out="index"),
        # A small, repeated run with the FP32-state engine.
        dict(name="plan_c4_mixed32", kind="plan", scheme="c4", precision="mixed32", orders=1, n_lambda=64,
             n_per_lambda=3125, frame=True, out="index"),
        # End to end from host memory, X and Y back: what bench.py calls e2e.
        dict(name="host_c1_mixed", kind="host", scheme="c1", precision="mixed", orders=31, n_lambda=64,
             n_per_lambda=504, state_out=0),
        # The reference's programs over the drop-in calls: one C0 beam.
        dict(name="dropin_c0", kind="dropin", scheme="c0", orders=1, n_lambda=1, n_per_lambda=100_000),
        # A design step at production size: the spot merit's 24 derivatives.
        dict(name="adjoint_c4", kind="adjoint", scheme="c4", merit="spot", orders=1, n_lambda=64,
             n_per_lambda=31250),
        # A design step on few rays, as an optimiser's inner loop runs it,
        # with the resolution merit and a sensitivity along one direction.
        dict(name="adjoint_c4_small", kind="adjoint", scheme="c4", merit="resolution", orders=1, n_lambda=64,
             n_per_lambda=157),
        # Products of a traced echelle exposure.
        dict(name="results_c1", kind="results", scheme="c1", orders=31, n_lambda=64, n_per_lambda=2017),
    ]


def draw(rng):
    def size(lo, hi, per):  # rays spread over their logarithm, as rays per wavelength
        return max(1, round(math.exp(rng.uniform(math.log(lo), math.log(hi))) / per))

    kind = rng.choice(("trace", "trace", "plan", "plan", "plan", "host", "dropin", "adjoint", "adjoint", "results"))
    if kind == "dropin":
        return dict(kind=kind, scheme="c0", orders=1, n_lambda=1, n_per_lambda=size(1e3, 1e6, 1))
    scheme = "c4" if kind == "adjoint" else rng.choice(("c0", "c1", "c1", "c4"))
    if kind == "plan" and rng.random() < 0.25:
        return dict(kind=kind, scheme="c3", precision=rng.choice(tuple(PRECISION)), orders=rng.randint(16, 512),
                    n_lambda=1, n_per_lambda=rng.randint(20, 250), frame=rng.random() < 0.7,
                    out=rng.choice(("index", "slot")))
    orders = rng.randint(1, 31) if scheme == "c1" else 1
    n_lambda = rng.choice((5, 64, rng.randint(2, 300)))
    c = dict(kind=kind, scheme=scheme, orders=orders, n_lambda=n_lambda)
    if kind == "trace":
        c.update(precision=rng.choice(tuple(PRECISION)), frame=rng.random() < 0.5, state_out=rng.randint(0, 1),
                 n_per_lambda=size(1e4, 8e6, orders * n_lambda))
    elif kind == "plan":
        c.update(precision=rng.choice(tuple(PRECISION)), frame=rng.random() < 0.7, out=rng.choice(("index", "slot")),
                 n_per_lambda=size(1e5, 2e7, orders * n_lambda))
    elif kind == "host":
        c.update(precision=rng.choice(tuple(PRECISION)), state_out=rng.randint(0, 1),
                 n_per_lambda=size(1e4, 4e6, orders * n_lambda))
    elif kind == "adjoint":
        c.update(merit=rng.choice(("spot", "resolution")), n_per_lambda=max(8, size(1e4, 4e6, n_lambda)))
    else:
        c.update(n_per_lambda=size(1e5, 8e6, orders * n_lambda))
    return c


# ---------------------------------------------------------------------------
# what a program has before the call

def _specs(case):
    return {"c0": S.littrow_free, "c1": S.echelle, "c3": S.echelle, "c4": S.littrow_free_asphere}[case["scheme"]]()


def _beams(case, seed):
    n, nl, sch = case["n_per_lambda"], case["n_lambda"], case["scheme"]
    key = S.SEED + 7919 * (seed % 1_000_003)
    if sch == "c3":      # n_per_lambda: the batch's scale in thousandths
        beams = S.c3_beams(case["orders"], scale=n / 1000.0)
        for i, b in enumerate(beams):
            b.seed = key + i
        return beams
    if sch == "c1":
        beams, first = [], 0
        for i in range(case["orders"]):
            beams.append(S.make_beam(first, n, nl, S.C1_RADIUS, S.C1_LAMBDA, key + 1000 + i,
                                     orders=(S.C1_ORDERS[i], 1)))
            first += n * nl
        return beams
    return [S.make_beam(0, n, nl, S.C0_RADIUS, S.C0_LAMBDA if sch == "c0" else S.C4_LAMBDA, key)]


def _camera(case):
    return S.ccd(S.C1_CCD if case["scheme"] in ("c1", "c3") else S.C0_CCD)


def _stream():
    """torch's current stream for the library; the default stream by its own
    handle, since a null one means the library's private stream."""
    return C.c_void_p(torch.cuda.current_stream().cuda_stream or 1)


def _owned(view, owner):
    """A view of memory that `owner` frees, keeping it alive."""
    view.owner = owner
    return view


def _frame(ccd):
    return (torch.zeros(int(ccd.xdim) * int(ccd.ydim), dtype=torch.int32, device="cuda"),
            torch.zeros(1, dtype=torch.int64, device="cuda"))


def _lambdas(case):
    lo, hi = S.C4_LAMBDA if case["scheme"] == "c4" else S.C0_LAMBDA
    n = case["n_lambda"]
    return lo + (hi - lo) / max(1, n - 1) * np.arange(n)


def _theta(base, seed):
    """An optimiser's iterate: the design with parts in 1e7 changed."""
    return base * (1.0 + 1e-7 * np.random.default_rng(seed).standard_normal(len(base)))


def prepare(case, seed):
    kind = case["kind"]
    specs = _specs(case)
    st = {"case": case, "scheme": S.to_c(specs, E.spline_init), "beams": _beams(case, seed)}
    st["n"] = n = S.total_rays(st["beams"])
    st["surfaces"] = st["scheme"].surfaces
    ccd = st["ccd"] = _camera(case)
    frame = {}
    if case.get("frame") or kind == "results":
        st["counts"], st["outside"] = _frame(ccd)
        frame = dict(ccd=ccd, counts=st["counts"], n_outside=st["outside"])
    if kind == "trace":
        st["opts"] = E.opts(precision=PRECISION[case["precision"]], fixes=TORIC_FIXES, state_out=case["state_out"],
                            **frame)
    elif kind == "plan":
        out = ffi.OUT_SLOT if case["out"] == "slot" else ffi.OUT_INDEX
        st["plan"] = E.Plan(st["surfaces"], st["beams"],
                            E.opts(precision=PRECISION[case["precision"]], fixes=TORIC_FIXES, state_out=0,
                                   out_order=out, **frame))
        st["view"] = {k: _owned(v, st["plan"]) for k, v in E.device_view(st["plan"].rays()[1]).items()
                      if k != "lambda_"}
    elif kind == "host":
        st["opts"] = E.opts(precision=PRECISION[case["precision"]], fixes=TORIC_FIXES, state_out=case["state_out"])
        source = E.generate(st["beams"], n)
        st["rays"] = E.PinnedRays(n)
        changed = E.FIELDS[:6] if case["state_out"] else E.FIELDS[:2]
        for f in E.FIELDS + ("flag", "lost_stage"):
            torch.from_numpy(getattr(st["rays"], f)).copy_(getattr(source, f))
        st["source"] = [(torch.from_numpy(getattr(st["rays"], f)), getattr(source, f).cpu().pin_memory())
                        for f in changed + ("flag", "lost_stage")]
        st["result"] = {f: _owned(torch.from_numpy(getattr(st["rays"], f)), st["rays"])
                        for f in changed + ("flag", "lost_stage")}
    elif kind == "dropin":
        st["rays"] = E.PinnedRays(n)
        st["result"] = {f: _owned(torch.from_numpy(getattr(st["rays"], f)), st["rays"]) for f in E.FIELDS + ("flag",)}
        st["lib"] = E.lib()
        st["index"] = ffi.TableHolder(value=1.0)     # of the air on both sides
        st["angles"] = [np.array([a * 3.14159265359 / 180.0 for a in s.angles]) for s in specs]
        st["specs"] = specs
    elif kind == "adjoint":
        st["rays"] = E.generate(st["beams"], n)
        st["adjoint"] = E.Adjoint(st["surfaces"], S.c4_params(), st["beams"], n, fixes=DESIGN_FIXES)
        st["theta"] = _theta(st["adjoint"].theta(), seed)
        st["lambdas"] = _lambdas(case)
        st["target"] = S.c4_target_x(st["lambdas"])
        st["direction"] = np.random.default_rng(seed + 1).standard_normal(len(st["theta"])) * 1e-6
    else:
        st["rays"] = E.generate(st["beams"], n)
        status, stats = E.trace(st["surfaces"], st["beams"], st["rays"], E.opts(fixes=TORIC_FIXES))
        good = st["rays"].flag == 1
        st["lambda"] = torch.cat((st["rays"].lambda_[good], st["rays"].lambda_[~good]))  # a .dat file's order
        st["n_good"] = int(good.sum())
    torch.cuda.synchronize()
    return st


# ---------------------------------------------------------------------------
# one pass

def run(state):
    return {"trace": _run_trace, "plan": _run_plan, "host": _run_host, "dropin": _run_dropin,
            "adjoint": _run_adjoint, "results": _run_results}[state["case"]["kind"]](state)


def _stats(s):
    return {"ray_surfaces": s.ray_surfaces, "n_good": s.n_good}


def _run_trace(st):
    out = {}
    stream = _stream()
    if "counts" in st:
        st["counts"].zero_()
        st["outside"].zero_()
        out.update(counts=st["counts"], outside=st["outside"])
    rays = E.generate(st["beams"], st["n"], stream)
    status, stats = E.trace(st["surfaces"], st["beams"], rays, st["opts"], stream)
    fields = E.FIELDS[:6] if st["case"]["state_out"] else E.FIELDS[:2]
    out.update({f: getattr(rays, f) for f in fields + ("flag", "lost_stage")})
    return {**out, **_stats(stats)}


def _run_plan(st):
    out = dict(st["view"])
    if "counts" in st:
        st["counts"].zero_()
        st["outside"].zero_()
        out.update(counts=st["counts"], outside=st["outside"])
    st["plan"].run(_stream())
    return out


def _run_host(st):
    for mine, source in st["source"]:
        mine.copy_(source)
    status, stats = E.trace_host(st["surfaces"], st["beams"], st["rays"], st["opts"])
    return {**st["result"], **_stats(stats)}


def _run_dropin(st):
    L, h, n, beam = st["lib"], st["rays"], C.c_size_t(st["n"]), st["beams"][0]
    pos = [ffi.vptr(getattr(h, f)) for f in E.FIELDS[:3]]
    cos = [ffi.vptr(getattr(h, f)) for f in E.FIELDS[3:6]]
    lam, flag = ffi.vptr(h.lambda_), ffi.vptr(h.flag)
    # Beam's constructor: positions, parallel cosines, wavelengths, flags
    ffi.check(L.rtb_beam_random(beam.shape, beam.disk, beam.center, n, *pos, C.c_uint64(beam.seed), C.c_uint64(0)),
              "rtb_beam_random")
    h.cX[:] = 0.0
    h.cY[:] = 0.0
    h.cZ[:] = 1.0
    h.flag[:] = 1
    ffi.check(L.rtb_uniform_range_beam(n, beam.range, lam), "rtb_uniform_range_beam")
    n_good = C.c_size_t(st["n"])
    # Scheme::run's loop over the surfaces, on the good rays
    air = C.byref(st["index"].table)
    for s, c, angles in zip(st["specs"], st["scheme"].array, st["angles"]):
        ffi.check(L.rtb_beam_transform(n_good, ffi.vptr(angles), c.distance, *pos, *cos), "rtb_beam_transform")
        ffi.check(L.rtb_normalize(n_good, *cos), "rtb_normalize")
        bad = C.c_size_t(0)
        ffi.check(L.rtb_surface_intersection(c.cls, c.params, n_good, *pos, *cos, C.byref(bad), flag),
                  "rtb_surface_intersection")
        if bad.value:
            ffi.check(L.rtb_rearrange(C.byref(n_good), *pos, *cos, lam, flag), "rtb_rearrange")
        bad = C.c_size_t(0)
        ffi.check(L.rtb_apply_constrains(0, c.shape, c.size, c.center, n_good, *pos[:2], flag, C.byref(bad)),
                  "rtb_apply_constrains")
        if bad.value:
            ffi.check(L.rtb_rearrange(C.byref(n_good), *pos, *cos, lam, flag), "rtb_rearrange")
        if s.type == ffi.MIRROR:
            ffi.check(L.rtb_surface_reflection(c.cls, c.params, n_good, *pos, *cos), "rtb_surface_reflection")
        elif s.type == ffi.GRATING:
            bad = C.c_size_t(0)
            ffi.check(L.rtb_surface_diffration(c.cls, c.grating_type, c.params, C.c_long(c.order),
                                               C.c_double(c.gr_const), n_good, *pos, *cos, lam, air, air,
                                               C.byref(bad), flag), "rtb_surface_diffration")
            if bad.value:
                ffi.check(L.rtb_rearrange(C.byref(n_good), *pos, *cos, lam, flag), "rtb_rearrange")
        ffi.check(L.rtb_normalize(n_good, *cos), "rtb_normalize")
    return {**st["result"], "n_good": n_good.value}


def _run_adjoint(st):
    a = st["adjoint"]
    status, stats = a.forward(st["theta"], st["rays"])
    if st["case"]["merit"] == "spot":
        merit, gX, gY = a.spot_merit(st["target"], TARGET_WEIGHT)
    else:
        merit, gX, gY = a.resolution_merit(st["lambdas"])
    out = {"X": a.X, "Y": a.Y, "flag": a.flag, "merit": merit, "gX": gX, "gY": gY, "grad": a.backward(gX, gY)}
    if st["case"]["merit"] == "resolution":
        out["dX"], out["dY"] = a.jvp(st["direction"])
    return {**out, **_stats(stats)}


def _run_results(st):
    st["counts"].zero_()
    st["outside"].zero_()
    E.ccd_frame(st["rays"], st["ccd"], st["counts"], st["outside"])
    order = E.reference_order(st["beams"], 3 * len(st["surfaces"]), st["rays"])
    nl = st["case"]["n_lambda"]
    ll, ratio = E.loss_ratios(st["lambda"], st["n_good"], nl)
    return {"counts": st["counts"], "outside": st["outside"], "order": order, "ll": ll, "ratio": ratio,
            "lambdas": E.unique_lambdas(st["lambda"], st["n_good"], nl)}


# ---------------------------------------------------------------------------
# what a pass cannot do without

# FP64 operations per ray of the plain formulas (add, subtract, multiply,
# divide and square root one each): rt_b200/data/flops_c1.json for C1, its
# rows for the same kinds of surface summed for the others.
_FLOPS = {"c0": 320, "c1": 879, "c3": 879, "c4": 660}


def work(case):
    n = S.total_rays(_beams(case, 0))
    ccd = _camera(case)
    flops = _FLOPS[case["scheme"]] * n
    kind = case["kind"]
    pixels = 4 * int(ccd.xdim) * int(ccd.ydim)
    if kind == "trace":      # the rays written once, with their results
        per = 58
    elif kind == "plan":     # 57 bytes in, X, Y, flag and stage out
        per = 57 + 18
    elif kind == "host":     # over the link: 58 bytes in, the results out
        per = 58 + (50 if case["state_out"] else 18)
    elif kind == "dropin":   # 57 bytes of every ray returned
        per = 57
    elif kind == "adjoint":  # 57 bytes in, X, Y, flag and two seeds out; values, then their derivatives
        per, flops = 57 + 33, 4 * flops
        if case["merit"] == "resolution":
            per, flops = per + 16, flops * 1.5
    else:                    # X, Y, flag, stage and wavelength in, the order out
        per, flops = 26 + 4, 10 * n
    return {"bytes": per * n + (pixels if case.get("frame") or kind == "results" else 0), "flops": flops}


# ---------------------------------------------------------------------------
# the same rays in plain torch, 64 bits

def _philox(index, key):
    """Philox4x32-10 (Salmon et al., SC'11) with counter (index, 0, 0, 0)."""
    m = 0xFFFFFFFF
    c = [index & m, index >> 32, torch.zeros_like(index), torch.zeros_like(index)]
    k0, k1 = key & m, (key >> 32) & m
    for _ in range(10):
        p0, p1 = c[0] * 0xD2511F53, c[2] * 0xCD9E8D57
        c = [((p1 >> 32) & m) ^ c[1] ^ k0, p1 & m, ((p0 >> 32) & m) ^ c[3] ^ k1, p0 & m]
        k0, k1 = (k0 + 0x9E3779B9) & m, (k1 + 0xBB67AE85) & m
    return c


def _entrance(beam):
    """Positions, cosines and wavelengths of a generated beam."""
    i = torch.arange(beam.n_rays, dtype=torch.int64, device="cuda")
    r = _philox(i, beam.seed)
    u1, u2 = (((((h << 21) | (l >> 11)) + 1).double() * 2.0 ** -53) for h, l in ((r[0], r[1]), (r[2], r[3])))
    rad = (beam.disk[2] - beam.disk[1]) * u1.sqrt() + beam.disk[1]
    phi = 6.28318531 * u2
    x, y = rad * phi.cos() + beam.center[0], rad * phi.sin() + beam.center[1]
    c = torch.tensor([math.tan(beam.field[0]), math.tan(beam.field[1]), 1.0], dtype=torch.float64)
    c = c / c.norm()
    step = (beam.range[1] - beam.range[0]) / (beam.n_lambda - 1) if beam.n_lambda > 1 else 0.0
    one = torch.ones_like(x)
    return [x, y, one * beam.center[2]], [one * float(v) for v in c], beam.range[0] + (i % beam.n_lambda).double() * step


def _table(t, lam):
    """Natural cubic spline through a two-column table, or a number."""
    if isinstance(t, (int, float)):
        return torch.full_like(lam, float(t))
    x, y = (np.asarray(v, dtype=np.float64) for v in t)
    n, h = len(x), np.diff(x)
    a = np.zeros((n, n))
    b = np.zeros(n)
    a[0, 0] = a[-1, -1] = 1.0
    for i in range(1, n - 1):
        a[i, i - 1:i + 2] = h[i - 1] / 6.0, (h[i - 1] + h[i]) / 3.0, h[i] / 6.0
        b[i] = (y[i + 1] - y[i]) / h[i] - (y[i] - y[i - 1]) / h[i - 1]
    x, y, y2 = (torch.as_tensor(v, device=lam.device) for v in (x, y, np.linalg.solve(a, b)))
    i = torch.searchsorted(x, lam).clamp(1, n - 1)
    h = x[i] - x[i - 1]
    u, v = (x[i] - lam) / h, (lam - x[i - 1]) / h
    return u * y[i - 1] + v * y[i] + ((u ** 3 - u) * y2[i - 1] + (v ** 3 - v) * y2[i]) * h * h / 6.0


def _along(p, c, t):
    return [a + b * t for a, b in zip(p, c)]


def _unit(c):
    n = (c[0] * c[0] + c[1] * c[1] + c[2] * c[2]).sqrt()
    return [v / n for v in c]


class _Surface:
    """A surface's numbers, any of them replaced by torch scalars."""

    def __init__(self, spec):
        self.spec = spec
        p = list(spec.params)
        self.c, self.k, n = p[0], p[1], int(p[2])
        self.poly = p[3:3 + n]
        self.cR = p[3 + n] if spec.cls == ffi.TORIC else 0.0
        self.distance, self.angles = list(spec.distance), list(spec.angles)
        self.density = 1000.0 / spec.gr_const if spec.type == ffi.GRATING else None
        self.plane = spec.cls == ffi.PLANE or (spec.cls == ffi.CONIC and n == 0 and p[0] == 0)
        self.parabola = spec.cls == ffi.CONIC and n == 0 and p[1] == -1

    def set(self, kind, index, v):
        if kind == ffi.PARAM_CURVATURE:
            self.c = v
        elif kind == ffi.PARAM_CONIC:
            self.k = v
        elif kind == ffi.PARAM_POLY:
            self.poly[index] = v
        elif kind == ffi.PARAM_DISTANCE:
            self.distance[index] = v
        elif kind == ffi.PARAM_ANGLE:
            self.angles[index] = v
        else:
            self.density = v

    def enter(self, p, c, moved):
        """Translation, then rotations about y, x and z."""
        p = [a - d for a, d in zip(p, self.distance)]
        c = list(c)
        for (i, j), ang in zip(((0, 2), (1, 2), (0, 1)), self.angles):
            if not moved and not isinstance(ang, torch.Tensor) and ang == 0.0:
                continue
            a = torch.as_tensor(ang * (3.14159265359 / 180.0), dtype=torch.float64, device=p[0].device)
            s, k = a.sin(), a.cos()
            p[i], p[j] = p[i] * k - p[j] * s, p[i] * s + p[j] * k
            c[i], c[j] = c[i] * k - c[j] * s, c[i] * s + c[j] * k
        return p, c

    def sag(self, r2):
        """Height of an even asphere and its derivative with respect to r^2 / 2."""
        q = (1.0 - (self.k + 1.0) * self.c * self.c * r2).sqrt()
        z, d = self.c * r2 / (1.0 + q), self.c / q
        for i, a in enumerate(self.poly, 1):
            z, d = z + a * r2 ** i, d + 2.0 * i * a * r2 ** (i - 1)
        return z, d

    def toric(self, p):
        """The toric's function and its gradient's last two components' parts."""
        y2 = p[1] * p[1]
        q = (1.0 - (self.k + 1.0) * self.c * self.c * y2).sqrt()
        f = self.c * y2 / (1.0 + q)
        return p[2] - f - 0.5 * self.cR * (p[0] * p[0] + p[2] * p[2] - f * f), f, self.c * p[1] / q

    def meet(self, p, c, fix_root):
        """The point on the surface, and whether there is one."""
        if self.plane:
            t = -p[2] / c[2]
            at = _along(p, c, t)
            return [at[0], at[1], torch.zeros_like(at[2])], t >= 0
        k1 = self.k + 1.0
        if self.spec.cls == ffi.TORIC:
            return self._meet_toric(p, c)
        if not self.poly:
            a = k1 * c[2] * c[2] + c[0] * c[0] + c[1] * c[1]
            b = 2.0 * (k1 * p[2] * c[2] + p[0] * c[0] + p[1] * c[1] - c[2] / self.c)
            d = k1 * p[2] * p[2] + p[0] * p[0] + p[1] * p[1] - 2.0 * p[2] / self.c
            if self.parabola:
                t = -d / b
                return _along(p, c, t), t >= 0
            disc = b * b - 4.0 * a * d
            root = disc.clamp(min=0).sqrt()
            t = (-b - root if self.c > 0 else -b + root) / 2.0 / a
            return _along(p, c, t), disc >= 0
        return self._meet_asphere(p, c, fix_root)

    def _meet_asphere(self, p, c, fix_root):
        """Newton from the plane z = 0, each ray until a step is below 1e-7;
        the point of the last step, or without fix_root of the one before."""
        s0 = -p[2] / c[2]
        ok = s0 >= 0
        base = _along(p, c, s0)

        def step(s):
            at = [base[0] + s * c[0], base[1] + s * c[1], s * c[2]]
            z, d = self.sag(at[0] * at[0] + at[1] * at[1])
            return s - (at[2] - z) / (c[2] - d * (at[0] * c[0] + at[1] * c[1]))

        with torch.no_grad():
            s1 = torch.zeros_like(s0)
            s2 = step(s1)
            for _ in range(60):
                more = ok & ((s2 - s1).abs() >= 1e-7)
                if not bool(more.any()):
                    break
                s1 = torch.where(more, s2, s1)
                s2 = torch.where(more, step(s1), s2)
        s = step(s1) if fix_root else s1
        return [base[0] + s * c[0], base[1] + s * c[1], s * c[2]], ok

    def _meet_toric(self, p, c):
        t = -p[2] / c[2]
        ok = t >= 0
        go, last = ok.clone(), torch.zeros_like(t)
        for _ in range(60):
            f = self.toric(_along(p, c, t))[0]
            go = go & ((last - f).abs() > 1e-7)
            if not bool(go.any()):
                break
            g = self.toric(_along(p, c, t + f))[0]
            go = go & (g - f != 0)
            new = torch.where(go, t - f * f / torch.where(go, g - f, torch.ones_like(f)), t)
            last = torch.where(go, f, last)
            go, t = go & ((new - t).abs() >= 1e-7), new
        return _along(p, c, t), ok

    def inside(self, p):
        s = self.spec
        x, y = p[0] - s.center[0], p[1] - s.center[1]
        if s.shape == ffi.CIRCLE:
            return x * x + y * y <= s.size[0] ** 2
        return (x.abs() <= s.size[0] / 2.0) & (y.abs() <= s.size[1] / 2.0)

    def normal(self, p):
        """Gradient of the surface function."""
        if self.spec.cls == ffi.TORIC:
            _, f, df = self.toric(p)
            return [-self.cR * p[0], (self.cR * f - 1.0) * df, 1.0 - self.cR * p[2]]
        d = self.sag(p[0] * p[0] + p[1] * p[1])[1]
        return [-d * p[0], -d * p[1], torch.ones_like(p[0])]

    def act(self, p, c, lam, order):
        s = self.spec
        if s.type == ffi.MIRROR:
            if self.plane:
                return [c[0], c[1], -c[2]], torch.ones_like(lam, dtype=torch.bool)
            g = self.normal(p)
            a = 2.0 * sum(u * v for u, v in zip(c, g)) / sum(v * v for v in g)
            return [u - a * v for u, v in zip(c, g)], torch.ones_like(lam, dtype=torch.bool)
        if s.type == ffi.LENS:
            mu = _table(s.n1, lam) / _table(s.n2, lam)
            g = self.normal(p)
            gg = sum(v * v for v in g)
            a = mu * sum(u * v for u, v in zip(c, g)) / gg
            b = a * a - (mu * mu - 1.0) / gg
            f = b.clamp(min=0).sqrt() - a
            return [mu * u + f * v for u, v in zip(c, g)], b >= 0
        if s.type == ffi.GRATING:     # plane, reflective
            w = order * lam / _table(s.n2, lam) * (self.density / 1000.0)
            b = c[2] * c[2] - w * w + 2.0 * w * c[0]
            return [c[0] - w, c[1], -b.clamp(min=0).sqrt()], b >= 0
        return c, torch.ones_like(lam, dtype=torch.bool)


def _traced(surfaces, beam, fix_root=False, moved=False):
    """One beam through the surfaces; a lost ray keeps the state it was lost with."""
    p, c, lam = _entrance(beam)
    good = torch.ones_like(lam, dtype=torch.bool)
    grating = 0
    for s in surfaces:
        q, e = s.enter(p, c, moved)
        e = _unit(e)
        keep = lambda new, old, m: [torch.where(m, a, b) for a, b in zip(new, old)]  # noqa: E731
        p, c = keep(q, p, good), keep(e, c, good)
        at, ok = s.meet(p, c, fix_root)
        p = keep(at, p, good & ok)
        good = good & ok & s.inside(p)
        order = s.spec.order
        if s.spec.type == ffi.GRATING:
            order = beam.orders[grating] if beam.n_orders else order
            grating += 1
        d, ok = s.act(p, c, lam, order)
        good = good & ok
        c = keep(_unit(d), c, good)
    return p, c, lam, good


def _exact_rays(case, seed):
    surfaces = [_Surface(s) for s in _specs(case)]
    parts = [_traced(surfaces, b) for b in _beams(case, seed)]
    join = lambda vs: torch.cat(list(vs))  # noqa: E731
    out = {f: join(q[0][i] for q in parts) for i, f in enumerate(E.FIELDS[:3])}
    out.update({f: join(q[1][i] for q in parts) for i, f in enumerate(E.FIELDS[3:6])})
    return out, join(q[2] for q in parts), join(q[3] for q in parts)


def _exact_dropin(case, seed):
    """C0's beam with the reference's reordering: each stage swaps the lost
    rays among the first ones with the last good ones."""
    beam = _beams(case, seed)[0]
    p, c, _ = _entrance(beam)
    n = beam.n_rays
    lam = beam.range[0] + torch.arange(n, dtype=torch.float64, device="cuda") * ((beam.range[1] - beam.range[0]) / max(1, n - 1))
    v = torch.stack(p + c + [lam])
    m = n

    def rearrange(good):
        nonlocal m, v
        kept = int(good.sum())
        front = torch.nonzero(~good[:kept]).flatten()
        back = torch.nonzero(good[kept:]).flatten().flip(0) + kept
        perm = torch.arange(v.shape[1], device="cuda")
        perm[front], perm[back] = back, front
        v, m = v[:, perm], kept

    for s in (_Surface(x) for x in _specs(case)):
        q, e = s.enter(list(v[:3, :m]), list(v[3:6, :m]), False)
        v[:6, :m] = torch.stack(q + _unit(e))
        at, ok = s.meet(list(v[:3, :m]), list(v[3:6, :m]), False)
        v[:3, :m] = torch.where(ok, torch.stack(at), v[:3, :m])
        rearrange(ok)
        rearrange(s.inside(v[:3, :m]))
        d, ok = s.act(list(v[:3, :m]), list(v[3:6, :m]), v[6, :m], s.spec.order)
        v[3:6, :m] = torch.where(ok, torch.stack(_unit(d)), v[3:6, :m])
        rearrange(ok)
    return {f: v[i] for i, f in enumerate(E.FIELDS)}


def _merit(case, x, y, good, lambdas):
    """The spot or the resolution merit of one composite beam."""
    nl = case["n_lambda"]
    x, y, w = x.view(-1, nl), y.view(-1, nl), good.view(-1, nl).double()
    n = w.sum(0)
    some = n > 0
    n1 = n.clamp(min=1)
    cx, cy = (x * w).sum(0) / n1, (y * w).sum(0) / n1
    dx, dy = (x - cx) * w, (y - cy) * w
    if case["merit"] == "spot":
        target = torch.as_tensor(S.c4_target_x(lambdas), device=x.device)
        rms = ((dx * dx + dy * dy).sum(0) / n1).sqrt()
        return torch.where(some, rms + TARGET_WEIGHT * (cx - target) ** 2, torch.zeros_like(rms)).sum()
    width = ((dx * dx).sum(0) / n1).sqrt()
    lam = torch.as_tensor(lambdas, device=x.device)
    pair = some[1:] & some[:-1]
    gap = (cx[1:] - cx[:-1]).abs()
    each = (width[1:] + width[:-1]) / 2.0 * (lam[1:] - lam[:-1]).abs() / gap / ((lam[1:] + lam[:-1]) / 2.0)
    return torch.where(pair, each, torch.zeros_like(each)).sum()


def _exact_adjoint(case, seed):
    specs = _specs(case)
    beam = _beams(case, seed)[0]
    params = S.c4_params()
    base = []
    for k, kind, i in params:
        s = specs[k]
        base.append({ffi.PARAM_CURVATURE: lambda: s.params[0], ffi.PARAM_CONIC: lambda: s.params[1],
                     ffi.PARAM_POLY: lambda: s.params[3 + i], ffi.PARAM_DISTANCE: lambda: s.distance[i],
                     ffi.PARAM_ANGLE: lambda: s.angles[i], ffi.PARAM_GROOVE_DENSITY: lambda: 1000.0 / s.gr_const}[kind]())
    theta = _theta(np.array(base), seed)
    lambdas = _lambdas(case)

    def forward(values):
        surfaces = [_Surface(s) for s in specs]
        for (k, kind, i), v in zip(params, values):
            surfaces[k].set(kind, i, v)
        p, _, _, good = _traced(surfaces, beam, fix_root=True, moved=True)
        return p[0], p[1], good

    values = [torch.tensor(v, dtype=torch.float64, device="cuda", requires_grad=True) for v in theta]
    x, y, good = forward(values)
    xs, ys = x.detach().requires_grad_(), y.detach().requires_grad_()
    m = _merit(case, xs, ys, good, lambdas)
    gx, gy = (torch.where(good, g, torch.zeros_like(g)) if g is not None else torch.zeros_like(x)
              for g in torch.autograd.grad(m, (xs, ys), allow_unused=True))
    grad = torch.autograd.grad((x, y), values, (gx, gy))
    out = {"X": x.detach(), "Y": y.detach(), "flag": None, "merit": float(m), "gX": gx, "gY": gy,
           "grad": torch.stack(grad)}
    if case["merit"] == "resolution":
        direction = np.random.default_rng(seed + 1).standard_normal(len(theta)) * 1e-6
        with torch.autograd.forward_ad.dual_level():
            dual = [torch.autograd.forward_ad.make_dual(v.detach(), torch.full_like(v.detach(), d))
                    for v, d in zip(values, direction)]
            x, y, good = forward(dual)
            out["dX"], out["dY"] = (torch.where(good, t.clone(), torch.zeros_like(t)) for t in
                                    (torch.autograd.forward_ad.unpack_dual(v).tangent for v in (x, y)))
    return out


def exact(case, seed):
    kind = case["kind"]
    n = S.total_rays(_beams(case, seed))
    if n > EXACT_RAYS or case.get("out") == "slot":    # too long; slots are the plan's own order
        return None
    if kind == "dropin":
        return _exact_dropin(case, seed)
    if kind == "adjoint":    # fewer rays: the backward pass keeps every intermediate
        return _exact_adjoint(case, seed) if n <= 2_100_000 else None
    rays, lam, good = _exact_rays(case, seed)
    if kind == "results":
        value, count = torch.unique(lam, return_counts=True)
        if len(value) != case["n_lambda"]:
            return None
        kept = torch.stack([(lam[good] == v).sum() for v in value])
        first = sorted((int(torch.nonzero(lam[good] == v)[0]), i) for i, v in enumerate(value) if kept[i])
        return {"ll": value, "ratio": kept.double() / count.double(), "lambdas": value[[i for _, i in first]]}
    if case["precision"] != "fp64" and case["scheme"] in ("c1", "c3"):
        return None     # two thirds are lost, and a mixed engine leaves those where it stopped following them
    full = case.get("state_out", 0)
    return {f: rays[f] for f in (E.FIELDS[:6] if full else E.FIELDS[:2])}
