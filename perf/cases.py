"""The work users of this framework have it do, as timed cases.

A case is a dict of plain values.  `prepare` makes what a user's program holds
before the call (grids, sources, an engine with its grid class), `run` makes
one pass through the public entry points: the batched engine, the forecast
server, the reference's C ABI (whole forecasts through `drive`, or the Fortran
driver's own sequence of calls), the allocation-free step, and the on-device
fault source.  Sizes are the framework's own workloads (361x301 local grid,
1201x1001 regional ensemble grid with a 601x501 child, 2401x2001 basin grid,
the 481x401 / 961x801 / 1921x1601 request grids) and odd sizes between.
"""
from __future__ import annotations

import ctypes as C
import math
import os
import sys

import numpy as np
import torch

_PKG = os.path.join(os.getcwd(), "gpu-comcot_b200")
if _PKG not in sys.path:
    sys.path.insert(0, _PKG)
os.environ.setdefault("GCOMCOT_QUIET", "1")  # the C ABI's own messages per layer

from comcot_b200 import _lib, synth  # noqa: E402
from comcot_b200.abi import ReferenceSession  # noqa: E402
from comcot_b200.engine import Engine  # noqa: E402
from comcot_b200.serving import ForecastServer, Request  # noqa: E402

F32 = np.float32
BUDGET = 40 << 30


def listed():
    return [
        # one step of one local grid by a code that owns its device memory: launch latency
        {"name": "step-local", "kind": "step", "nx": 361, "ny": 301, "grids": 1},
        # one step of a batch of regional grids (a warning centre's scenarios) the same way
        {"name": "step-batch", "kind": "step", "nx": 1201, "ny": 1001, "grids": 6},
        # a two-hour local forecast on the smallest configured grid, a chain of short launches
        {"name": "forecast-local", "kind": "forecast", "nx": 361, "ny": 301, "dx": 2.0, "dt": 2.0, "steps": 3600,
         "gauges": 8, "members": 1},
        # an hour on the headline basin grid: OPEN on four sides, max-eta, arrival, 32 gauges
        {"name": "forecast-basin", "kind": "forecast", "nx": 2401, "ny": 2001, "dx": 1.0, "dt": 1.0, "steps": 3600,
         "gauges": 32, "members": 1},
        # an ensemble of sources over one shared regional bathymetry
        {"name": "ensemble-regional", "kind": "forecast", "nx": 1201, "ny": 1001, "dx": 2.0, "dt": 2.0, "steps": 1200,
         "gauges": 0, "members": 24},
        # a regional grid with a nonlinear wet/dry shelf child (ratio 5, one sub-step per step)
        {"name": "nested-shelf", "kind": "nested", "nx": 1201, "ny": 1001, "cw": 120, "ch": 100, "ratio": 5, "sub": 1,
         "steps": 1200, "gauges": 8},
        # a request-size grid whose child takes three sub-steps per step (edge forecast, JNZ at the middle one)
        {"name": "nested-substeps", "kind": "nested", "nx": 481, "ny": 401, "cw": 61, "ch": 47, "ratio": 3, "sub": 3,
         "steps": 600, "gauges": 4},
        # the Fortran driver's whole run through the C ABI: layer upload, drive, fields read back
        {"name": "abi-drive", "kind": "drive", "nx": 961, "ny": 801, "laygov": 0, "steps": 1800, "gauges": 16},
        # the same sequence call by call, every gauge returned every step
        {"name": "abi-calls", "kind": "calls", "nx": 481, "ny": 401, "laygov": 0, "steps": 300, "gauges": 8},
        # a nonlinear spherical outer layer with Manning friction (CONMASS_S / CONMOME_S), an odd size
        {"name": "abi-nonlinear", "kind": "drive", "nx": 723, "ny": 603, "laygov": 1, "steps": 300, "gauges": 4},
        # a burst of mixed forecast requests (three grid sizes, some nested) through the server
        {"name": "serve-burst", "kind": "serve", "requests": 8, "steps": 900, "scale": 1.0},
        # a finite-fault source of 24 sub-faults turned into surface and depth changes
        {"name": "fault-source", "kind": "fault", "nx": 961, "ny": 801, "faults": 24},
    ]


def _log(rng, lo, hi):
    """a whole number spread over the logarithm of [lo, hi]"""
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["step", "step", "forecast", "forecast", "ensemble", "nested", "nested", "drive", "drive",
                       "calls", "serve", "fault"])
    if kind == "step":
        return {"kind": kind, "nx": _log(rng, 150, 1921), "ny": _log(rng, 130, 1601), "grids": _log(rng, 1, 6)}
    if kind in ("forecast", "ensemble"):
        many = kind == "ensemble"
        return {"kind": "forecast", "nx": _log(rng, 200, 1201 if many else 2401),
                "ny": _log(rng, 180, 1001 if many else 2001), "dx": rng.choice([1.0, 2.0]), "dt": 1.0,
                "steps": _log(rng, 200, 1200), "gauges": rng.choice([0, 5, 16, 33]),
                "members": _log(rng, 2, 24) if many else 1}
    if kind == "nested":
        nx, ny = _log(rng, 301, 1201), _log(rng, 251, 1001)
        return {"kind": kind, "nx": nx, "ny": ny, "cw": rng.randint(30, 60 if nx < 601 else 120),
                "ch": rng.randint(30, 60 if ny < 501 else 100), "ratio": rng.choice([2, 3, 5]),
                "sub": rng.choice([1, 1, 2, 3]), "steps": _log(rng, 100, 600), "gauges": rng.choice([0, 4, 12])}
    if kind == "drive":
        return {"kind": kind, "nx": _log(rng, 200, 1201), "ny": _log(rng, 180, 1001),
                "laygov": rng.choice([0, 0, 1, 2]), "steps": _log(rng, 60, 600), "gauges": rng.choice([0, 4, 16])}
    if kind == "calls":
        return {"kind": kind, "nx": _log(rng, 200, 961), "ny": _log(rng, 180, 801), "laygov": 0,
                "steps": _log(rng, 50, 300), "gauges": rng.choice([1, 8, 32])}
    if kind == "serve":
        return {"kind": kind, "requests": rng.randint(2, 8), "steps": _log(rng, 150, 900),
                "scale": rng.choice([0.5, 0.75, 1.0])}
    return {"kind": kind, "nx": _log(rng, 200, 1201), "ny": _log(rng, 180, 1001), "faults": _log(rng, 1, 24)}


# ---------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------
def _single(case, seed, laygov=0, gauges=0):
    """seeded bathymetry (basin, seamounts, shelf, land strip) with a dipole source"""
    nx, ny = case["nx"], case["ny"]
    return synth.single_layer_case("case", nx, ny, case.get("dx", 2.0), case.get("dt", 2.0), case.get("steps", 1),
                                   seed=seed, n_seamounts=max(4, nx // 40), shelf_cols=max(4, nx // 15),
                                   land_cols=max(2, nx // 40), source="dipole", ngauges=gauges, laygov=laygov)


def _nested(case, seed):
    """a parent with an east-side shelf window under a nonlinear Cartesian child"""
    nx, ny, cw, ch = case["nx"], case["ny"], case["cw"], case["ch"]
    i0, j0 = nx - cw - 24, (ny - ch) // 2
    c = synth.nested_case("case", nx, ny, 2.0, 2.0, [i0, i0 + cw - 1, j0, j0 + ch - 1], case["ratio"], case["steps"],
                          seed=seed, rel_time=case["sub"], n_seamounts=max(4, nx // 40), ngauges=case["gauges"])
    # the wave is on the shelf: still water would leave the child's terms unevaluated
    P, K = c.layers
    K.Z0 = np.where(K.H > 1.0, synth.gaussian_hump(K.x, K.y, float(K.x[K.nx // 3]), float(K.y[K.ny // 2]), 1.5, 25.0),
                    F32(0.0)).astype(F32)
    return c


def _requests(case, seed):
    """requests over three grid classes, one in three nested, each with its own source and length"""
    sizes = [(int(nx * case["scale"]), int(ny * case["scale"])) for nx, ny in ((481, 401), (961, 801), (1441, 1201))]
    templates = synth.config_c5_templates(seed=seed, sizes=sizes)
    rng = np.random.default_rng(seed)
    out = []
    for k in range(case["requests"]):
        steps = int(case["steps"] * (1.0 - 0.4 * (k * 0.618 % 1.0)))  # requests end at different times
        out.append(synth.c5_request_case(templates, sizes[k % 3], steps, k % 3 == 1 and k % 2 == 1,
                                         int(rng.integers(0, 2 ** 31))))
    return out


def _faults(case, seed):
    """a rectangular rupture cut into sub-faults with their own slip and rake"""
    x, y = synth.pc.axes(140.0, 20.0, case["nx"], case["ny"], 2.0)
    rng = np.random.default_rng(seed)
    lon, lat = float(x[case["nx"] // 3]), float(y[case["ny"] // 2])
    strike = float(rng.uniform(0.0, 360.0))
    out = []
    for k in range(case["faults"]):
        a, b = 0.35 * (k // 2 - case["faults"] / 4.0), 0.2 * (k % 2)
        t = math.radians(strike)
        out.append(dict(hh=float(rng.uniform(5e3, 15e3)) + 8e3 * (k % 2), l=40e3, w=25e3,
                        d=float(rng.uniform(0.5, 6.0)), th=strike, dl=float(rng.uniform(10.0, 35.0)),
                        rd=float(rng.uniform(60.0, 110.0)), x0=lon + a * math.sin(t) + b * math.cos(t),
                        y0=lat + a * math.cos(t) - b * math.sin(t), sw=0))
    return x, y, synth.bathymetry(x, y, rng, n_seamounts=8), out


class _StepIO(C.Structure):
    """gc_grid_step_io (include/gcomcot.h)"""
    _fields_ = ([("nx", C.c_int), ("ny", C.c_int), ("pitch", C.c_int)]
                + [(n, C.c_void_p) for n in ("z1", "m1", "n1", "z2", "m2", "n2", "h", "rows", "zmax")])


def _pitched(a):
    pitch = (a.shape[1] + 31) // 32 * 32
    t = torch.zeros((a.shape[0], pitch), dtype=torch.float32, device="cuda")
    t[:, :a.shape[1]] = torch.from_numpy(np.ascontiguousarray(a, dtype=F32)).cuda()
    return t


def _step_fields(case, seed):
    """grids in mid-propagation: a surface and the fluxes of a wave travelling in a seeded direction"""
    L = _single(case, seed).root
    rng = np.random.default_rng(seed + 1)
    speed = np.sqrt(9.807 * np.maximum(L.H, 0.0))
    out = []
    for _ in range(case["grids"]):
        a, b = float(rng.uniform(0.0, 2.0 * math.pi)), float(rng.uniform(0.5, 2.0))
        z = np.where(L.H > 0.0, b * L.Z0, 0.0).astype(F32)
        out.append((z, (speed * z * math.cos(a)).astype(F32), (speed * z * math.sin(a)).astype(F32)))
    return L, out


# ---------------------------------------------------------------------------
# prepare
# ---------------------------------------------------------------------------
class _Held:
    """an engine or server that is closed with the state that holds it"""

    def __init__(self, obj):
        self.obj = obj

    def __del__(self):
        try:
            self.obj.close()
        except Exception:
            pass


def prepare(case, seed):
    kind = case["kind"]
    st = {"case": case}
    if kind == "step":
        L, fields = _step_fields(case, seed)
        rec = np.zeros((L.ny, 8), F32)
        rec[:, :7] = L.coefs.rows().T
        h, rows = _pitched(L.H), torch.from_numpy(rec).cuda()
        arr, bufs = (_StepIO * len(fields))(), []
        for q, (z, m, n) in zip(arr, fields):
            b = {"z1": _pitched(z), "m1": _pitched(m), "n1": _pitched(n), "zmax": _pitched(np.maximum(z, 0.0))}
            b.update({k: torch.zeros_like(b["z1"]) for k in ("z2", "m2", "n2")})
            q.nx, q.ny, q.pitch = L.nx, L.ny, h.shape[1]
            for k, t in dict(b, h=h, rows=rows).items():
                setattr(q, k, t.data_ptr())
            bufs.append(b)
        st.update(lib=_lib.load(), arr=arr, ptr=C.cast(arr, C.c_void_p), bufs=bufs, keep=(h, rows), nx=L.nx)
    elif kind == "forecast":
        c = _single(case, seed, gauges=case["gauges"])
        eng = Engine(budget=BUDGET)
        cls = eng.add_class(c.root)
        z0 = [c.root.Z0]
        if case["members"] > 1:
            z0 = synth.ensemble_sources(c.root.x, c.root.y, case["members"], seed)
        st.update(held=_Held(eng), eng=eng, cls=cls, c=c, z0=z0)
    elif kind == "nested":
        c = _nested(case, seed)
        eng = Engine(budget=BUDGET)
        st.update(held=_Held(eng), eng=eng, cls=eng.add_nested_class(*c.layers), c=c)
    elif kind in ("drive", "calls"):
        c = _single(case, seed, laygov=case["laygov"], gauges=case["gauges"])
        # the Fortran-order arrays a caller holds for the whole run
        s = ReferenceSession(c, init_layers=False, host_cache=st.setdefault("cache", {}))
        s.close()
        st.update(c=c)
    elif kind == "serve":
        srv = ForecastServer(budget_bytes=BUDGET)
        st.update(held=_Held(srv), srv=srv, cases=_requests(case, seed))
    else:
        x, y, H, faults = _faults(case, seed)
        h = _pitched(H)
        st.update(lib=_lib.load(), arr=_lib.faults_array(faults), n=len(faults), h0=h, z=torch.zeros_like(h),
                  h=h.clone(), x=torch.from_numpy(x).cuda(), y=torch.from_numpy(y).cuda())
    return st


# ---------------------------------------------------------------------------
# run
# ---------------------------------------------------------------------------
def run(st):
    case = st["case"]
    kind = case["kind"]
    if kind == "step":
        rc = st["lib"].gcomcot_fused_step_noalloc(len(st["bufs"]), st["ptr"],
                                                  C.c_void_p(torch.cuda.current_stream().cuda_stream))
        if rc != 0:
            raise RuntimeError(f"gcomcot_fused_step_noalloc failed: {rc}")
        return [{k: b[k][:, :st["nx"]] for k in ("z2", "m2", "n2", "zmax")} for b in st["bufs"]]
    if kind == "fault":
        st["z"].zero_()
        st["h"].copy_(st["h0"])
        rc = st["lib"].gc_okada_apply(C.cast(st["arr"], C.c_void_p), st["n"], 0, case["nx"], case["ny"],
                                      st["h"].shape[1], st["x"].data_ptr(), st["y"].data_ptr(), 0.0, 0.0,
                                      st["z"].data_ptr(), st["h"].data_ptr(),
                                      C.c_void_p(torch.cuda.current_stream().cuda_stream))
        if rc != 0:
            raise RuntimeError(f"gc_okada_apply failed: {rc}")
        return {"z": st["z"][:, :case["nx"]], "h": st["h"][:, :case["nx"]]}
    if kind == "forecast":
        eng, c = st["eng"], st["c"]
        ids = [eng.add(c, z0=z, cls=st["cls"]) for z in st["z0"]]
        eng.step(case["steps"] + 1)  # the step after the last samples the last gauges
        eng.sync()
        if len(ids) == 1:
            out = [eng.read(ids[0])]
        else:  # an ensemble's products
            pend = [eng.read_async(i) for i in ids]
            out = [p.take() for p in pend]
        for i in ids:
            eng.release(i)
        return out
    if kind == "nested":
        eng = st["eng"]
        mid = eng.add(st["c"], cls=st["cls"])
        eng.step(case["steps"])
        eng.sync()
        out = eng.read(mid)
        eng.release(mid)
        return out
    if kind in ("drive", "calls"):
        s = ReferenceSession(st["c"], host_cache=st["cache"])
        try:
            if kind == "drive":
                ts = s.drive(case["steps"])
            else:
                ts = np.array([s.step() for _ in range(case["steps"])], F32)
            m, n = s.getmn()
            return {"ts": ts, "z": s.getz(), "m": m, "n": n, "zmax": s.getzmax()}
        finally:
            s.close()
    reqs = [Request(k, 0.0, c) for k, c in enumerate(st["cases"])]
    st["srv"].serve(reqs, speed=float("inf"))
    return [r.result for r in reqs]


# ---------------------------------------------------------------------------
# work
# ---------------------------------------------------------------------------
_FLOPS_LINEAR = 36      # MASS_S 8, MOMT_S 26, max-eta and its test 2, per cell and step
_FLOPS_NONLINEAR = 150  # CONMASS, CONMOME with advection and friction on both faces
_FLOPS_FAULT = 700      # projection and eight corner terms per cell and sub-fault


def work(case):
    """inputs read once and outputs written once, and the scheme's arithmetic"""
    kind = case["kind"]
    cells = case["nx"] * case["ny"] if "nx" in case else 0
    if kind == "step":
        # Z, M, N, max-eta per grid and the shared H in; Z, M, N, max-eta out
        return {"bytes": 4 * cells * (8 * case["grids"] + 1), "flops": _FLOPS_LINEAR * cells * case["grids"]}
    if kind == "fault":
        return {"bytes": 16 * cells, "flops": _FLOPS_FAULT * cells * case["faults"]}
    if kind == "forecast":
        # Z0 per member and H in; the fields and series read back out
        fields = 5 if case["members"] == 1 else 2
        return {"bytes": case["members"] * (4 * cells * (1 + fields) + 4 * case["steps"] * case["gauges"]) + 4 * cells,
                "flops": _FLOPS_LINEAR * cells * case["steps"] * case["members"]}
    if kind == "nested":
        kids = (case["cw"] * case["ratio"] + 1) * (case["ch"] * case["ratio"] + 1)
        return {"bytes": 4 * cells * 7 + 4 * kids * 7,
                "flops": case["steps"] * (_FLOPS_LINEAR * cells + _FLOPS_NONLINEAR * kids * case["sub"])}
    if kind in ("drive", "calls"):
        per = _FLOPS_NONLINEAR if case["laygov"] == 1 else _FLOPS_LINEAR
        return {"bytes": 4 * cells * 6 + 16 * case["steps"] * case["gauges"], "flops": per * cells * case["steps"]}
    area = sum(int(a * case["scale"]) * int(b * case["scale"]) for a, b in ((481, 401), (961, 801), (1441, 1201))) // 3
    return {"bytes": 4 * area * 4 * case["requests"],
            "flops": int(0.8 * _FLOPS_LINEAR * area * case["steps"] * case["requests"])}


# ---------------------------------------------------------------------------
# the same in 64 bits, plain torch
# ---------------------------------------------------------------------------
_G, _GX, _EPS, _UB = 9.807, 1.0e-5, 1.0e-10, 99.0


class _Plain:
    """MASS_S, OPEN and MOMT_S of one outer layer in double precision"""

    def __init__(self, L, dev):
        t = lambda a: torch.from_numpy(np.ascontiguousarray(a, dtype=np.float64)).to(dev)
        self.h = t(L.H)
        self.wet = self.h > _GX
        r1, r11, r6, r3, r5, cx, cy = (t(r)[:, None] for r in L.coefs.rows())
        self.r1, self.r11, self.r6, self.r3, self.r5 = r1, r11, r6, r3, r5
        self.r2 = cx * (0.5 * (self.h[:, :-1] + self.h[:, 1:]))
        self.r4 = (cy * 0.5)[:-1] * (self.h[:-1] + self.h[1:])
        self.wx = self.wet[:, :-1] & self.wet[:, 1:]
        self.wy = self.wet[:-1] & self.wet[1:]
        self.c = torch.sqrt(_G * torch.where(self.wet, self.h, torch.ones_like(self.h)))

    def _open(self, a, b, neg, c, wet):
        z = torch.sqrt(a * a + b * b) / c
        z = torch.where(neg, -z, z)
        return torch.where(wet & (z.abs() <= _UB), z, torch.zeros_like(z))

    def step(self, z, m, n):
        h, zero = self.h, torch.zeros((), dtype=torch.float64, device=z.device)
        nr = n * self.r6
        zn = torch.empty_like(z)
        i = (slice(1, -1), slice(1, -1))
        zz = z[i] - self.r1[1:-1] * (m[1:-1, 1:-1] - m[1:-1, :-2]) - self.r11[1:-1] * (nr[1:-1, 1:-1] - nr[:-2, 1:-1])
        zz = torch.where(zz.abs() < _EPS, zero, zz)
        zz = torch.where(zz + h[i] <= _EPS, -h[i], zz)
        zn[i] = torch.where(self.wet[i], zz, zero)
        c, w, k = self.c, self.wet, slice(1, -1)
        zn[0, k] = self._open(0.5 * (m[0, k] + m[0, :-2]), n[0, k], n[0, k] > 0, c[0, k], w[0, k])
        zn[-1, k] = self._open(0.5 * (m[-1, k] + m[-1, :-2]), n[-2, k], n[-2, k] < 0, c[-1, k], w[-1, k])
        side = torch.where(w[:-2, 0], 0.5 * (n[k, 0] + n[:-2, 0]), n[k, 0])
        zn[k, 0] = self._open(side, m[k, 0], m[k, 0] > 0, c[k, 0], w[k, 0])
        zn[k, -1] = self._open(0.5 * (n[k, -1] + n[:-2, -1]), m[k, -2], m[k, -2] < 0, c[k, -1], w[k, -1])
        for j, jn in ((0, 0), (-1, -2)):
            for q, qm in ((0, 0), (-1, -2)):
                a, b = m[j, qm], n[jn, q]
                neg = ((a > 0) if q == 0 else (a < 0)) | ((b > 0) if j == 0 else (b < 0))
                zn[j, q] = self._open(a, b, neg, c[j, q], w[j, q])
        ns = torch.cat([n[:1], n[:-1]])
        mn, nn = torch.zeros_like(m), torch.zeros_like(n)
        tot = n[:, :-1] + n[:, 1:] + ns[:, :-1] + ns[:, 1:]
        v = m[:, :-1] - self.r2 * (zn[:, 1:] - zn[:, :-1]) + self.r3 * tot
        mn[:, :-1] = torch.where(self.wx & (v.abs() >= _EPS), v, zero)
        mw = torch.cat([m[:, :1], m[:, :-1]], dim=1)
        tot = mw[:-1] + mw[1:] + m[:-1] + m[1:]
        v = n[:-1] - self.r4 * (zn[1:] - zn[:-1]) - self.r5[:-1] * tot
        nn[:-1] = torch.where(self.wy & (v.abs() >= _EPS), v, zero)
        return zn, mn, nn


def _plain_run(L, z0, steps, gauges, raw, dev):
    """fields after `steps` steps from rest, their maximum and every step's gauges"""
    P = _Plain(L, dev)
    z = torch.from_numpy(np.ascontiguousarray(z0, dtype=np.float64)).to(dev)
    m, n, top = torch.zeros_like(z), torch.zeros_like(z), z.clone()
    gi = torch.tensor([g[1] - 1 for g in gauges], dtype=torch.long, device=dev)
    gj = torch.tensor([g[2] - 1 for g in gauges], dtype=torch.long, device=dev)
    cx = torch.tensor([float(F32(g[3])) for g in gauges], dtype=torch.float64, device=dev)
    cy = torch.tensor([float(F32(g[4])) for g in gauges], dtype=torch.float64, device=dev)
    series = []
    for _ in range(steps):
        z, m, n = P.step(z, m, n)
        top = torch.maximum(top, z)
        if len(gauges):
            a, b, c, d = z[gj, gi], z[gj, gi + 1], z[gj + 1, gi], z[gj + 1, gi + 1]
            if raw:
                series.append(torch.stack([a, b, c, d], dim=1))
            else:
                series.append(a * (1 - cx) * (1 - cy) + b * cx * (1 - cy) + c * (1 - cx) * cy + d * cx * cy)
    ts = torch.stack(series).cpu().numpy() if series else np.zeros((steps, 0, 4) if raw else (steps, 0))
    return {"z": z.cpu().numpy(), "m": m.cpu().numpy(), "n": n.cpu().numpy(), "zmax": top.cpu().numpy(), "ts": ts}


def _stereo64(lon, lat, lon0, lat0):
    """the oblique stereographic projection of the fault source on WGS84 (x east, y north, metres)"""
    rad, pole = 0.01745329252, 3.14159265358979 / 2.0 - 1.0e-10
    clip = lambda v: np.clip(v, -pole, pole)
    lat, lon, lt0, ln0 = clip(lat * rad), lon * rad, clip(lat0 * rad), lon0 * rad
    e, f2 = 0.08181919092891, 0.00669438000426
    s0, c0 = math.sin(lt0), math.cos(lt0)
    t0 = math.sqrt(1.0 - f2 * s0 * s0)
    big = math.sqrt(6378137.0 * (1.0 - f2) / t0 ** 3 * float(int(6378137.0 / t0))) * 2.0 * 0.9996
    n = math.sqrt(1.0 + f2 * c0 ** 4 / (1.0 - f2))
    conf = lambda s: ((1.0 + s) / (1.0 - s) * ((1.0 - e * s) / (1.0 + e * s)) ** e) ** n
    w1 = conf(s0)
    x0 = (w1 - 1.0) / (w1 + 1.0)
    c = (n + s0) * (1.0 - x0) / (n - s0) / (1.0 + x0)
    xi0 = math.asin((c * w1 - 1.0) / (c * w1 + 1.0))
    w = c * conf(np.sin(lat))
    xi = np.arcsin((w - 1.0) / (w + 1.0))[:, None]
    d = (n * (lon - ln0))[None, :]
    b = 1.0 + np.sin(xi) * math.sin(xi0) + np.cos(xi) * math.cos(xi0) * np.cos(d)
    return (big * np.cos(xi) * np.sin(d) / b,
            big * (np.sin(xi) * math.cos(xi0) - np.cos(xi) * math.sin(xi0) * np.cos(d)) / b)


def _fault64(x, y, f):
    """vertical displacement of the free surface above one rectangular fault (Okada 1985)"""
    rad, tau = 0.01745329252, 2.0 * 3.14159
    dip, rake, strike = f["dl"] * rad, f["rd"] * rad, f["th"] * rad
    sn, cs, half = math.sin(dip), math.cos(dip), 0.5 * f["w"]
    hh = f["hh"] + half * sn
    xs, ys = _stereo64(x.astype(np.float64), y.astype(np.float64), f["x0"], f["y0"])
    xs = xs - half * cs * math.cos(strike)
    ys = ys + half * cs * math.sin(strike)
    x1 = xs * math.sin(strike) + ys * math.cos(strike)
    x2 = -(xs * math.cos(strike) - ys * math.sin(strike))
    p = x2 * cs + hh * sn
    q = x2 * sn - hh * cs
    us, ud = 0.0, 0.0
    for a, b, sign in ((_half(f), 0.0, 1), (_half(f), f["w"], -1), (-_half(f), 0.0, -1), (-_half(f), f["w"], 1)):
        y1, y2 = x1 + a, p - b
        db = y2 * sn - q * cs
        r = np.sqrt(y1 * y1 + y2 * y2 + q * q)
        xx = np.sqrt(y1 * y1 + q * q)
        a4 = 0.5 / cs * (np.log(np.maximum(r + db, 1e-10)) - sn * np.log(np.maximum(r + y2, 1e-10)))
        us = us - sign * (db * q / r / (r + y2) + q * sn / (r + y2) + a4 * sn) / tau
        a5 = np.arctan((y2 * (xx + q * cs) + xx * (r + xx) * sn) / y1 / (r + xx) / cs) / cs
        ud = ud - sign * (db * q / r / (r + y1) + sn * np.arctan(y1 * y2 / q / r) - a5 * sn * cs) / tau
    out = 0.0
    for v in (us * f["d"] * math.cos(rake), ud * f["d"] * math.sin(rake)):
        v = np.where(np.isfinite(v), v, 0.0)
        out = out + np.where(np.abs(v) <= _GX, 0.0, v)
    return out


def _half(f):
    return 0.5 * f["l"]


def exact(case, seed):
    """what `run` returns, in 64 bits; None for the nested and nonlinear schemes and the server's mix (cell by cell
    branches on wet and dry faces: minutes in plain torch)"""
    kind = case["kind"]
    dev = torch.device("cuda" if torch.cuda.is_available() else "cpu")
    if kind == "step":
        L, fields = _step_fields(case, seed)
        P, out = _Plain(L, dev), []
        for z, m, n in fields:
            t = [torch.from_numpy(a.astype(np.float64)).to(dev) for a in (z, m, n)]
            a, b, c = P.step(*t)
            top = torch.maximum(torch.from_numpy(np.maximum(z, 0.0).astype(np.float64)).to(dev), a)
            out.append(dict(zip(("z2", "m2", "n2", "zmax"), (v.cpu().numpy() for v in (a, b, c, top)))))
        return out
    if kind == "fault":
        x, y, H, faults = _faults(case, seed)
        d = sum(_fault64(x, y, f) for f in faults)
        return {"z": d, "h": H.astype(np.float64) - d}
    if kind == "forecast" and dev.type == "cuda":
        c = _single(case, seed, gauges=case["gauges"])
        one = case["members"] == 1
        cost = max(0.5e-3, 4.0e-10 * case["nx"] * case["ny"]) * case["steps"] * case["members"]
        if cost > 16.0:  # seconds, about
            return None
        out = []
        for z0 in [c.root.Z0] if one else synth.ensemble_sources(c.root.x, c.root.y, case["members"], seed):
            r = _plain_run(c.root, z0, case["steps"], c.gauges, False, dev)
            if not one:  # the products: max-eta, arrival and, with gauges, their series
                r = {k: r[k] for k in (("zmax", "ts") if case["gauges"] else ("zmax",))}
            out.append(dict(r, arrival=None))
        return out
    if kind in ("drive", "calls") and case["laygov"] == 0 and dev.type == "cuda":
        c = _single(case, seed, gauges=case["gauges"])
        return _plain_run(c.root, c.root.Z0, case["steps"], c.gauges, kind == "drive", dev)
    return None
