"""The work that programs give this library, as measurable cases: fields through the calculators
and the device entry points, multi-focus solvers, many patterns on one geometry, uneven batches
and request serving.  Geometries, attenuations and size ranges follow workloads.py, the tests and
the benchmark; every input is made from a seed.

A case is a dict of plain values; `kind` selects the entry points:
  calculate  a calculator object (AFC_Calculate) on a grid slice or scatter points, host results
  field      AFC_FieldGridDevice / AFC_FieldScatterDevice on buffers that live on the GPU
  solve      an Optimizer method (AFO_*) that rewrites a system's drive
  multi      AFC_MultiPatternApply, with AFC_MultiPatternBuildG before it where `build` is set
  batch      AFC_BatchRun of a tuned plan
  serve      a burst of requests through AFC_ServeSubmit* / AFC_ServeWait
"""
import ctypes
import math
import os
import sys

import numpy as np
import torch

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
PKG = os.path.join(ROOT, "acoustic-field-calculator_gb300")
if PKG not in sys.path:
    sys.path.insert(0, PKG)

import afc  # noqa: E402
import workloads as W  # noqa: E402
from afc import nativemethods as nm  # noqa: E402

TILINGS = {249: (1, 1), 498: (2, 1), 996: (2, 2), 2490: (5, 2), 3984: (4, 4)}
PRESSURE, POWER, COMPLEX = 0, 1, 2
BF16X3, FP16 = 1, 2
ALPHA = 1.15e-2  # /mm, the large-grid configuration's attenuation
SLICE = 201  # side of a served hologram's pressure slice
CALCULATORS = {"cpu": afc.CpuCalculator, "accurate": afc.AccurateCalculator,
               "gpu": afc.GpuCalculator}
BUFFERS = (afc.PressureFieldBuffer, afc.PowerFieldBuffer, afc.ComplexPressureFieldBuffer)


def listed():
    return [
        # the reference's own example: one array, one focus, the pressure around it; what an
        # interactive program calls after every edit of the drive, so its latency counts
        dict(name="focus_slice", kind="calculate", calc="gpu", n=249, st=1, field=PRESSURE,
             shape="slice", side=101, alpha=0.0, drive="focus"),
        # the Accurate calculator on the slice that follows a hologram on a 2 x 2 array
        dict(name="accurate_slice", kind="calculate", calc="accurate", n=996, st=1,
             field=PRESSURE, shape="slice", side=SLICE, alpha=0.0, drive="random"),
        # the headline: a 4 x 4 array's complex field in a volume
        dict(name="grid_256", kind="field", n=3984, st=1, field=COMPLEX, shape="grid", c0=256,
             c1=256, c2=256, alpha=ALPHA),
        # the same array seen from scattered points (one pattern of the multi-pattern geometry)
        dict(name="scatter_65536", kind="field", n=3984, st=1, field=COMPLEX, shape="scatter",
             m=65536, alpha=ALPHA),
        # a haptics or levitation frame: a few foci, solved many times a second
        dict(name="gspat_8", kind="solve", solver="gs_pat", n=996, st=1, foci=8),
        # a dense hologram: more foci than the serving mix asks for
        dict(name="gspat_128", kind="solve", solver="gs_pat", n=996, st=1, foci=128),
        # the reference's nonlinear least-squares optimizer on the solver tests' problem
        dict(name="lm_16", kind="solve", solver="lm", n=996, st=1, foci=16),
        # the reference's matrix optimizer on the matrix tests' mid-size problem
        dict(name="horn_31", kind="solve", solver="horn", n=996, st=1, foci=31),
        # a library of patterns against a resident geometry, at the accurate precision
        dict(name="patterns_bf16x3", kind="multi", precision=BF16X3, n=3984, st=1, m=65536,
             patterns=1024, build=False),
        # a new geometry for a few patterns: G is built for it, then applied, at FP16
        dict(name="geometry_fp16", kind="multi", precision=FP16, n=3984, st=1, m=65536,
             patterns=128, build=True),
        # uneven independent jobs, grid slices and scatter sets, replayed as one plan
        dict(name="batch_64", kind="batch", jobs=64, m_hi=1000000, mix=3),
        # a burst of served requests: 70 % field jobs, 30 % holograms
        dict(name="serve_48", kind="serve", requests=48, m_hi=1000000, foci_hi=64, mix=4),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["calculate", "calculate", "field", "field", "solve", "solve", "multi",
                       "multi", "batch", "serve"])
    n = rng.choice([249, 498, 996, 2490, 3984])
    st = rng.choice([1, 1, 1, 0])
    alpha = rng.choice([0.0, ALPHA])
    if kind == "calculate":
        shape = rng.choice(["slice", "slice", "points"])
        return dict(kind=kind, calc=rng.choice(["cpu", "accurate", "gpu"]), n=n, st=st,
                    field=rng.choice([PRESSURE, POWER, COMPLEX]), shape=shape,
                    side=_log(rng, 21, 401) if shape == "slice" else 0,
                    m=0 if shape == "slice" else _log(rng, 100, 20000), alpha=alpha,
                    drive=rng.choice(["focus", "random"]))
    if kind == "field":
        if rng.random() < 0.5:
            return dict(kind=kind, n=n, st=st, field=rng.choice([PRESSURE, POWER, COMPLEX]),
                        shape="grid", c0=_log(rng, 24, 256), c1=_log(rng, 24, 256),
                        c2=_log(rng, 1, 160), alpha=alpha)
        return dict(kind=kind, n=n, st=st, field=rng.choice([PRESSURE, POWER, COMPLEX]),
                    shape="scatter", m=_log(rng, 1000, 1000000), alpha=alpha)
    if kind == "solve":
        solver = rng.choice(["gs_pat", "gs_pat", "lm", "horn"])
        n = rng.choice([249, 498, 996, 2490])
        hi = {"gs_pat": 256, "lm": 24, "horn": 64}[solver]
        return dict(kind=kind, solver=solver, n=n, st=st, foci=_log(rng, 2, hi))
    if kind == "multi":
        return dict(kind=kind, precision=rng.choice([BF16X3, FP16]), n=n, st=st,
                    m=_log(rng, 500, 65536), patterns=_log(rng, 16, 1024),
                    build=rng.random() < 0.5)
    if kind == "batch":
        return dict(kind=kind, jobs=_log(rng, 8, 64), m_hi=_log(rng, 30000, 1000000),
                    mix=rng.randrange(1000))
    return dict(kind=kind, requests=_log(rng, 4, 48), m_hi=_log(rng, 30000, 1000000),
                foci_hi=_log(rng, 8, 64), mix=rng.randrange(1000))


# ---------------------------------------------------------------- inputs (host, from the seed)


def _rng(case, seed):
    return np.random.default_rng([int(seed), sum(case["kind"].encode())])


def _array(n, st, alpha, amp, phase):
    pos = W.tiled_array(*TILINGS[n])
    rec = (W.t4010a1_records if st == 1 else W.sphere_records)(pos, amp, phase)
    k = np.full(n, W.wavenumber(), np.float32)
    return rec, k, np.full(n, alpha, np.float32), W.array_center(pos)


def _pattern(rng, n, drive="random"):
    if drive == "random":
        return (rng.uniform(0.5, 1.0, n).astype(np.float32),
                rng.uniform(0.0, 2.0 * math.pi, n).astype(np.float32))
    pos = W.tiled_array(*TILINGS[n])
    cen = W.array_center(pos)
    focus = (cen[0] + rng.uniform(-30, 30), cen[1] + rng.uniform(-30, 30), 150.0)
    return np.ones(n, np.float32), W.focal_phases(pos, focus).astype(np.float32)


def _grid(cen, counts, res, z):
    """An XYZ grid centred on the array, z upwards from z: (GridSpec, origin, counts, res).  The
    ranges are padded by half a step so that the f32 counts come out exact."""
    lo = [float(np.float32(cen[0] - (counts[0] - 1) * res / 2)),
          float(np.float32(cen[1] - (counts[1] - 1) * res / 2)), float(np.float32(z))]
    hi = [o + (c - 1) * res + 0.5 * res for o, c in zip(lo, counts)]
    dim = 3 if counts[2] > 1 else 2
    if dim == 2:
        hi[2] = lo[2]
    spec = W.GridSpec(dim, list(zip(lo, hi)), res, (W.AXIS_X, W.AXIS_Y, W.AXIS_Z))
    return spec, lo, list(counts), res


def _box(rng, cen, m, half=100.0, z=(50.0, 200.0)):
    pts = rng.random((m, 3), dtype=np.float32)
    lo = np.array([cen[0] - half, cen[1] - half, z[0]], np.float32)
    span = np.array([2 * half, 2 * half, z[1] - z[0]], np.float32)
    return lo + span * pts


def _foci(rng, cen, m):
    foci = np.empty((m, 3), np.float32)
    foci[:, :2] = cen[:2] + rng.uniform(-50, 50, (m, 2))
    foci[:, 2] = rng.uniform(100.0, 200.0, m)
    return foci, rng.uniform(0.5, 1.0, m).astype(np.float32)


def _job(mix, rng, m_hi, grid):
    """One job of the uneven mix: 249 to 2,490 sources, 1,000 to m_hi points (the sizes from `mix`,
    which belongs to the case, the values from the seed's rng)."""
    n = int(mix.choice([249, 498, 996, 2490]))
    amp, ph = _pattern(rng, n)
    rec, k, a, cen = _array(n, 1, ALPHA, amp, ph)
    m = int(round(math.exp(mix.uniform(math.log(1000), math.log(m_hi)))))
    job = dict(n=n, rec=rec, k=k, a=a, amp=amp, ph=ph, field=int(mix.integers(0, 3)), grid=None,
               pts=None)
    if grid:
        side = max(2, int(round(math.sqrt(m))))
        job["grid"] = _grid(cen, (side, side, 1), float(rng.uniform(0.5, 2.0)),
                            float(rng.uniform(50.0, 200.0)))
        job["m"] = side * side
    else:
        job["pts"] = _box(rng, cen, m, half=float(rng.uniform(30.0, 120.0)))
        job["m"] = m
    return job


def _inputs(case, seed):
    rng = _rng(case, seed)
    kind = case["kind"]
    if kind in ("calculate", "field"):
        amp, ph = _pattern(rng, case["n"], case.get("drive", "random"))
        rec, k, a, cen = _array(case["n"], case["st"], case["alpha"], amp, ph)
        x = dict(rec=rec, k=k, a=a, grid=None, pts=None)
        if case["shape"] == "slice":
            x["grid"] = _grid(cen, (case["side"], case["side"], 1), 1.0, 150.0)
        elif case["shape"] == "grid":
            x["grid"] = _grid(cen, (case["c0"], case["c1"], case["c2"]), 0.5, 50.0)
        else:
            x["pts"] = _box(rng, cen, case["m"])
        return x
    if kind == "solve":
        rec, k, a, cen = _array(case["n"], case["st"], 0.0, 1.0, 0.0)
        foci, amps = _foci(rng, cen, case["foci"])
        return dict(rec=rec, k=k, a=a, foci=foci, amps=amps)
    if kind == "multi":
        rec, k, a, cen = _array(case["n"], case["st"], ALPHA, 1.0, 0.0)
        size = (case["patterns"], case["n"])
        return dict(rec=rec, k=k, a=a, pts=_box(rng, cen, case["m"]),
                    amps=rng.random(size, dtype=np.float32) * np.float32(0.5) + np.float32(0.5),
                    phases=rng.random(size, dtype=np.float32) * np.float32(2 * math.pi))
    mix = np.random.default_rng(case["mix"])
    if kind == "batch":
        return [_job(mix, rng, case["m_hi"], i % 2 == 0) for i in range(case["jobs"])]
    out = []
    cen = W.array_center(W.tiled_array(2, 2))
    for i in range(case["requests"]):
        if i % 10 not in (2, 5, 8):  # 70 % of them
            out.append(dict(_job(mix, rng, case["m_hi"], mix.random() < 0.5), hologram=False))
        else:
            foci, amps = _foci(rng, cen, int(mix.integers(2, case["foci_hi"] + 1)))
            out.append(dict(hologram=True, n=996, foci=foci, amps=amps, m=SLICE * SLICE, field=0,
                            grid=_grid(cen, (SLICE, SLICE, 1), 1.0, float(foci[:, 2].mean()))))
    return out


# ---------------------------------------------------------------- states


def _gpu(a):
    return torch.from_numpy(np.ascontiguousarray(a).reshape(-1)).cuda()


def _ok(rc):
    if rc < 0:
        raise RuntimeError(afc.last_error())


def _system(x, st):
    s = afc.UniformSystem(300.0)
    s.add_records(st, x["rec"], x["k"], x["a"])
    return s


class _Owner:
    """A native handle that is freed with the object."""

    def __init__(self, handle, free):
        self.h, self.free = handle, free

    def __del__(self):
        if self.h:
            self.free(self.h)
            self.h = None


def _floats(field):
    return 2 if field == COMPLEX else 1


def _aligned(n):
    return (n + 63) // 64 * 64


def prepare(case, seed):
    x = _inputs(case, seed)
    return {"calculate": _prepare_calculate, "field": _prepare_field, "solve": _prepare_solve,
            "multi": _prepare_multi, "batch": _prepare_batch,
            "serve": _prepare_serve}[case["kind"]](case, x)


def _prepare_calculate(case, x):
    if x["grid"]:
        area = afc.grid_from_spec(x["grid"][0])
    else:
        area = afc.ScatterArea()
        area.add_observe_points(x["pts"])
    return dict(kind="calculate", calc=CALCULATORS[case["calc"]](), system=_system(x, case["st"]),
                area=area, buffer=BUFFERS[case["field"]]())


def _prepare_field(case, x):
    n = case["n"]
    s = dict(kind="field", st=case["st"], field=case["field"], n=n, src=_gpu(x["rec"]),
             k=_gpu(x["k"]), a=_gpu(x["a"]), desc=None, pts=None, m=case.get("m", 0))
    if x["grid"]:
        s["desc"] = afc.grid_from_spec(x["grid"][0]).grid_desc()
        s["m"] = case["c0"] * case["c1"] * case["c2"]
    else:
        s["pts"] = _gpu(x["pts"])
    s["out"] = torch.empty(s["m"] * _floats(s["field"]), device="cuda")
    s["ws_bytes"] = afc.DLL.AFC_FieldWorkspaceBytes(n)
    s["ws"] = torch.empty(s["ws_bytes"], dtype=torch.uint8, device="cuda")
    return s


def _prepare_solve(case, x):
    system = _system(x, case["st"])
    return dict(kind="solve", solver=getattr(afc.Optimizer, case["solver"]), system=system,
                records=system.records(), iamp=6 if case["st"] == 1 else 3, foci=x["foci"],
                amps=x["amps"])


def _prepare_multi(case, x):
    n, m, K, p = case["n"], case["m"], case["patterns"], case["precision"]
    ws_bytes = afc.DLL.AFC_MultiPatternWorkspaceBytes(n, m, K, p)
    ws = torch.empty(ws_bytes + 256, dtype=torch.uint8, device="cuda")
    s = dict(kind="multi", build=case["build"], st=case["st"], n=n, m=m, K=K, p=p,
             src=_gpu(x["rec"]), k=_gpu(x["k"]), a=_gpu(x["a"]), pts=_gpu(x["pts"]),
             amps=_gpu(x["amps"]), phases=_gpu(x["phases"]), ws=ws, ws_bytes=ws_bytes,
             base=(ws.data_ptr() + 255) // 256 * 256, out=torch.empty(2 * m * K, device="cuda"))
    if not case["build"]:
        _build_g(s)
    return s


def _build_g(s):
    _ok(afc.DLL.AFC_MultiPatternBuildG(
        s["st"], s["p"], s["src"].data_ptr(), s["k"].data_ptr(), s["a"].data_ptr(), s["n"],
        s["pts"].data_ptr(), s["m"], s["K"], s["base"], s["ws_bytes"],
        torch.cuda.current_stream().cuda_stream))


def _prepare_batch(case, x):
    arr = (nm.FieldJob * len(x))()
    out = torch.empty(sum(_aligned(j["m"] * _floats(j["field"])) for j in x), device="cuda")
    at, keep, outs = 0, [], []
    for f, j in zip(arr, x):
        src, k, a = _gpu(j["rec"]), _gpu(j["k"]), _gpu(j["a"])
        keep += [src, k, a]
        f.n_sources, f.field_type = j["n"], j["field"]
        f.d_sources, f.d_wavenums, f.d_attens = src.data_ptr(), k.data_ptr(), a.data_ptr()
        if j["grid"]:
            f.is_grid, f.grid = 1, afc.grid_from_spec(j["grid"][0]).grid_desc()
        else:
            pts = _gpu(j["pts"])
            keep.append(pts)
            f.is_grid, f.d_points, f.n_points = 0, pts.data_ptr(), j["m"]
        size = j["m"] * _floats(j["field"])
        f.d_out = out[at:].data_ptr()
        outs.append((at, size))
        at += _aligned(size)
    for a, size in outs:  # the gaps between the jobs' outputs are never written
        out[a + size:a + _aligned(size)] = 0
    plan = ctypes.c_void_p()
    _ok(afc.DLL.AFC_BatchCreate(1, arr, len(x), 1, ctypes.byref(plan),
                                torch.cuda.current_stream().cuda_stream))
    return dict(kind="batch", plan=_Owner(plan, afc.DLL.AFC_BatchFree), keep=keep, out=out)


def _prepare_serve(case, x):
    cfg = nm.ServeConfig(1 << 30, 256 << 20, 32)
    h = ctypes.c_void_p()
    _ok(afc.DLL.AFC_ServeCreate(ctypes.byref(cfg), ctypes.byref(h)))
    owner = _Owner(h, afc.DLL.AFC_ServeDestroy)
    ids = {}
    for n, alpha in [(249, ALPHA), (498, ALPHA), (996, ALPHA), (2490, ALPHA), (996, 0.0)]:
        rec, k, a, _ = _array(n, 1, alpha, 1.0, 0.0)
        gid = ctypes.c_int32()
        _ok(afc.DLL.AFC_ServeAddGeometry(h, 1, rec.ctypes.data, k.ctypes.data, a.ctypes.data, n,
                                         ctypes.byref(gid)))
        ids[n, alpha] = gid.value
    out = np.zeros(sum(_aligned(r["m"] * _floats(r["field"])) for r in x), np.float32)
    drives = np.zeros((sum(r["hologram"] for r in x), 996, 2), np.float32)
    at, d, calls = 0, 0, []
    for r in x:
        desc = afc.grid_from_spec(r["grid"][0]).grid_desc() if r["grid"] else None
        to = out[at:].ctypes.data
        at += _aligned(r["m"] * _floats(r["field"]))
        if r["hologram"]:
            calls.append((afc.DLL.AFC_ServeSubmitGspat,
                          (h, ids[996, 0.0], r["foci"].ctypes.data, r["amps"].ctypes.data,
                           len(r["amps"]), ctypes.byref(desc), to, drives[d].ctypes.data)))
            d += 1
        else:
            pts = None if r["grid"] else r["pts"].ctypes.data
            calls.append((afc.DLL.AFC_ServeSubmitField,
                          (h, ids[r["n"], ALPHA], r["amp"].ctypes.data, r["ph"].ctypes.data,
                           r["field"], 1 if r["grid"] else 0,
                           ctypes.byref(desc) if r["grid"] else None, pts,
                           0 if r["grid"] else r["m"], to)))
    return dict(kind="serve", h=h, owner=owner, keep=x, calls=calls, out=out, drives=drives)


# ---------------------------------------------------------------- one pass


def run(s):
    kind, dll = s["kind"], afc.DLL
    if kind == "calculate":
        return s["calc"].calculate(s["system"], s["area"], s["buffer"])
    if kind == "field":
        args = (s["st"], s["field"], 0, s["src"].data_ptr(), s["k"].data_ptr(),
                s["a"].data_ptr(), s["n"])
        rest = (s["out"].data_ptr(), s["ws"].data_ptr(), s["ws_bytes"],
                torch.cuda.current_stream().cuda_stream)
        if s["desc"] is not None:
            _ok(dll.AFC_FieldGridDevice(*args, ctypes.byref(s["desc"]), *rest))
        else:
            _ok(dll.AFC_FieldScatterDevice(*args, s["pts"].data_ptr(), s["m"], *rest))
        return s["out"]
    if kind == "solve":
        # the solvers write the drive over the system's; each starts from unit amplitudes
        rec, i = s["records"], s["iamp"]
        rec[:, i] = 1.0
        s["solver"](s["system"], s["foci"], s["amps"])
        amp, phase = rec[:, i], rec[:, i + 1]
        return np.stack([amp * np.cos(phase), amp * np.sin(phase)])
    if kind == "multi":
        if s["build"]:
            _build_g(s)
        _ok(dll.AFC_MultiPatternApply(s["p"], s["amps"].data_ptr(), s["phases"].data_ptr(),
                                      s["n"], s["m"], s["K"], s["out"].data_ptr(), s["base"],
                                      s["ws_bytes"], torch.cuda.current_stream().cuda_stream))
        return s["out"]
    if kind == "batch":
        _ok(dll.AFC_BatchRun(s["plan"].h, torch.cuda.current_stream().cuda_stream))
        return s["out"]
    ids = [fn(*args) for fn, args in s["calls"]]
    latency, queued = ctypes.c_double(), ctypes.c_double()
    for i in ids:
        _ok(i)
        _ok(dll.AFC_ServeWait(s["h"], i, ctypes.byref(latency), ctypes.byref(queued)))
    amp, phase = s["drives"][..., 0], s["drives"][..., 1]
    return [s["out"], amp * np.cos(phase), amp * np.sin(phase)]


# ---------------------------------------------------------------- what a pass cannot do without

EVAL = 37.0  # FP32 and special-function operations of one source-point pair


def _field_work(n, m, field, scatter):
    return 44.0 * n + (12.0 * m if scatter else 0.0) + 4.0 * _floats(field) * m, EVAL * n * m


def _gspat_work(n, m):
    # G, its column sums, R = G B, 101 products with R, the back-propagation
    return 52.0 * n + 16.0 * m, EVAL * n * m + 4.0 * n * m + 8.0 * n * m * m + 808.0 * m * m + 8.0 * n * m


def work(case):
    kind = case["kind"]
    n = case.get("n", 0)
    if kind == "calculate":
        m = case["side"] ** 2 if case["shape"] == "slice" else case["m"]
        b, f = _field_work(n, m, case["field"], case["shape"] != "slice")
    elif kind == "field":
        grid = case["shape"] == "grid"
        m = case["c0"] * case["c1"] * case["c2"] if grid else case["m"]
        b, f = _field_work(n, m, case["field"], not grid)
    elif kind == "solve":
        m = case["foci"]
        b, f = _gspat_work(n, m)
        if case["solver"] == "lm":  # up to 200 steps of U U^T and four products with B
            f = EVAL * n * m + 200.0 * (8.0 * n * m * m + 32.0 * n * m)
        elif case["solver"] == "horn":  # K, 100 m steps of an m x m product, the back-projection
            f = EVAL * n * m + 4.0 * n * m * m + 800.0 * m ** 3 + 8.0 * n * m
    elif kind == "multi":
        m, K, planes = case["m"], case["patterns"], 2.0 if case["precision"] == BF16X3 else 1.0
        b = 8.0 * n * K + 8.0 * m * K + planes * 4.0 * n * m
        f = 8.0 * n * m * K * (3.0 if case["precision"] == BF16X3 else 1.0)
        if case["build"]:
            b += planes * 4.0 * n * m
            f += EVAL * n * m
    else:  # the means of the mix: 1,058 sources; log-uniform point counts
        jobs = case["jobs"] if kind == "batch" else 0.7 * case["requests"]
        m = (case["m_hi"] - 1000.0) / math.log(case["m_hi"] / 1000.0)
        b, f = (jobs * v for v in _field_work(1058.0, m, PRESSURE, False))
        if kind == "serve":
            g = 0.3 * case["requests"]
            for v in (_gspat_work(996.0, case["foci_hi"] / 2), _field_work(996, SLICE ** 2, 0, False)):
                b, f = b + g * v[0], f + g * v[1]
    return {"bytes": b, "flops": f}


# ---------------------------------------------------------------- the same in 64 bits

# The T4010A1 directivity's cubic per 10-degree bin, a + b x + c x^2 + d x^3 in the angle past the
# bin's start (the reference's f32 table); bins 0 to 2 are 1, bins past 9 are 0.
_DIR = np.array([
    [1.0, 0.0, 0.0, 0.0], [1.0, 0.0, 0.0, 0.0], [1.0, 0.0, 0.0, 0.0],
    [1.0, -0.2633589359691162, -2.586746661956269, 0.0009174516976956062],
    [0.891250938, -0.8910683499820542, -1.0097633564074366, 0.0001704413361662757],
    [0.707945784, -1.1924098538381465, -0.7167962799004945, 4.362034715924911],
    [0.501187234, -1.0439934287916925, 0.027352097655185065, -2.238476800444034],
    [0.354813389, -0.7015151838490918, 0.39509604454751995, 1.274774620435337],
    [0.251188643, -0.4471050803642494, 1.0625664749725618, -1.1276955684895724],
    [0.199526231, -0.179254124486545, 0.008242027161100222, -0.9016569137759131],
    [0.0, 0.0, 0.0, 0.0]], np.float32).astype(np.float64)


def _f64(a):
    return torch.from_numpy(np.asarray(a)).cuda().double()


def _pairs64(st, rec, k, a, pts):
    """(amplitude factor, phase) of every point (rows) and source (columns): D e^{-alpha r} / r
    and k r, without the sources' own amplitudes and phases."""
    d = pts[:, None, :] - rec[None, :, :3]
    r = d.square().sum(-1).sqrt()
    w = torch.exp(-a * r) / r
    if st == 1:
        th = torch.acos(((d * rec[None, :, 3:6]).sum(-1) / r).clamp(-1.0, 1.0))
        b = torch.ceil(th / (math.pi / 18.0)).clamp(0.0, 10.0).long()
        x = th - (b - 1) * (math.pi / 18.0)
        c = _f64(_DIR)[b]
        w = w * (c[..., 0] + (c[..., 1] + (c[..., 2] + c[..., 3] * x) * x) * x)
    return w, k * r


def _chunks(pts, n):
    step = max(1, int(1.2e7 // max(n, 1)))
    return (pts[i:i + step] for i in range(0, len(pts), step))


def _g64(st, rec, k, a, pts):
    """G of unit amplitudes and zero phases, points by sources."""
    return torch.cat([torch.polar(*_pairs64(st, rec, k, a, p)) for p in _chunks(pts, len(rec))])


def _field64(st, rec, k, a, pts, q=None):
    """Complex field at pts of the drive q (the records' own where None)."""
    if q is None:
        i = 6 if st == 1 else 3
        q = torch.polar(rec[:, i].contiguous(), rec[:, i + 1].contiguous())
    return torch.cat([torch.polar(*_pairs64(st, rec, k, a, p)) @ q
                      for p in _chunks(pts, len(rec))])


def _points64(x):
    if x["grid"] is None:
        return _f64(x["pts"])
    _, lo, counts, res = x["grid"]
    # coordinates are f32 numbers: origin + index * spacing, rounded after each operation
    ax = [np.float32(o) + np.arange(c, dtype=np.float32) * np.float32(res) if c > 1
          else np.full(1, o, np.float32) for o, c in zip(lo, counts)]
    z, y, xx = np.meshgrid(ax[2], ax[1], ax[0], indexing="ij")
    return _f64(np.stack([xx, y, z], -1).reshape(-1, 3))


def _as_field(p, field):
    return p if field == COMPLEX else p.abs() if field == PRESSURE else p.abs().square()


def _gspat64(g, amps):
    den2 = g.abs().sum(0).square()
    r = (g / den2) @ g.conj().T
    p0 = amps.to(g.dtype)
    gam = r @ p0
    for _ in range(100):
        gam = r @ (gam / gam.abs() * p0)
    return (g.conj().T @ (gam / gam.abs().square() * p0.square())) / den2


def _horn64(g, amps):
    g, amps = g.cpu().numpy(), amps.cpu().numpy()
    m = len(amps)
    inv = np.linalg.inv(g @ g.conj().T + 1e-10 * np.eye(m))
    mm = amps[:, None] * inv * amps
    mm /= np.abs(mm).max()
    x = np.eye(m, dtype=np.complex128)
    state, mask = 0x243F6A8885A308D3, (1 << 64) - 1  # SplitMix64: the order of the coordinates
    for _ in range(100 * m):
        state = (state + 0x9E3779B97F4A7C15) & mask
        z = ((state ^ (state >> 30)) * 0xBF58476D1CE4E5B9) & mask
        z = ((z ^ (z >> 27)) * 0x94D049BB133111EB) & mask
        v = np.float32((z ^ (z >> 31)) >> 41) * np.float32(2.0 ** -23)
        i = min(int(np.float32(m) * v), m - 1)
        c = mm[:, i].copy()
        c[i] = 0
        xb = x @ c
        xb[i] = 0
        gamma = np.vdot(xb, c).real
        new = -math.sqrt(0.8 / gamma) * xb if gamma > 0 else np.zeros_like(xb)
        keep = x[i, i]
        x[:, i], x[i, :] = new, new.conj()
        x[i, i] = keep
    u = np.linalg.eigh(x)[1][:, -1]
    u = u * (abs(u[0]) / u[0])  # first entry real and positive
    q = g.conj().T @ (inv @ (amps * u))
    return torch.from_numpy(q / (np.abs(q.real) + np.abs(q.imag)).max()).cuda()


def _drive64(q):
    return torch.stack([q.real, q.imag])


def exact(case, seed):
    kind = case["kind"]
    if kind == "calculate" or kind == "field":
        if work(case)["flops"] > EVAL * 2e10:
            return None
        x = _inputs(case, seed)
        p = _as_field(_field64(case["st"], _f64(x["rec"]), _f64(x["k"]), _f64(x["a"]),
                               _points64(x)), case["field"])
        if kind == "calculate":
            return p.cpu().numpy()
        return torch.view_as_real(p).reshape(-1) if case["field"] == COMPLEX else p
    x = _inputs(case, seed)
    if kind == "solve":
        if case["solver"] == "lm":
            return None  # which of many equal optima 200 f32 steps end in is not a 64-bit value
        g = _g64(case["st"], _f64(x["rec"]), _f64(x["k"]), _f64(x["a"]), _f64(x["foci"]))
        solver = {"gs_pat": _gspat64, "horn": _horn64}[case["solver"]]
        return _drive64(solver(g, _f64(x["amps"]))).cpu().numpy()
    if kind == "multi":
        rec, k, a = _f64(x["rec"]), _f64(x["k"]), _f64(x["a"])
        q = torch.polar(_f64(x["amps"]), _f64(x["phases"])).T.contiguous()
        p = torch.cat([torch.polar(*_pairs64(case["st"], rec, k, a, c)) @ q
                       for c in _chunks(_f64(x["pts"]), case["n"])])
        return torch.view_as_real(p).reshape(-1)
    if kind == "batch":
        parts = []
        for j in x:
            p = _as_field(_field64(1, _f64(j["rec"]), _f64(j["k"]), _f64(j["a"]), _points64(j)),
                          j["field"])
            p = torch.view_as_real(p).reshape(-1) if p.is_complex() else p
            parts.append(torch.nn.functional.pad(p, (0, _aligned(len(p)) - len(p))))
        return torch.cat(parts)
    parts, drives = [], []
    rec0, k0, a0, _ = _array(996, 1, 0.0, 1.0, 0.0)
    for r in x:
        if r["hologram"]:
            rec, k, a = _f64(rec0), _f64(k0), _f64(a0)
            q = _gspat64(_g64(1, rec, k, a, _f64(r["foci"])), _f64(r["amps"]))
            drives.append(q)
            p = _field64(1, rec, k, a, _points64(r), q).abs()
        else:
            p = _as_field(_field64(1, _f64(r["rec"]), _f64(r["k"]), _f64(r["a"]), _points64(r)),
                          r["field"])
            p = torch.view_as_real(p).reshape(-1) if p.is_complex() else p
        parts.append(torch.nn.functional.pad(p, (0, _aligned(len(p)) - len(p))))
    q = torch.stack(drives) if drives else torch.zeros((0, 996), dtype=torch.complex128)
    return [torch.cat(parts).cpu().numpy(), q.real.cpu().numpy(), q.imag.cpu().numpy()]
