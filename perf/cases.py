"""The work a user of stencil3d_gb300 has it do, as cases that can be timed.

Four kinds of program call the library:

  march  fields live on the device: a context is filled once, then advanced
         `steps` steps per call and both time levels are copied out into device
         arrays of the reference layout (a snapshot), again and again;
  shot   one simulation after another in one context: upload v, s and u from
         device arrays, `steps` steps, copy both levels out;
  call   the drop-in ITERATE call on host arrays, pinned or pageable;
  batch  many uneven grids of mixed stencil orders advancing together, then
         every grid's two levels copied out.

Fields follow the repository's workloads: "uniform" seeds every point, halos
included (the boundary is fixed: v carries u's halo), "blobs" sums eight
Gaussian blobs over a zero halo with v = u.  Mode W carries a Ricker source at
the grid centre.
"""
import ctypes as C
import math
import random

import numpy as np
import torch

import stencil3d_gb300 as S

VEL, DX, FREQ = 1500.0, 10.0, 15.0
# reference flops per point and step
FLOPS = {2: 2, 7: 12, 13: 29, 25: 41}
AXIS = {7: (1.0,), 13: (0.3, 0.2), 25: (0.4, 0.3, 0.2, 0.1)}


def listed():
    def one(name, kind, points, mode, storage, xs, ys, zs, steps, init="uniform", **more):
        return dict(name=name, kind=kind, points=points, mode=mode, storage=storage, xs=xs, ys=ys,
                    zs=zs, steps=steps, init=init, **more)

    return [
        # a small source-gather box between two snapshots: launches and latency
        one("wave7_64", "march", 7, "wave", "f32", 64, 64, 64, 20),
        # the plain 7-point method at its stated size and length
        one("wave7_256", "march", 7, "wave", "f32", 256, 256, 256, 20),
        # one shot after another on a grid that no tile divides
        one("wave13_ragged", "shot", 13, "wave", "f32", 301, 187, 423, 20),
        # the 25-point method, 4-point halos, a snapshot every 40 steps
        one("wave25_528", "march", 25, "wave", "f32", 528, 528, 528, 40),
        # the headline workload
        one("wave25_1024", "march", 25, "wave", "f32", 1024, 1024, 1024, 20, "blobs"),
        # the reference's own update on resident fields
        one("ref25_512", "march", 25, "ref", "f32", 512, 512, 512, 20),
        # the reference's program as it stands: ITERATE on ordinary host arrays
        one("ref7_call_256", "call", 7, "ref", "f32", 256, 256, 256, 20, pinned=False),
        # a solver that keeps its arrays in pinned host memory
        one("wave25_call_512", "call", 25, "wave", "f32", 512, 512, 512, 20, "blobs", pinned=True),
        # the precision form at its stated size
        one("f16_wave25_1024", "march", 25, "wave", "f16", 1024, 1024, 1024, 20, "blobs"),
        # the hi/lo pair, shot after shot
        one("f16hl_wave25_512", "shot", 25, "wave", "f16_hl", 512, 512, 512, 20, "blobs"),
        # the double run that judges drift
        one("f64_wave25_256", "march", 25, "wave", "f64", 256, 256, 256, 10),
        # independent shots of uneven sizes and mixed orders
        dict(name="batch_24", kind="batch", grids=24, pick=2024, low=64, high=320, steps=50,
             schedule="graph"),
    ]


def _log(rng, lo, hi):
    return math.exp(rng.uniform(math.log(lo), math.log(hi)))


def _sizes(rng, points):
    """Three axes of about `points` points in all, none of them alike."""
    edge = points ** (1.0 / 3.0)
    a, b = _log(rng, 0.6, 1.6), _log(rng, 0.6, 1.6)
    return [max(9, int(round(edge * f))) for f in (a, b, 1.0 / (a * b))]


def draw(rng):
    r = rng.random()
    if r < 0.1:
        return dict(kind="batch", grids=rng.randint(3, 28), pick=rng.randint(1, 10 ** 6), low=48,
                    high=rng.randint(96, 288), steps=rng.randint(10, 60),
                    schedule=rng.choice(["graph", "pipelined", "persistent"]))
    if r < 0.5:  # FP32 wave on resident fields
        kind, mode, storage = rng.choice(["march", "march", "shot"]), "wave", "f32"
        pts, most, steps = rng.choice([7, 13, 25]), _log(rng, 40 ** 3, 800 ** 3), rng.randint(6, 40)
    elif r < 0.6:
        kind, mode, storage = "march", "ref", rng.choice(["f32", "f32", "f64"])
        pts, most, steps = rng.choice([2, 7, 13, 25]), _log(rng, 40 ** 3, 560 ** 3), rng.randint(1, 24)
        if storage == "f64":
            most = min(most, 220.0 ** 3)
    elif r < 0.75:  # the drop-in call
        kind, storage, mode = "call", "f32", rng.choice(["ref", "wave"])
        pts, most, steps = rng.choice([7, 13, 25]), _log(rng, 48 ** 3, 400 ** 3), rng.randint(2, 24)
    elif r < 0.92:  # 16-bit storage
        kind, mode = rng.choice(["march", "shot"]), "wave"
        storage = rng.choice(["f16", "f16", "bf16", "f16_hl", "f16_hl", "f16_hilo"])
        pts, most, steps = rng.choice([7, 13, 25]), _log(rng, 64 ** 3, 640 ** 3), rng.randint(6, 30)
    else:
        kind, mode, storage = rng.choice(["march", "shot"]), "wave", "f64"
        pts, most, steps = rng.choice([7, 13, 25]), _log(rng, 40 ** 3, 260 ** 3), rng.randint(2, 12)
    xs, ys, zs = _sizes(rng, most)
    sixteen = storage in ("f16", "bf16", "f16_hl", "f16_hilo")
    case = dict(kind=kind, points=pts, mode=mode, storage=storage, xs=xs, ys=ys, zs=zs, steps=steps,
                init="blobs" if sixteen or (mode == "wave" and rng.random() < 0.4) else "uniform")
    if kind == "call":
        case["pinned"] = rng.random() < 0.5
    return case


# ---------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------
def _dt(points):
    return 1e-3 if points == 7 else 5e-4


def _grid(case):
    return S.Grid(case["xs"], case["ys"], case["zs"], 4, 4, 16 if case["kind"] == "call" else 4)


def _shape(case):
    zh = 16 if case["kind"] == "call" else 4
    return (case["xs"] + 8, case["ys"] + 8, case["zs"] + 2 * zh), zh


def _inner(a, zh):
    return a[4:-4, 4:-4, zh:-zh]


def _device():
    return torch.device("cuda" if torch.cuda.is_available() else "cpu")


def _blobs(shape, zh, seed, dtype):
    """Eight seeded Gaussian blobs (20 cells wide, narrower on small grids) over a zero halo."""
    dev, rng = _device(), random.Random(seed)
    n = (shape[0] - 8, shape[1] - 8, shape[2] - 2 * zh)
    width = min(20.0, 0.15 * min(n))
    lines, amps = [[], [], []], []
    for _ in range(8):
        for ax in range(3):
            x = torch.arange(n[ax], device=dev, dtype=torch.float64) - rng.random() * n[ax]
            lines[ax].append(torch.exp(-0.5 * (x / width) ** 2))
        amps.append(2.0 * rng.random() - 1.0)
    a, b, c = (torch.stack(v).to(dtype) for v in lines)
    u = torch.zeros(shape, device=dev, dtype=dtype)
    inner = _inner(u, zh)
    for q in range(8):
        inner += amps[q] * (a[q][:, None] * b[q])[:, :, None] * c[q]
    return u


def _fields(case, seed):
    """v, s and u in the reference layout, on the device."""
    shape, zh = _shape(case)
    dev = _device()
    dtype = torch.float64 if case["storage"] == "f64" else torch.float32
    if case["init"] == "blobs":
        u = _blobs(shape, zh, seed, dtype)
        return u.clone(), torch.zeros_like(u), u
    g = torch.Generator(device=dev)
    g.manual_seed(seed)

    def rand(lo, hi):
        x = torch.rand(shape, generator=g, device=dev, dtype=dtype)
        return x.mul_(hi - lo).add_(lo)

    if case["mode"] == "ref":
        return rand(-1.0, 1.0), rand(0.5, 1.5), rand(-1.0, 1.0)
    u, v = rand(-1e-3, 1e-3), rand(-1e-3, 1e-3)
    w = u.clone()  # the fixed boundary is u's in both levels
    _inner(w, zh).copy_(_inner(v, zh))
    return w, torch.zeros_like(u), u


def _batch_specs(case):
    """Sizes, orders and source points of a batch's grids, from its `pick`."""
    rng = random.Random(case["pick"])
    specs = []
    for _ in range(case["grids"]):
        n = [rng.randint(case["low"], case["high"]) for _ in range(3)]
        specs.append((dict(kind="march", points=rng.choice([7, 13, 25]), mode="wave", storage="f32",
                           xs=n[0], ys=n[1], zs=n[2], init="uniform"),
                      tuple(rng.randrange(x) for x in n)))
    return specs


# ---------------------------------------------------------------------------
# the calls
# ---------------------------------------------------------------------------
def _check(status):
    if status != 0:
        raise S.St3dError(status, S.last_error())


def _upload(st, v, s, u):
    """Reference-layout device arrays into a context (st3d_upload takes them as they are)."""
    _check(S.lib().st3d_upload(st.handle, *(C.c_void_p(x.data_ptr()) for x in (v, s, u))))


def _download(st, v, u):
    _check(S.lib().st3d_download(st.handle, C.c_void_p(v.data_ptr()),
                                 C.c_void_p(u.data_ptr()) if u is not None else None))


def prepare(case, seed):
    if case["kind"] == "batch":
        specs = _batch_specs(case)
        grids = [_grid(c) for c, _ in specs]
        batch = S.Batch(grids, [c["points"] for c, _ in specs], dt=[_dt(c["points"]) for c, _ in specs],
                        srcs=[p for _, p in specs])
        outs = []
        for i, (c, _) in enumerate(specs):
            v, s, u = _fields(c, seed * 1000 + i)
            torch.cuda.current_stream().synchronize()
            _upload(batch.context(i), v, s, u)
            batch.context(i).synchronize()
            outs.append((v, u))
        return dict(case=case, batch=batch, outs=outs)
    v, s, u = _fields(case, seed)
    state = dict(case=case, zh=_shape(case)[1], grid=_grid(case))
    wave = case["mode"] == "wave"
    if case["kind"] == "call":
        host = [torch.empty(x.shape, dtype=x.dtype, pin_memory=case["pinned"]) for x in (v, s, u)]
        for h, x in zip(host, (v, s, u)):
            h.copy_(x)
        state["host"] = [h.numpy() for h in host]
        if case["pinned"] or wave:
            kw = dict(dt=_dt(case["points"])) if wave else {}
            state["st"] = S.Stencil(state["grid"], case["points"], case["mode"], "f32", **kw)
        return state
    kw = dict(dt=_dt(case["points"])) if wave else {}
    state["st"] = st = S.Stencil(state["grid"], case["points"], case["mode"], case["storage"], **kw)
    state["out"] = (v.clone(), u.clone() if wave else None)
    torch.cuda.current_stream().synchronize()
    if case["kind"] == "shot":
        state["in"] = (v, s, u)
    else:
        _upload(st, v, s, u)
        st.synchronize()
    return state


def run(state):
    case = state["case"]
    if case["kind"] == "batch":
        batch = state["batch"]
        batch.iterate(case["steps"], case["schedule"])
        for i, (v, u) in enumerate(state["outs"]):
            _download(batch.context(i), v, u)
        return [(_inner(v, 4), _inner(u, 4)) for v, u in state["outs"]]
    if case["kind"] == "call":
        v, s, u = state["host"]
        if "st" in state:
            state["st"].iterate_host(v, s, u, case["steps"])
        else:
            S.iterate_gb300(v, s, u, state["grid"], 64, 1, case["steps"], 1, points=case["points"])
    else:
        if case["kind"] == "shot":
            _upload(state["st"], *state["in"])
        state["st"].iterate(case["steps"])
        v, u = state["out"]
        _download(state["st"], v, u)
    out = {"v": _inner(v, state["zh"])}
    if case["mode"] == "wave":
        out["u"] = _inner(u, state["zh"])
    return out


# ---------------------------------------------------------------------------
# what a pass cannot do without, and its result in 64 bits
# ---------------------------------------------------------------------------
def work(case):
    if case["kind"] == "batch":
        each = [work(dict(c, steps=case["steps"])) for c, _ in _batch_specs(case)]
        return {k: sum(w[k] for w in each) for k in ("bytes", "flops")}
    points = float(case["xs"]) * case["ys"] * case["zs"]
    # one read of u, v (the time difference in the delta forms) and s, one
    # write of v, and of u where it changes
    wave = case["mode"] == "wave"
    per = {"f32": 4, "f64": 8, "f16": 2, "bf16": 2, "f16_hl": 2, "f16_hilo": 2}[case["storage"]]
    arrays = 5 if wave else 2 if case["points"] == 2 else 4
    size = arrays * per + {"f16_hl": 4, "f16_hilo": 4}.get(case["storage"], 0)
    return {"bytes": points * size, "flops": points * case["steps"] * FLOPS[case["points"]]}


def _f32(x):
    return float(np.float32(x))


def _weights(case):
    """(axis, radius, weight): the reference's coefficients, the y and z ones products of floats."""
    points, ref = case["points"], case["mode"] == "ref"
    dbl = ref and case["storage"] == "f64"
    out = []
    for r, w in enumerate(AXIS[points], 1):
        if points == 7:
            f = [0.5] * 3 if ref else [1.0] * 3
        elif dbl:
            f = [_f32(w), _f32(w) * _f32(1.1), _f32(w) * _f32(0.9)]
        else:
            f = [_f32(w), _f32(np.float32(w) * np.float32(1.1)), _f32(np.float32(w) * np.float32(0.9))]
        out += [(ax, r, f[ax]) for ax in range(3)]
    return out


def _pairs(x, zh, weights, centre):
    """sum of w * (x[-r] + x[+r]) + centre * x over the interior."""
    n = (x.shape[0] - 8, x.shape[1] - 8, x.shape[2] - 2 * zh)
    at = [4, 4, zh]

    def view(ax, d):
        o = list(at)
        o[ax] += d
        return x[o[0]:o[0] + n[0], o[1]:o[1] + n[1], o[2]:o[2] + n[2]]

    acc = view(0, 0) * centre
    for ax, r, w in weights:
        acc.add_(view(ax, -r), alpha=w)
        acc.add_(view(ax, r), alpha=w)
    return acc


def _ricker(t):
    a = (math.pi * FREQ * (t - 1.0 / FREQ)) ** 2
    return (1.0 - 2.0 * a) * math.exp(-a)


def _exact_one(case, seed, src):
    v, s, u = (x.double() for x in _fields(case, seed))
    zh = _shape(case)[1]
    points, steps = case["points"], case["steps"]
    vi = _inner(v, zh)
    if points == 2:
        vi.copy_(0.5 * (_inner(u, zh) + u[4:-4, 4:-4, zh + 1:u.shape[2] - zh + 1]))
        return {"v": vi}
    weights = _weights(case)
    if case["mode"] == "ref":
        coef0, k = {7: (1.5, 3.5), 13: (1.5, 3.5), 25: (1.25, 6.25)}[points]
        change = _pairs(u, zh, weights, coef0).mul_(_inner(s, zh)).sub_(_inner(u, zh), alpha=k)
        return {"v": vi.add_(change, alpha=steps)}
    dt = _dt(points)
    c1, c2 = (VEL * dt / DX) ** 2, dt * dt
    if case["storage"] != "f64":
        c1, c2 = _f32(c1), _f32(c2)
    centre = -2.0 * sum(w for _, _, w in weights)
    for n in range(steps):
        new = _pairs(u, zh, weights, centre).mul_(c1).add_(_inner(s, zh), alpha=c2)
        new[src] += c2 * _ricker(n * dt)
        new.add_(_inner(u, zh), alpha=2.0).sub_(_inner(v, zh))
        _inner(v, zh).copy_(new)
        u, v = v, u
    return {"v": _inner(v, zh), "u": _inner(u, zh)}


def exact(case, seed):
    if case["kind"] == "batch":
        got = [_exact_one(dict(c, steps=case["steps"]), seed * 1000 + i, p)
               for i, (c, p) in enumerate(_batch_specs(case))]
        return [(g["v"], g["u"]) for g in got]
    return _exact_one(case, seed, (case["xs"] // 2, case["ys"] // 2, case["zs"] // 2))
