"""What a user of the engine runs, as measurable cases.

Each case is one call pattern through the public entry points: steps of a bed
in the native engine (mixed and FP64, dry and wet, one packing or many, with
the formula or the learned closure), a state import with its list rebuild, the
round trip of a program that owns the state on the host, the reference's own
entry points in main.cpp's order, and the closure network's gradient and
inference.

Beds are cut from the stored packed bed of 200,000 log-normal spheres
(tests/golden/packed_wet200k.npz): its lowest n spheres inside a narrower
cylinder, or, beyond 200,000, square cuts of it side by side in a wider one.
The seed turns and mirrors the bed and draws small velocities and spins, those
of a settled bed that still creeps.  A pass is a few steps and the read of the
state: long enough to be the steps' time, short enough that a sliding contact,
whose friction law is decided by the last bit of its spring, does not make two
correct runs part.  What the FP32 force path produces (velocities, spins,
forces) is returned as float32, positions as the FP64 they are kept in.

exact() steps the same beds in plain torch FP64: the elasto-plastic contact
law, the capillary bridges, the cylinder wall and the integrator, on the pairs
near enough to meet within a pass."""
import ctypes as C
import math
from pathlib import Path

import numpy as np
import torch

from gpucode_gb300 import CapNet, Engine, Setup, _abi, configs
from gpucode_gb300.dropin import DropInDriver

BED = Path(__file__).resolve().parent.parent / "tests" / "golden" / "packed_wet200k.npz"
REAL = 2.0e-3  # the reduced length unit: the largest diameter [m]
SKIN = 0.05  # list skin, reduced
WARM = 2  # steps taken before a pass is measured: lists and histories exist
LIQUID = {"vol_min": 0.005, "vol_max": 0.02, "theta_max": math.pi / 6}
PI = 3.1415926  # the reference's


def listed():
    return [
        # the smallest configured run: 5,000 dry spheres, launch- and latency-bound
        dict(name="dry5k-steps", kind="steps", n=5000, wet=False, levels=1, steps=12),
        # the headline: the packed wet bed, steps chained on the device between outputs
        dict(name="wet200k-steps", kind="steps", n=200000, wet=True, levels=4, steps=6),
        # production size, larger than any cache
        dict(name="wet2m-steps", kind="steps", n=2000000, wet=True, levels=4, steps=4),
        # many independent packings of uneven sizes, every other one wet
        dict(name="ensemble-steps", kind="ensemble", systems=64, low=1000, high=8000, seed0=3, steps=5),
        # configured liquid (per-contact volumes and angles) with the learned closure
        dict(name="wet200k-closure", kind="closure", n=200000, steps=6),
        # a state moved by the caller: import, forced list rebuild, a few steps, export
        dict(name="wet200k-rebuild", kind="rebuild", n=200000, wet=True, levels=4, steps=2),
        # a program that owns the state: one step per host round trip
        dict(name="wet199k-advance", kind="advance", n=199001, wet=True, levels=4, steps=1),
        # validation runs in full FP64
        dict(name="wet200k-fp64", kind="fp64", n=200000, wet=True, levels=4, steps=2),
        # the reference's entry points as its unchanged main.cpp calls them
        dict(name="wet200k-dropin-fp64", kind="dropin", n=200000, wet=True, levels=4, steps=1, precision="fp64"),
        dict(name="wet200k-dropin-mixed", kind="dropin", n=200000, wet=True, levels=4, steps=3, precision="mixed"),
        # one training batch of the closure: the gradient
        dict(name="capnet-grad-8k", kind="grad", n=8192),
        # a trained closure checked on a sample set: FP32 network, warp tiles, tcgen05
        dict(name="capnet-infer-1m", kind="infer", n=1000003, modes="fp32,warp,tcgen05"),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["steps", "steps", "steps", "ensemble", "closure", "rebuild", "advance", "fp64", "dropin",
                       "grad", "infer"])
    if kind == "grad":
        return dict(kind=kind, n=_log(rng, 100, 500000))
    if kind == "infer":
        return dict(kind=kind, n=_log(rng, 1000, 2000000), modes=rng.choice(["fp32", "warp", "tcgen05"]))
    if kind == "ensemble":
        return dict(kind=kind, systems=rng.randint(2, 96), low=500, high=_log(rng, 1000, 12000),
                    seed0=rng.randint(0, 99), steps=rng.randint(2, 5))
    if kind == "closure":
        return dict(kind=kind, n=_log(rng, 2000, 400000), steps=rng.randint(2, 6))
    if kind == "dropin":
        precision = rng.choice(["fp64", "mixed"])
        return dict(kind=kind, n=_log(rng, 1000, 300000), wet=rng.random() < 0.6, levels=rng.randint(1, 4),
                    steps=1 if precision == "fp64" else rng.randint(1, 4), precision=precision)
    if kind in ("rebuild", "advance"):
        return dict(kind=kind, n=_log(rng, 1000, 600000), wet=rng.random() < 0.6, levels=rng.randint(1, 4),
                    steps=rng.randint(1, 4))
    if kind == "fp64":
        return dict(kind=kind, n=_log(rng, 1000, 300000), wet=rng.random() < 0.6, levels=rng.randint(1, 4), steps=2)
    n = _log(rng, 700, 1500000)
    wet = rng.random() < 0.6
    return dict(kind=kind, n=n, wet=wet, levels=rng.randint(1, 4),
                steps=rng.randint(2, 4) if n > 300000 else rng.randint(4, 6 if wet or n > 20000 else 12))


# ---------------- beds ----------------

_cache = {}


def _packed():
    if "packed" not in _cache:
        w = configs.load_bed(BED)
        _cache["packed"] = (w.pos_reduced, w.setup.rad)
    return _cache["packed"]


def _cut(n):
    """positions (axis at the origin, floor at 0), radii and cylinder radius of n spheres"""
    pos, rad = _packed()
    if n == len(rad):
        return pos, rad, 12.5
    R = 12.5 * (1.1 * (n / 200000) ** (1 / 3) if n < len(rad) else 1.05 * (n / 200000) ** 0.5)
    side = 17.6
    inside = (np.abs(pos[:, :2]).max(1) + rad) <= side / 2
    while True:
        p, r = pos, rad
        if n > len(rad):
            k = int(math.ceil(R / side + 0.5))
            p = np.concatenate([pos[inside] + (side * i, side * j, 0.0)
                                for i in range(-k, k + 1) for j in range(-k, k + 1)])
            r = np.tile(rad[inside], (2 * k + 1) ** 2)
        keep = np.flatnonzero(np.hypot(p[:, 0], p[:, 1]) + r <= R)
        if len(keep) >= n:
            keep = np.sort(keep[np.argsort(p[keep, 2], kind="stable")[:n]])
            return p[keep], r[keep], R
        R *= 1.04


def _input(n, levels, R, H, dia, wet):
    yldp = configs.yldp_for_yield_overlap(0.01, configs.E_YOUNG, configs.NU)
    cut = SKIN * dia.max() / dia.min()
    return configs.make_input(n, levels, REAL, cut, R * REAL, H * REAL, configs.RHO, configs.E_YOUNG, configs.NU,
                              configs.MU, 6.6e-6, yldp, 1 if wet else 0,
                              liquid=(0.072, 0.075, 5e-6) if wet else (0.0, 0.0, 0.0), dt=5e-7)


def _bed(n, wet, levels):
    key = (n, wet, levels)
    if key not in _cache:
        pos, rad, R = _cut(n)
        dia = 2.0 * rad * REAL
        H = float((pos[:, 2] + rad).max()) + 10.0
        inp = _input(n, levels, R, H, dia, wet)
        _cache[key] = (pos, configs.Workload(f"bed{n}", inp, dia, pos * REAL, Setup.build(inp, dia), 0))
    return _cache[key]


def _turn(pos, seed):
    """one of the square's eight symmetries"""
    p = pos.copy()
    if seed & 1:
        p[:, 0] = -p[:, 0]
    if seed & 2:
        p[:, 1] = -p[:, 1]
    return p[:, [1, 0, 2]] if seed & 4 else p


def _motion(n, seed):
    rng = np.random.default_rng(seed)
    return 5e-4 * rng.standard_normal((n, 3)), 2e-3 * rng.standard_normal((n, 3))


def _ensemble(case):
    """systems on a square grid of cylinders: (pos, system, cylinders, wet, workload)"""
    key = tuple(sorted((k, v) for k, v in case.items() if k not in ("name", "steps")))
    if key in _cache:
        return _cache[key]
    rng = np.random.default_rng(case["seed0"])
    ns = rng.integers(case["low"], case["high"] + 1, case["systems"])
    cuts = [_cut(int(n)) for n in ns]
    pitch = 2 * max(c[2] for c in cuts) + 3.0
    m = int(math.ceil(math.sqrt(len(cuts))))
    half = 0.5 * pitch * m
    top = max(float((c[0][:, 2] + c[1]).max()) for c in cuts) + 10.0
    pos, cyl = [], []
    for k, (p, r, R) in enumerate(cuts):
        cx, cy = pitch * (k % m + 0.5) - half, pitch * (k // m + 0.5) - half
        pos.append(p + (cx, cy, 0.0))
        c = _abi.CylinderBC()
        c.cir_x, c.cir_y, c.R, c.Tw, c.Bw, c.topv, c.btmv = cx, cy, R, top, 0.0, 0.0, 0.0
        cyl.append(c)
    pos = np.concatenate(pos)
    rad = np.concatenate([c[1] for c in cuts])
    system = np.repeat(np.arange(len(cuts), dtype=np.int32), ns)
    wet = np.arange(len(cuts), dtype=np.int32) % 2
    dia = 2.0 * rad * REAL
    inp = _input(len(rad), 4, half, top, dia, True)
    w = configs.Workload("ensemble", inp, dia, pos * REAL, Setup.build(inp, dia), 0)
    _cache[key] = (pos, system, cyl, wet, w)
    return _cache[key]


# ---------------- the closure network ----------------


def _closure_rows(n, seed):
    """raw features (separation, 8 V, contact angle, radius ratio) of wet pairs and the regression's outputs"""
    g = torch.Generator(device="cuda").manual_seed(seed)
    u = torch.rand((6, n), generator=g, device="cuda", dtype=torch.float64)
    rmin = 0.125 + 0.3 * u[0]
    vol = 8.0 * (0.005 + 0.015 * u[1]) * (PI / 6) * (2 * rmin) ** 3
    sep = 0.0025 * torch.exp(3.0 * torch.clamp(u[2] - 0.4, min=0.0))
    theta = 0.5 * (u[3] + u[4]) * LIQUID["theta_max"]
    ratio = 0.3 + 0.7 * u[5]
    x = torch.stack([sep, vol, theta, ratio], 1).float()
    xd = x.double()
    y = torch.stack([_willett(xd[:, 0], xd[:, 1], xd[:, 2]), _rupture(xd[:, 1] / 8.0, xd[:, 2])], 1).float()
    return x, y


def _features(x):
    return torch.stack([x[:, 0].log(), x[:, 1].log(), x[:, 2], x[:, 3]], 1)


def _net():
    """a fitted 4 -> 64 -> 64 -> 2 network (random hidden layers, least-squares head) and its standardisation"""
    if "net" not in _cache:
        x, y = (v.double() for v in _closure_rows(20000, 5))
        f = _features(x)
        norm = torch.cat([f.mean(0), f.std(0), y.mean(0), y.std(0), x.min(0).values * 0.98 - 1e-3,
                          x.max(0).values * 1.02])
        norm[12], norm[13] = 0.0024, float(x[:, 1].min()) * 0.5
        g = torch.Generator().manual_seed(9)
        w1 = (torch.randn(64, 4, generator=g, dtype=torch.float64) * 0.6).cuda()
        b1 = (torch.randn(64, generator=g, dtype=torch.float64) * 0.5).cuda()
        w2 = (torch.randn(64, 64, generator=g, dtype=torch.float64) * 0.3).cuda()
        b2 = (torch.randn(64, generator=g, dtype=torch.float64) * 0.5).cuda()
        p = [v.float().double() for v in (w1, b1, w2, b2)]
        nz = norm.float().double()
        h = torch.nn.functional.silu(torch.nn.functional.silu(((f - nz[:4]) / nz[4:8]) @ p[0].T + p[1]) @ p[2].T + p[3])
        a = torch.cat([h, torch.ones_like(h[:, :1])], 1)
        t = (y - nz[8:10]) / nz[10:12]
        s = torch.linalg.solve(a.T @ a + 1e-3 * len(x) * 1e-4 * torch.eye(65, device="cuda", dtype=torch.float64),
                               a.T @ t)
        params = torch.cat([p[0].reshape(-1), p[1], p[2].reshape(-1), p[3], s[:64].T.reshape(-1), s[64]])
        _cache["net"] = (params.float().cpu().numpy(), norm.float().cpu().numpy())
    return _cache["net"]


def _capnet():
    net = CapNet(seed=0)
    net.set(*_net())
    return net


def _net_forward(params, norm, x):
    """the network in FP64 on raw features: standardised outputs"""
    w1, b1, w2, b2, w3, b3 = torch.split(params, [256, 64, 4096, 64, 128, 2])
    f = (_features(x) - norm[:4]) / norm[4:8]
    h = torch.nn.functional.silu(f @ w1.view(64, 4).T + b1)
    h = torch.nn.functional.silu(h @ w2.view(64, 64).T + b2)
    return h @ w3.view(2, 64).T + b3


# ---------------- prepare / run ----------------


class _Host:
    """page-locked arrays the program reads the state into"""

    def __init__(self, n):
        self.all = torch.empty((4, n, 3), dtype=torch.float64).pin_memory()
        self.a = list(self.all)
        self.p = [C.c_void_p(t.data_ptr()) for t in self.a]

    def out(self):
        vel, ang, force = self.all[1:].float()
        return {"pos": self.a[0], "vel": vel, "angvel": ang, "force": force}


def prepare(case, seed):
    kind = case["kind"]
    if kind in ("grad", "infer"):
        x, y = _closure_rows(case["n"], seed)
        return {"case": case, "net": _capnet(), "x": x, "y": y}
    if kind == "ensemble":
        pos, system, cyl, wet, w = _ensemble(case)
        vel, ang = _motion(len(pos), seed)
        e = Engine(w.setup)
        e.set_systems(system, cyl, wet)
    else:
        n, wet = case["n"], case.get("wet", True)
        pos, w = _bed(n, wet, case.get("levels", 4))
        pos = _turn(pos, seed)
        vel, ang = _motion(n, seed)
        if kind == "dropin":
            d = DropInDriver(w, pos, vel, ang, torch)
            s = {"case": case, "drv": d}
            _precision(d.lib, case)
            for _ in range(WARM):
                d.step()
            return s
        if kind == "closure":
            e = Engine(w.setup, capillary="mlp")
            net = _capnet()
            e.set_liquid_model("per_contact", seed=2, **LIQUID)
            e.set_capnet(net)
        else:
            e = Engine(w.setup, precision="fp64" if kind == "fp64" else "mixed")
    e.set_state(pos, vel, ang)
    e.step(WARM)
    e.sync()
    s = {"case": case, "eng": e, "host": _Host(e.n)}
    if kind in ("advance", "rebuild"):
        _abi.check(e.lib.dem_get_state(e.h, *s["host"].p, None), "dem_get_state")
    return s


def _precision(lib, case):
    _abi.check(lib.dem_compat_set_precision(_abi.PREC_FP64 if case["precision"] == "fp64" else _abi.PREC_MIXED),
               "dem_compat_set_precision")


def run(state):
    case, kind = state["case"], state["case"]["kind"]
    if kind == "grad":
        g, loss = state["net"].grad(state["x"], state["y"])
        return {"grad": g, "loss": np.float32(loss)}
    if kind == "infer":
        modes = {"fp32": False, "warp": "warp", "tcgen05": "tcgen05"}
        return {m: state["net"].infer(state["x"], modes[m]) for m in case["modes"].split(",")}
    if kind == "dropin":
        d = state["drv"]
        _precision(d.lib, case)
        for _ in range(case["steps"]):
            d.step()
        f = (lambda t: t) if case["precision"] == "fp64" else (lambda t: t.float())
        return {"pos": d.pos, "vel": f(d.vel), "angvel": f(d.ang), "force": f(d.force), "mom": f(d.mom),
                "bridges": d.lqd}
    e, h = state["eng"], state["host"]
    lib = e.lib
    if kind == "advance":
        _abi.check(lib.dem_advance(e.h, *h.p, case["steps"]), "dem_advance")
        return h.out()
    if kind == "rebuild":
        _abi.check(lib.dem_set_state(e.h, *h.p[:3]), "dem_set_state")
    _abi.check(lib.dem_step(e.h, case["steps"]), "dem_step")
    _abi.check(lib.dem_get_state(e.h, *h.p, None), "dem_get_state")
    if kind == "fp64":
        return dict(zip(("pos", "vel", "angvel", "force"), h.a))
    return h.out()


def work(case):
    """per sphere and step: the state read and written (152 B) and, per pair of the packed bed's measured 4.33
    listed, 3.21 touching and 0.42 bridged pairs a sphere, its entry, 64-byte history read and written, and flag"""
    kind = case["kind"]
    if kind in ("grad", "infer"):
        passes = 3 if kind == "grad" else len(case["modes"].split(","))
        return {"bytes": 24.0 * case["n"] * (1 if kind == "grad" else passes) + 4 * 4610,
                "flops": 2.0 * 4480 * passes * case["n"]}
    n = case["n"] if "n" in case else case["systems"] * 0.5 * (case["low"] + case["high"])
    pairs = 4.33 * 4 + 3.21 * 128 + 0.42 * 8
    return {"bytes": n * (case["steps"] * (152 + pairs) + 96.0 + (72.0 if kind in ("advance", "rebuild") else 0.0)),
            "flops": n * case["steps"] * (3.21 * 300 + 4.33 * 60 + 60) + (
                n * case["steps"] * 3.6 * 2 * 4480 if kind == "closure" else 0)}


# ---------------- exact: the same in torch FP64 ----------------


def _willett(s, v, t):
    """the capillary regression with its contact-angle terms (Willett et al. 2000)"""
    t2, L = t * t, v.log()
    f1 = ((-0.44507 + 0.050832 * t - 1.1466 * t2) + (-0.1119 - 0.000411 * t - 0.1490 * t2) * L
          + (-0.012101 - 0.0036456 * t - 0.01255 * t2) * L ** 2 + (-0.0005 - 0.0003505 * t - 0.00029076 * t2) * L ** 3)
    f2 = ((1.9222 - 0.57473 * t - 1.2918 * t2) + (-0.0668 - 0.1201 * t - 0.22574 * t2) * L
          + (-0.0013375 - 0.0068988 * t - 0.01137 * t2) * L ** 2)
    f3 = ((1.268 - 0.01396 * t - 0.23566 * t2) + (0.198 + 0.092 * t - 0.06418 * t2) * L
          + (0.02232 + 0.02238 * t - 0.009853 * t2) * L ** 2 + (0.0008585 + 0.001318 * t - 0.00053 * t2) * L ** 3)
    f4 = ((-0.010703 + 0.073776 * t - 0.34742 * t2) + (0.03345 + 0.04543 * t - 0.09056 * t2) * L
          + (0.0018574 + 0.004456 * t - 0.006257 * t2) * L ** 2)
    ls = (s / v.sqrt()).log()
    return (f1 - f2 * (f3 * ls + f4 * ls * ls).exp()).exp()


def _rupture(V, t):
    return (1.0 + 0.5 * t) * 0.99 * V ** 0.33


_M64 = (1 << 64) - 1


def _mix64(z):
    z = (z ^ (z >> np.uint64(30))) * np.uint64(0xBF58476D1CE4E5B9)
    z = (z ^ (z >> np.uint64(27))) * np.uint64(0x94D049BB133111EB)
    return z ^ (z >> np.uint64(31))


def _unit(z):
    return torch.from_numpy((z >> np.uint64(11)).astype(np.float64) * 2.0 ** -53).cuda()


def _near_pairs(pos, rad, cut):
    """i < j of every pair with a gap below cut"""
    n = len(rad)
    size = float(2 * rad.max() + cut)
    c = ((pos - pos.min(0).values) / size).long() + 1
    dims = c.max(0).values + 2
    key = (c[:, 2] * dims[1] + c[:, 1]) * dims[0] + c[:, 0]
    cells = int(dims.prod())
    order = torch.argsort(key)
    count = torch.bincount(key, minlength=cells)
    start = torch.cumsum(count, 0) - count
    depth = int(count.max())
    found = []
    step = max(1, (1 << 26) // depth)
    for dz in (-1, 0, 1):
        for dy in (-1, 0, 1):
            for dx in (-1, 0, 1):
                other = key + int((dz * int(dims[1]) + dy) * int(dims[0]) + dx)
                for a in range(0, n, step):
                    o = other[a:a + step]
                    k = torch.arange(depth, device=pos.device)
                    at = start[o][:, None] + k
                    ok = k < count[o][:, None]
                    j = order[at.clamp(max=n - 1)]
                    i = torch.arange(a, a + len(o), device=pos.device)[:, None].expand_as(j)
                    ok &= j > i
                    i, j = i[ok], j[ok]
                    d = (pos[i] - pos[j]).norm(dim=1)
                    m = d - rad[i] - rad[j] < cut
                    found.append(torch.stack([i[m], j[m]]))
    return torch.cat(found, 1)


def _law(cal, mat, R, nrm, u, cpv, h, on, wall, dmp, dt):
    """the elasto-plastic normal force, damping, tangential spring and friction on the contacts `on`; h: the
    history, updated there.  Returns the normal force and the tangential force vector."""
    nrm = torch.where(on, nrm, torch.ones_like(nrm))
    sq = (R * nrm).sqrt()
    k = 4.0 / 3.0 * cal.emod
    st1 = nrm < h["pd"]
    st34 = ~st1 & (nrm < torch.maximum(h["nd"], h["mx"]))
    st2 = ~st1 & ~st34
    elastic = nrm < cal.ydsp_t * R if wall else nrm <= cal.ydsp_t * R
    fh = k * sq * nrm
    fp = cal.yforce_t * R * R + cal.ystiff_t * R * (nrm - cal.ydsp_t * R)
    rp = torch.where(elastic, R.expand_as(nrm), R * fh / fp)
    dp = torch.where(elastic, torch.zeros_like(nrm), nrm - (fp / (k * R.sqrt())).abs() ** (2.0 / 3.0))
    fN = torch.where(st2, torch.where(elastic, fh, fp),
                     torch.where(st34, k * h["pr"].sqrt() * (nrm - h["pd"]).clamp(min=0.0) ** 1.5,
                                 torch.zeros_like(nrm)))
    ld2 = st2 & on
    h["pr"] = torch.where(ld2, rp, h["pr"])
    h["pd"] = torch.where(ld2, dp, h["pd"])
    h["mx"] = torch.where(ld2, nrm, h["mx"])
    h["nd"] = torch.where(on, nrm, h["nd"])
    vn = (cpv * u).sum(1)
    fD = -2.0 * dmp * cal.emod * sq * vn
    vt = cpv - vn[:, None] * u
    eps = 1e-10 if wall else 1e-7
    old = h["d"]
    d = old - u * (u * old).sum(1, keepdim=True)
    ln = d.norm(dim=1)
    d = torch.where((ln > eps)[:, None], d * (old.norm(dim=1) / ln.clamp(min=1e-300))[:, None], d) + vt * dt
    dsmx = 3.0 * cal.sfrc * fN / (16.0 * (1 - cal.pois) * cal.emod / (4.0 - 2.0 * cal.pois) * sq)
    ln = d.norm(dim=1)
    stick = ln < dsmx
    ratio = torch.where(stick & (dsmx > eps), 1.0 - (1.0 - ln / dsmx.clamp(min=1e-300)).clamp(min=0.0) ** 1.5,
                        torch.ones_like(ln))
    slid = d * torch.where(ln > eps, dsmx / ln.clamp(min=1e-300), dsmx)[:, None]
    d = torch.where(stick[:, None], d, slid)
    h["d"] = torch.where(on[:, None], d, old)
    ln = d.norm(dim=1)
    way = torch.where(stick[:, None], d, vt)
    lw = way.norm(dim=1)
    fT = torch.where((lw > 1e-10)[:, None], way * (-cal.sfrc * fN * ratio / lw.clamp(min=1e-300))[:, None],
                     torch.zeros_like(way))
    return torch.where(on, fN, torch.zeros_like(fN)), torch.where(on, fD, torch.zeros_like(fD)), torch.where(
        on[:, None], fT, torch.zeros_like(fT))


def _history(n):
    z = lambda *s: torch.zeros(*s, device="cuda", dtype=torch.float64)  # noqa: E731
    return {"d": z(n, 3), "nd": z(n), "mx": z(n), "pr": z(n), "pd": z(n)}


def _steps64(s, rad, pos, vel, ang, steps, axis, wet=None, liquid=None, net=None):
    """`steps` steps of a bed in FP64.  axis: (centre x, centre y, radius) per sphere; wet: which spheres carry
    liquid; liquid: the per-contact model's seed (None: the reference's model); net: the closure's (params, norm)"""
    t = lambda a: torch.tensor(np.ascontiguousarray(a), device="cuda", dtype=torch.float64)  # noqa: E731
    x, v, w, r, ax = t(pos), t(vel), t(ang), t(rad), t(axis)
    n, dt, lq = len(r), s.prm.dt, s.lqd
    i, j = _near_pairs(x, r, s.prm.SearchGap * 1.02)
    ri, rj = r[i], r[j]
    R = ri * rj / (ri + rj)
    h, hw = _history(len(i)), [_history(n) for _ in range(3)]
    mass = (2 * r) ** 3
    inert = 0.1 * (2 * r) ** 5
    dpp, dpw = s.mat[0].dmpn, math.sqrt(s.mat[0].dmpn * s.mat[1].dmpn)
    bridged = torch.zeros(len(i), device="cuda", dtype=torch.bool)
    count = torch.zeros(n, device="cuda", dtype=torch.float64)
    wp = None if wet is None else torch.from_numpy(np.ascontiguousarray(wet)).cuda().bool()[i]
    if liquid is not None:
        lo, hi = i.cpu().numpy().astype(np.uint64), j.cpu().numpy().astype(np.uint64)
        with np.errstate(over="ignore"):
            one, seed = np.uint64(1), np.uint64(liquid)
            z = _mix64(_mix64(seed ^ (np.uint64(0xD1B54A32D192ED03) * (lo + one)))
                       + np.uint64(0x9E3779B97F4A7C15) * (hi + one))
            zt = _mix64(seed + np.uint64(0x9E3779B97F4A7C15) * (np.arange(n, dtype=np.uint64) + one))
        V = (LIQUID["vol_min"] + (LIQUID["vol_max"] - LIQUID["vol_min"]) * _unit(z)) * (PI / 6) * (
            2 * torch.minimum(ri, rj)) ** 3
        th = LIQUID["theta_max"] * _unit(zt)
        th = 0.5 * (th[i] + th[j])
    force = torch.zeros_like(x)
    mom = torch.zeros_like(x)
    for _ in range(steps):
        force, mom, nb = torch.zeros_like(x), torch.zeros_like(x), torch.zeros_like(count)
        force[:, 2] -= mass
        d = x[i] - x[j]
        dist = d.norm(dim=1)
        gap = dist - ri - rj
        u = d / dist[:, None]
        cpv = v[i] - v[j] - torch.linalg.cross(w[i] * ri[:, None] + w[j] * rj[:, None], u)
        fN, fD, fT = _law(s.cal, s.mat, R, -gap, u, cpv, h, gap < 0, False, dpp, dt)
        f = (fN + fD)[:, None] * u + fT
        if wp is not None:
            if liquid is None:
                share = lq.vol * mass / count.clamp(min=12.0)
                V = share[i] + share[j]
                th = torch.zeros_like(V)
            form = gap < 2 * lq.layer * (ri + rj)
            sep = gap.clamp(min=lq.gapmn)
            fc, rup = _willett(sep, 8 * V, th), _rupture(V, th)
            if net is not None:
                rows = torch.stack([sep, 8 * V, th, torch.minimum(ri, rj) / torch.maximum(ri, rj)], 1)
                box = ((rows >= net[1][12:16]) & (rows <= net[1][16:20])).all(1)
                y = _net_forward(net[0], net[1], rows) * net[1][10:12] + net[1][8:10]
                fc, rup = torch.where(box, y[:, 0], fc), torch.where(box, y[:, 1], rup)
            bridged = wp & (form | (bridged & (gap <= rup)))
            f = f - torch.where(bridged, 2 * PI * 2 * R * lq.stension * fc, torch.zeros_like(fc))[:, None] * u
            nb.index_add_(0, i, bridged.double())
            nb.index_add_(0, j, bridged.double())
        force.index_add_(0, i, f)
        force.index_add_(0, j, -f)
        tq = torch.linalg.cross(u, fT)
        mom.index_add_(0, i, -(ri + gap / 2)[:, None] * tq)
        mom.index_add_(0, j, -(rj + gap / 2)[:, None] * tq)
        rel = x[:, :2] - ax[:, :2]
        rho = rel.norm(dim=1)
        for kind in range(3):
            up = torch.zeros_like(x)
            if kind == 2:
                gw = ax[:, 2] - rho
                up[:, :2] = -rel / rho.clamp(min=1e-300)[:, None]
            else:
                gw = s.cyl.Tw - x[:, 2] if kind == 0 else x[:, 2] - s.cyl.Bw
                up[:, 2] = -1.0 if kind == 0 else 1.0
            cw = v - torch.linalg.cross(w * r[:, None], up)
            fN, fD, fT = _law(s.pwcal, s.mat, r, r - gw, up, cw, hw[kind], gw < r, True, dpw, dt)
            force += (fN + fD)[:, None] * up + fT
            mom += -(r - (r - gw) / 2)[:, None] * torch.linalg.cross(up, fT) * (gw < r)[:, None]
        count = nb
        v = v + force * (dt / mass)[:, None]
        x = x + v * dt
        w = w + mom * (dt / inert)[:, None]
    return {"pos": x, "vel": v, "angvel": w, "force": force, "mom": mom, "bridges": None}


def exact(case, seed):
    kind = case["kind"]
    if kind in ("grad", "infer"):
        x, y = _closure_rows(case["n"], seed)
        p, nz = (torch.from_numpy(a).cuda().double() for a in _net())
        if kind == "infer":
            out = _net_forward(p, nz, x.double()) * nz[10:12] + nz[8:10]
            return {m: out for m in case["modes"].split(",")}
        p.requires_grad_(True)
        loss = ((_net_forward(p, nz, x.double()) - (y.double() - nz[8:10]) / nz[10:12]) ** 2).sum() / case["n"]
        loss.backward()
        return {"grad": p.grad, "loss": loss.detach()}
    steps = WARM + case["steps"]
    if kind == "ensemble":
        pos, system, cyl, wet, w = _ensemble(case)
        vel, ang = _motion(len(pos), seed)
        axis = np.array([(c.cir_x, c.cir_y, c.R) for c in cyl])[system]
        out = _steps64(w.setup.s, w.setup.rad, pos, vel, ang, steps, axis, wet[system])
    else:
        pos, w = _bed(case["n"], case.get("wet", True), case.get("levels", 4))
        vel, ang = _motion(case["n"], seed)
        c = w.setup.s.cyl
        axis = np.tile((c.cir_x, c.cir_y, c.R), (case["n"], 1))
        net = tuple(torch.from_numpy(a).cuda().double() for a in _net()) if kind == "closure" else None
        out = _steps64(w.setup.s, w.setup.rad, _turn(pos, seed), vel, ang, steps, axis,
                       np.ones(case["n"], bool) if case.get("wet", True) else None, 2 if kind == "closure" else None,
                       net)
    return out if kind == "dropin" else {k: out[k] for k in ("pos", "vel", "angvel", "force")}
