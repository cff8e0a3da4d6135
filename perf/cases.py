"""What this framework is used for, as calls that can be timed and compared.

Walks of the four tiling models through the Tiler classes (host tilings in and
out, as the reference's Walk; or resident on the device with height
statistics), exact samples by coupling from the past, batches of many chains,
the six-vertex walk, training of the coordinate MLP, and the set-up of a warm
start.  Sizes come from the benchmark (the 500-hexagon, the Aztec diamond of
order 100, the mixed batch, the six-vertex grid of n = 1000, the MLP's batch
of 16,384), from the tests, or are generic.
"""
from __future__ import annotations

import math

import numpy as np
import torch

import randomtilings_b200 as rt
from randomtilings_b200 import builders, workloads
from randomtilings_b200.heights import HeightPlan
from randomtilings_b200.mlp import NPARAM, CoordinateMLP
from randomtilings_b200.project import project_heights

RNG = {"tinymt": rt.RT_RNG_TINYMT, "philox": rt.RT_RNG_PHILOX, "planes": rt.RT_RNG_PLANES}


def listed():
    return [
        # The smallest call: a demonstration-sized diamond, a few hundred
        # steps, the reference's generator, the tiling in host memory.
        {"name": "walk domino 24", "kind": "walk", "model": "domino", "rng": "tinymt", "a": 24, "b": 0, "c": 0, "steps": 400},
        # The bit-exact replay the reference's users know: the order-100 Aztec
        # diamond, 10,000 checkerboard sweeps.
        {"name": "walk domino 100", "kind": "walk", "model": "domino", "rng": "tinymt", "a": 100, "b": 0, "c": 0, "steps": 20000},
        # The benchmark's headline walk: the 500 x 500 x 500 hexagon, 3,000
        # colour steps a call.
        {"name": "walk lozenge 500", "kind": "walk", "model": "lozenge", "rng": "tinymt", "a": 500, "b": 500, "c": 500, "steps": 3000},
        # Volume-weighted lozenges on a ragged hexagon, counter-based draws
        # (how a warm-start dataset's large q chains run).
        {"name": "walk qlozenge 190x131x83", "kind": "walk", "model": "qlozenge", "rng": "philox", "a": 190, "b": 131, "c": 83, "steps": 3000},
        # Rectangle-triangle tilings of the side-64 hexagon, bit-exact.
        {"name": "walk recttri 64", "kind": "walk", "model": "recttri", "rng": "tinymt", "a": 64, "b": 0, "c": 0, "steps": 1500},
        # Bibone tilings of the side-64 hexagon, bit-exact.
        {"name": "walk tridimer 64", "kind": "walk", "model": "tridimer", "rng": "tinymt", "a": 64, "b": 0, "c": 0, "steps": 600},
        # One segment of a large chain kept on the device: bit-plane walk, then
        # its heights added to the running sums.
        {"name": "sample domino 1000", "kind": "sample", "model": "domino", "rng": "planes", "a": 1000, "b": 0, "c": 0, "steps": 4000},
        # An exact sample by coupling from the past, bit-exact draws.
        {"name": "cftp domino 32", "kind": "cftp", "model": "domino_hb", "rng": "tinymt", "a": 32, "b": 0, "c": 0, "steps": 1024},
        # A group of chains of all four models and uneven sizes in one graph,
        # between two samples of their tilings.
        {"name": "batch 256", "kind": "batch", "chains": 256, "steps": 200},
        # The six-vertex walk of the benchmark's size.
        {"name": "sixv 1000", "kind": "sixv", "a": 1000, "steps": 100},
        # Training the warm start's network at the batch it is trained with.
        {"name": "train 16384", "kind": "train", "rows": 200000, "batch": 16384, "steps": 30},
        # Setting up a warm start on an evaluation domain: extremal tilings,
        # the network's forward pass over every vertex, the projection of a
        # height surface, and the heights of a tiling.
        {"name": "warm domino 400", "kind": "warm", "model": "domino", "a": 400, "b": 0, "c": 0},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _sizes(rng, model, rng_kind):
    """Sides of a walk's domain: TinyMT keeps generator states on chip, which
    bounds its lattices; the counter-based modes go further."""
    if model in ("domino", "domino_hb"):
        return _log_int(rng, 8, 600 if rng_kind == "tinymt" else 1000), 0, 0
    if model in ("lozenge", "qlozenge"):
        hi = 500 if rng_kind == "tinymt" else 600
        return tuple(_log_int(rng, 6, hi) for _ in range(3))
    return _log_int(rng, 7, 64), 0, 0


def draw(rng):
    kind = rng.choice(["walk", "walk", "walk", "walk", "walk", "walk", "sample", "cftp", "batch", "sixv", "train", "warm"])
    if kind == "walk":
        model = rng.choice(["domino", "domino_hb", "lozenge", "qlozenge", "recttri", "tridimer"])
        modes = ["tinymt", "tinymt", "philox"] + (["planes"] if model in ("domino", "domino_hb", "lozenge") else [])
        mode = rng.choice(modes)
        a, b, c = _sizes(rng, model, mode)
        steps = _log_int(rng, 30, 600) if model == "tridimer" else _log_int(rng, 30, 3000)
        return {"kind": kind, "model": model, "rng": mode, "a": a, "b": b, "c": c, "steps": steps}
    if kind == "sample":
        model = rng.choice(["domino", "domino_hb", "lozenge"])
        a, b, c = _sizes(rng, model, "planes")
        return {"kind": kind, "model": model, "rng": rng.choice(["planes", "philox"]), "a": a, "b": b, "c": c,
                "steps": _log_int(rng, 100, 3000)}
    if kind == "cftp":
        model = rng.choice(["domino_hb", "lozenge"])
        a, b, c = (_log_int(rng, 6, 40), 0, 0) if model == "domino_hb" else tuple(_log_int(rng, 4, 16) for _ in range(3))
        return {"kind": kind, "model": model, "rng": rng.choice(["tinymt", "philox", "planes"]), "a": a, "b": b, "c": c,
                "steps": 1024}
    if kind == "batch":
        return {"kind": kind, "chains": _log_int(rng, 8, 256), "steps": _log_int(rng, 10, 200)}
    if kind == "sixv":
        return {"kind": kind, "a": _log_int(rng, 10, 1000), "steps": _log_int(rng, 5, 100)}
    if kind == "train":
        return {"kind": kind, "rows": _log_int(rng, 3000, 200000), "batch": _log_int(rng, 200, 16384), "steps": _log_int(rng, 3, 30)}
    model = rng.choice(["domino", "lozenge"])
    a, b, c = (_log_int(rng, 10, 400), 0, 0) if model == "domino" else tuple(_log_int(rng, 8, 250) for _ in range(3))
    return {"kind": kind, "model": model, "a": a, "b": b, "c": c}


def _domain(model, a, b, c):
    if model in ("domino", "domino_hb"):
        return rt.DominoTiler.AztecDiamond(a)
    return rt.LozengeTiler.Hexagon(a, b, c)


def _extremes(model, d):
    cls = rt.DominoTiler if model in ("domino", "domino_hb") else rt.LozengeTiler
    return cls.MinTiling(d), cls.MaxTiling(d)


def _tiler(model, mode):
    if model in ("domino", "domino_hb"):
        return rt.DominoTiler(rng=RNG[mode], kernel=rt.RT_KERNEL_CFTP if model == "domino_hb" else rt.RT_KERNEL_DEFAULT)
    if model == "lozenge":
        return rt.LozengeTiler(rng=RNG[mode])
    if model == "qlozenge":
        return rt.LozengeTiler(rng=RNG[mode], kernel=rt.RT_KERNEL_QWEIGHT, q=0.99)
    return rt.RectTriangleTiler(rng=RNG[mode]) if model == "recttri" else rt.TriangleDimerTiler(rng=RNG[mode])


def _start(model, a, b, c):
    if model == "recttri":
        return rt.RectTriangleTiler.minHex(a)
    if model == "tridimer":
        return rt.TriangleDimerTiler.BiboneHexagon(a)
    return _extremes(model, _domain(model, a, b, c))[0]


def _mlp_rows(seed, n):
    """Features as the warm start's (positions in the unit square, model flag,
    ratios, weight, 16 / side) and a smooth target surface in [0, 1]."""
    g = np.random.default_rng(seed)
    x = np.zeros((n, 8), dtype=np.float32)
    x[:, :2] = g.uniform(-1, 1, (n, 2))
    flag = g.integers(0, 2, n)
    x[:, 2] = 2 * flag - 1
    x[:, 3:6] = g.uniform(-0.5, 0.5, (n, 3)) * (1 - flag)[:, None]
    x[:, 3] += flag * (2 * g.integers(0, 2, n) - 1)
    x[:, 6] = g.uniform(0, 2, n) * (1 - flag)
    x[:, 7] = 16.0 / g.uniform(16, 384, n)
    r2 = x[:, 0] ** 2 + x[:, 1] ** 2
    t = 1.0 / (1.0 + np.exp(-(1.5 * x[:, 0] - 1.2 * x[:, 1] * x[:, 2] + 0.6 * (1 - r2))))
    return x, t.astype(np.float32)


def _mlp_params(seed):
    """The state of a partly trained network: fan-in scaled weights, small biases."""
    g = np.random.default_rng(seed + 77)
    parts = []
    for rows, fan in ((128, 8), (128, 128), (128, 128), (1, 128)):
        parts.append(g.uniform(-1, 1, rows * fan) / math.sqrt(fan))
        parts.append(g.uniform(-0.05, 0.05, rows))
    return np.concatenate(parts).astype(np.float32)


def prepare(case, seed):
    k = case["kind"]
    if k in ("walk", "sample", "cftp"):
        m = case["model"]
        s = {"case": case, "tiler": _tiler(m, case["rng"]), "seed": seed * 1000003 % 2**31, "calls": 0}
        if k == "cftp":
            s["tmin"], s["tmax"] = _extremes(m, _domain(m, case["a"], case["b"], case["c"]))
        else:
            s["t"] = np.array(_start(m, case["a"], case["b"], case["c"]), dtype=np.int32)
        if k == "sample":
            d = _domain(m, case["a"], case["b"], case["c"])
            s["plan"] = HeightPlan(rt.RT_LOZENGE if m == "lozenge" else rt.RT_DOMINO, d)
            s["sums"] = torch.zeros(s["plan"].n ** 2, dtype=torch.int64, device="cuda")
            torch.cuda.synchronize()
            s["tiler"].upload(s["t"])
        return s
    if k == "batch":
        b = rt.Batch()
        on_device, on_host, at = [], [], 0
        for i in range(case["chains"]):
            model, t = workloads.mixed_chain(i)
            b.add(model, t, key=seed * 4096 + i)
            if model == rt.RT_TRIDIMER:  # their tilings are merged on the host
                on_host.append(i)
            else:
                on_device.append((i, 4 * at))
                at += len(t)
        b.run(8)  # the burn-in; the first run also settles the plan
        out = torch.empty(at, dtype=torch.int32, device="cuda")
        return {"case": case, "batch": b, "out": out, "on_device": on_device, "on_host": on_host}
    if k == "sixv":
        return {"case": case, "tiler": rt.SixVertexTiler(), "h": rt.SixVertexTiler.MinHeights(case["a"]), "seed": seed, "calls": 0}
    if k == "train":
        x, t = _mlp_rows(seed, case["rows"])
        net = CoordinateMLP()
        net.params = _mlp_params(seed)
        net.set_data(x, t)
        return {"case": case, "net": net, "seed": seed}
    m = case["model"]
    d = np.asarray(_domain(m, case["a"], case["b"], case["c"]), dtype=np.int32)
    model = rt.RT_LOZENGE if m == "lozenge" else rt.RT_DOMINO
    ext, _ = builders.extremal_tilings(model, d)
    lo, hi = np.minimum(ext["hmin"], ext["hmax"]), np.maximum(ext["hmin"], ext["hmax"])
    inside = lo != np.iinfo(np.int32).max
    g = np.random.default_rng(seed)
    n = math.isqrt(lo.size)
    x = _mlp_rows(seed, int(inside.sum()))[0]
    # A smooth surface between the extremal ones, as a trained network's.
    i, j = np.divmod(np.arange(n * n), n)
    f = 0.5 + 0.35 * np.sin(3.0 * i / n + g.uniform(0, 6)) * np.cos(2.5 * j / n + g.uniform(0, 6))
    target = np.zeros(n * n, dtype=np.float32)
    target[inside] = (lo + f * (hi.astype(np.float64) - lo))[inside]
    net = CoordinateMLP()
    net.params = _mlp_params(seed)
    out = {v: torch.empty(n * n, dtype=torch.int32, device="cuda") for v in ("tmin", "tmax", "hmin", "hmax", "h")}
    return {"case": case, "model": model, "d": d, "lo": lo, "hi": hi, "x": x, "target": target, "net": net, "out": out,
            "plan": HeightPlan(model, d)}


def run(s):
    case = s["case"]
    k = case["kind"]
    if k == "walk":
        s["calls"] += 1
        s["tiler"].Walk(s["t"], case["steps"], s["seed"] + s["calls"])
        return s["t"]
    if k == "sample":
        s["calls"] += 1
        tl = s["tiler"]
        tl.run(case["steps"], s["seed"] + s["calls"])
        s["plan"].accumulate(tl.device_tiling(), s["sums"].data_ptr(), tl.stream)
        tl.synchronize()
        return s["sums"]
    if k == "cftp":
        s["calls"] += 1
        t, st = s["tiler"].CFTP(s["tmax"], s["tmin"], first_steps=case["steps"], master_seed=s["seed"] + s["calls"])
        return [t, st["total_steps"]]
    if k == "batch":
        b = s["batch"]
        b.run(case["steps"])
        for i, at in s["on_device"]:
            b.device_tiling(i, s["out"].data_ptr() + at)
        return [s["out"], np.concatenate([b.download(i) for i in s["on_host"]])]
    if k == "sixv":
        s["calls"] += 1
        s["tiler"].Walk(s["h"], case["steps"], s["seed"] + s["calls"])
        return s["h"]
    if k == "train":
        loss = s["net"].train(case["steps"], batch=case["batch"], lr=2e-3, seed=s["seed"])
        return [loss, s["net"].params]
    o = s["out"]
    builders.extremal_tilings_device(s["model"], s["d"], *(o[v].data_ptr() for v in ("tmin", "tmax", "hmin", "hmax")))
    y = s["net"].predict(s["x"])
    h, _ = project_heights(s["model"], s["d"], s["lo"], s["hi"], s["target"])
    s["plan"].heights(o["tmax"].data_ptr(), o["h"].data_ptr())
    return [o["tmin"], o["tmax"], o["hmin"], o["hmax"], y, h, o["h"]]


def _side(model, a, b, c):
    """About the side of the tiling array."""
    if model in ("domino", "domino_hb"):
        return 2 * a + 6
    if model in ("lozenge", "qlozenge"):
        return max(a + b, b + c, a + c) + 8
    return 2 * a + 8


_ATTEMPT = 50  # integer operations of one flip attempt: the draw, the neighbours, the rule
_MLP_FLOPS = 2 * (8 * 128 + 2 * 128 * 128 + 128)  # one row's forward pass


def work(case):
    k = case["kind"]
    if k in ("walk", "sample", "cftp"):
        m = case["model"]
        n2 = _side(m, case["a"], case["b"], case["c"]) ** 2
        steps = case["steps"] * (2 if k == "cftp" else 1)
        attempts = n2 // (2 if m.startswith("domino") else 3 if m != "tridimer" else 4)
        return {"bytes": 8 * n2 * (2 if k == "sample" else 1), "flops": _ATTEMPT * attempts * steps}
    if k == "batch":
        # Mean attempts a sweep and array size of the four kinds of chain.
        return {"bytes": 8 * 40000 * case["chains"], "flops": _ATTEMPT * 140000 * case["chains"] * case["steps"]}
    if k == "sixv":
        return {"bytes": 8 * (case["a"] + 1) ** 2, "flops": _ATTEMPT * case["a"] ** 2 * case["steps"]}
    if k == "train":
        return {"bytes": (36 * case["batch"] + 7 * 4 * NPARAM) * case["steps"], "flops": 3 * _MLP_FLOPS * case["batch"] * case["steps"]}
    n2 = _side(case["model"], case["a"], case["b"], case["c"]) ** 2
    rows = n2 // 2 if case["model"] == "domino" else (3 * n2) // 4
    return {"bytes": 36 * rows + 40 * n2, "flops": _MLP_FLOPS * rows}


# --- the values in 64 bits ---------------------------------------------------

_C = math.sqrt(2 / math.pi)
_SHAPES = ((128, 8), (128,), (128, 128), (128,), (128, 128), (128,), (128,), (1,))


def _gelu(z):
    return 0.5 * z * (1 + torch.tanh(_C * (z + 0.044715 * z ** 3)))


def _unflatten(p):
    out, at = [], 0
    for shape in _SHAPES:
        n = math.prod(shape)
        out.append(p[at:at + n].reshape(shape))
        at += n
    return out


def _forward(p, x):
    w0, b0, w1, b1, w2, b2, w3, b3 = _unflatten(p)
    h = _gelu(x @ w0.T + b0)
    h = _gelu(h @ w1.T + b1)
    h = _gelu(h @ w2.T + b2)
    return h @ w3 + b3


def _philox(c0, c1, c2, c3, k0, k1):
    """Philox4x32-10: the counters' first two output words."""
    u = np.uint64
    lo = u(0xFFFFFFFF)
    c = [np.asarray(v, dtype=u) for v in (c0, c1, c2, c3)]
    for _ in range(10):
        p0, p1 = u(0xD2511F53) * c[0], u(0xCD9E8D57) * c[2]
        c = [(p1 >> u(32)) ^ c[1] ^ u(k0), p1 & lo, (p0 >> u(32)) ^ c[3] ^ u(k1), p0 & lo]
        k0, k1 = (k0 + 0x9E3779B9) & 0xFFFFFFFF, (k1 + 0xBB67AE85) & 0xFFFFFFFF
    return c[0], c[1]


def exact(case, seed):
    k = case["kind"]
    if k not in ("train", "warm"):
        return None  # integer states: nothing is rounded
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    p = torch.tensor(_mlp_params(seed), dtype=torch.float64, device=dev)
    if k == "warm":
        d = _domain(case["model"], case["a"], case["b"], case["c"])
        rows = HeightPlan(rt.RT_LOZENGE if case["model"] == "lozenge" else rt.RT_DOMINO, d).vertices
        x = torch.tensor(_mlp_rows(seed, rows)[0], dtype=torch.float64, device=dev)
        y = torch.cat([_forward(p, v) for v in x.split(1 << 18)])
        return [None, None, None, None, y, None, None]
    x, t = (torch.tensor(v, dtype=torch.float64, device=dev) for v in _mlp_rows(seed, case["rows"]))
    m1, m2 = torch.zeros_like(p), torch.zeros_like(p)
    loss = 0.0
    row = np.arange(case["batch"])
    for step in range(case["steps"]):
        w0, w1 = _philox(row, np.full_like(row, step), 0 * row, np.full_like(row, 0x4D4C50), seed & 0xFFFFFFFF, seed >> 32)
        at = torch.from_numpy((((w0 << np.uint64(32)) | w1) % np.uint64(case["rows"])).astype(np.int64)).to(dev)
        q = p.detach().requires_grad_(True)
        e = ((_forward(q, x[at]) - t[at]) ** 2).mean()
        (g,) = torch.autograd.grad(e, q)
        loss = float(e.detach())
        m1, m2 = 0.9 * m1 + 0.1 * g, 0.999 * m2 + 0.001 * g * g
        p = p - 2e-3 * (m1 / (1 - 0.9 ** (step + 1))) / (torch.sqrt(m2 / (1 - 0.999 ** (step + 1))) + 1e-8)
    return [loss, p]
