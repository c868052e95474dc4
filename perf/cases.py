"""Performance cases: the optical-flow work a program gives this library, through its Python entry points.

listed() names the cases, draw() gives more of the same ranges, prepare() makes the inputs and handles a program holds before
the call, run() is one pass, work() the bytes and operations it cannot do without, exact() its result in 64 bits with plain
torch.  Frames are seeded synthetic pairs (blurred-noise textures under affine and independent motion, value noise under a
vortex) as in the benchmark and the training set."""
from __future__ import annotations

import math
import os
import sys

import numpy as np
import torch
import torch.nn.functional as F

_PKG = os.path.join(os.getcwd(), "sycl-optic-flow_b200")
if _PKG not in sys.path:
    sys.path.insert(0, _PKG)

import oflow  # noqa: E402
from oflow import synth_gpu, warmstart  # noqa: E402

MIXED_SIZES = ((320, 240), (640, 480), (1024, 436), (1280, 720), (1920, 1080))
MAX_PX = 32 * 1024 * 436  # pixels per call of the largest cases


# ------------------------------------------------------------------ cases
def _tvl1(**k):
    return dict({"kind": "tvl1", "dtype": "u8", "host": False, "nscales": 100, "iters": 300, "tuned": False}, **k)


def listed():
    return [
        # a single call on small, odd-sized host frames with the reference's default parameters: latency, launches
        _tvl1(name="tvl1_odd_pair_host", w=161, h=117, pairs=1, dtype="f32", host=True),
        # one VGA pair already on the device, default parameters: the ordinary call of an interactive program
        _tvl1(name="tvl1_vga_pair", w=640, h=480, pairs=1),
        # the benchmark's throughput call: 32 pairs of 1024x436, 5 scales, 5 warps, at most 50 iterations, autotuned
        _tvl1(name="tvl1_batch", w=1024, h=436, pairs=32, nscales=5, iters=50, tuned=True),
        # full-HD float frames, a few at a time (film post-production)
        _tvl1(name="tvl1_hd", w=1920, h=1080, pairs=4, dtype="f32", nscales=5, iters=50),
        # a live 720p video: each new pinned host frame against the previous one, and the demo's colour image of the flow
        {"name": "stream_color", "kind": "stream", "w": 1280, "h": 720, "lanes": 1, "nscales": 5, "iters": 50},
        # a batch of uneven sizes, half Horn-Schunck (200 sweeps) and half TV-L1, as one schedule
        {"name": "mixed_batch", "kind": "mixed", "per_size": 2, "sizes": 5},
        # Horn-Schunck at its benchmark configuration: 64 pairs of 320x240, one level, 200 sweeps, autotuned
        {"name": "hs_batch", "kind": "hs", "w": 320, "h": 240, "pairs": 64, "dtype": "f32", "alpha": 15.0, "levels": 1,
         "warps": 1, "sweeps": 200, "tuned": True},
        # Horn-Schunck with the reference demo's parameters on one odd-sized pair
        {"name": "hs_pyramid_pair", "kind": "hs", "w": 641, "h": 479, "pairs": 1, "dtype": "u8", "alpha": 0.2, "levels": 5,
         "warps": 3, "sweeps": 150, "tuned": False},
        # pyramidal Lucas-Kanade at its benchmark configuration: 64 pairs of 640x480, 3 levels of 3 refinements
        {"name": "pyrlk_batch", "kind": "pyrlk", "w": 640, "h": 480, "pairs": 64, "dtype": "f32", "spac": 3, "window": 5,
         "levels": 3, "iters": 3},
        # single-step Lucas-Kanade over a ring of 720p frames
        {"name": "lk_ring", "kind": "lk", "w": 1280, "h": 720, "spac": 5, "temp": 5, "window": 7},
        # one training step of the warm-start network (forward, backward, Adam) at its training batch
        {"name": "net_train", "kind": "train", "w": 1024, "h": 436, "pairs": 16},
        # TV-L1 started from the network's flow: 32 pairs, 2 warps of 20 iterations from scale 3
        {"name": "warm_batch", "kind": "warm", "w": 1024, "h": 436, "pairs": 32, "warps": 2, "iters": 20},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _size(rng, lo=64, hi=1920):
    w = _log(rng, lo, hi)
    return w, max(48, min(1080, int(w * rng.uniform(0.4, 1.0))))


def _count(rng, w, h, most, px=MAX_PX):
    return _log(rng, 1, max(1, min(most, px // (w * h))))


def draw(rng):
    kind = rng.choice(("tvl1", "tvl1", "tvl1", "stream", "mixed", "hs", "hs", "pyrlk", "lk", "train", "warm"))
    if kind == "tvl1":
        w, h = _size(rng)
        n, long = _count(rng, w, h, 32), rng.random() < 0.4
        if long:
            n = max(1, min(n, MAX_PX // 4 // (w * h)))
        return _tvl1(w=w, h=h, pairs=n, dtype=rng.choice(("u8", "f32")), host=n <= 2 and rng.random() < 0.3,
                     nscales=100 if long else 5, iters=300 if long else 50)
    if kind == "stream":
        w, h = _size(rng, 160, 1920)
        return {"kind": kind, "w": w, "h": h, "lanes": rng.choice((1, 1, 2, 4)), "nscales": 5, "iters": 50}
    if kind == "mixed":
        return {"kind": kind, "per_size": rng.randint(1, 2), "sizes": rng.randint(2, 5), "shrink": rng.randint(0, 60)}
    if kind == "hs":
        w, h = _size(rng, 96, 1280)
        levels = rng.randint(1, 4)
        warps = rng.randint(1, 3)
        return {"kind": kind, "w": w, "h": h, "pairs": _count(rng, w, h, 64, 64 * 320 * 240 // warps),
                "dtype": rng.choice(("u8", "f32")), "alpha": rng.choice((0.2, 1.0, 15.0)), "levels": levels, "warps": warps,
                "sweeps": rng.randint(50, 200), "tuned": False}
    if kind == "pyrlk":
        w, h = _size(rng, 96, 1280)
        return {"kind": kind, "w": w, "h": h, "pairs": _count(rng, w, h, 64), "dtype": rng.choice(("u8", "f32")),
                "spac": rng.choice((3, 5)), "window": rng.choice((5, 7, 9)), "levels": rng.randint(2, 3), "iters": rng.randint(1, 4)}
    if kind == "lk":
        w, h = _size(rng, 96, 1920)
        return {"kind": kind, "w": w, "h": h, "spac": rng.choice((3, 5, 7)), "temp": rng.choice((2, 3, 5)),
                "window": rng.choice((5, 7, 9))}
    w, h = _log(rng, 256, 1024), _log(rng, 192, 436)
    if kind == "train":
        return {"kind": kind, "w": w, "h": h, "pairs": rng.randint(4, 16)}
    return {"kind": kind, "w": w, "h": h, "pairs": rng.randint(1, 32), "warps": rng.randint(1, 3), "iters": rng.choice((10, 20, 30))}


# ------------------------------------------------------------------ inputs
_shared = {}  # what a program keeps for its whole life: the context, its stream, the network weights, the sizes it tuned


def _ctx():
    if "ctx" not in _shared:
        _shared["stream"] = torch.cuda.Stream()
        _shared["ctx"] = oflow.Context(0)
        _shared["ctx"].set_stream(_shared["stream"].cuda_stream)
        _shared["tuned"] = set()
    return _shared["ctx"]


def _weights():
    if "weights" not in _shared:
        _shared["weights"] = warmstart.load()[0]
    return _shared["weights"]


def _frames(n, w, h, seed, dtype, radius=None):
    """n textured pairs with affine motion and one independently moving disc: [n, h, w] u8, or f32 with fractional values."""
    a, b, *_ = synth_gpu.tvl1_pairs(n, w, h, seed=seed, radius=radius or min(80.0, 0.18 * min(w, h)))
    if dtype == "u8":
        return a, b
    g = torch.Generator(device="cuda")
    g.manual_seed(seed + 1)
    out = []
    for x in (a, b):
        out.append((x.float() + torch.rand(x.shape, generator=g, device="cuda") - 0.5).clamp_(0, 255))
    return tuple(out)


def _value_noise(n, w, h, seed, dtype, peak=8.0):
    """n pairs of 4-octave value noise under a smooth vortex plus pixel noise (the Lucas-Kanade workload)."""
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    I0 = torch.zeros((n, 1, h, w), device="cuda")
    for k in range(4):
        cell = 32 / 2 ** k
        grid = torch.rand((n, 1, int(h / cell) + 3, int(w / cell) + 3), generator=g, device="cuda")
        big = F.interpolate(grid, scale_factor=cell, mode="bilinear", align_corners=False)
        I0 += 0.5 ** k * big[:, :, :h, :w]
    I0 = I0[:, 0]
    lo, hi = I0.amin(dim=(1, 2), keepdim=True), I0.amax(dim=(1, 2), keepdim=True)
    I0 = (I0 - lo) * 255.0 / (hi - lo)
    yy, xx = torch.meshgrid(torch.arange(h, device="cuda", dtype=torch.float32),
                            torch.arange(w, device="cuda", dtype=torch.float32), indexing="ij")
    cx, cy, sig = (w - 1) / 2.0, (h - 1) / 2.0, 0.25 * min(w, h)
    sx, sy = xx, yy
    for _ in range(6):  # inverse of the vortex by fixed point
        dx, dy = sx - cx, sy - cy
        m = peak * math.exp(0.5) / sig * torch.exp(-(dx * dx + dy * dy) / (2 * sig * sig))
        sx, sy = xx + dy * m, yy - dx * m
    grid = torch.stack([sx / (w - 1) * 2 - 1, sy / (h - 1) * 2 - 1], -1).expand(n, h, w, 2)
    I1 = F.grid_sample(I0[:, None], grid, mode="bilinear", padding_mode="border", align_corners=True)[:, 0]
    I1 = (I1 + torch.randn((n, h, w), generator=g, device="cuda")).clamp(0, 255)
    if dtype == "u8":
        return tuple(x.round().to(torch.uint8) for x in (I0, I1))
    return I0.contiguous(), I1.contiguous()


def _source(case):
    """The frames of a case: Lucas-Kanade and pyramids of Horn-Schunck get texture at every scale."""
    return _value_noise if case["kind"] == "pyrlk" or case.get("levels", 1) > 1 else _frames


def _mixed_jobs(case, seed):
    """(solver, frames0, frames1) groups of the mixed batch."""
    groups = []
    s = case.get("shrink", 0)
    for k, (w, h) in enumerate(MIXED_SIZES[: case["sizes"]]):
        for solver in ("hs", "tvl1"):
            groups.append((solver,) + tuple(_frames(case["per_size"], w - s, h - s, seed + 10 * k + (solver == "hs"), "u8")))
    return groups


def _tv_params(case):
    return oflow.TVL1Params(nscales=case["nscales"], max_iterations=case["iters"])


def _out(n, h, w):
    o = torch.empty((n, 2, h, w), dtype=torch.float32, device="cuda")
    return o, [(o[i, 0], o[i, 1]) for i in range(n)]


def _train_io(case, seed):
    w, h, n = case["w"], case["h"], case["pairs"]
    a, b, u, v, _ = synth_gpu.tvl1_pairs(n, w, h, seed=seed, ndiscs_max=3, speed_max=16.0, radius=min(80.0, 0.18 * min(w, h)))
    target = F.avg_pool2d(torch.stack([u, v], 1), 8, ceil_mode=True) / 8.0
    return torch.stack([a, b], 1).contiguous(), target.permute(0, 2, 3, 1).contiguous()


def _net(w, h, n, ctx):
    net = oflow.WarmNet(w, h, n, ctx)
    torch.cuda.synchronize()  # its buffers are cleared on the default stream, its weights copied on the context's
    net.set_params(_weights())
    return net


def prepare(case, seed):
    kind, ctx = case["kind"], _ctx()
    st = {"kind": kind, "ctx": ctx}
    if kind == "mixed":
        jobs, outs, views = [], [], []
        hp, tp = oflow.HSParams(15.0, 1, 1, 200), oflow.TVL1Params(nscales=5, max_iterations=50)
        for solver, a, b in _mixed_jobs(case, seed):
            o, v = _out(*a.shape)
            outs.append(o)
            views += v
            jobs += [(solver, a[i], b[i], hp if solver == "hs" else tp) for i in range(a.shape[0])]
        st.update(jobs=jobs, outs=outs, views=views)
        return st
    w, h = case["w"], case["h"]
    if kind == "train":
        st["frames"], st["target"] = _train_io(case, seed)
        st["net"] = _net(w, h, case["pairs"], ctx)
        return st
    if kind == "stream":
        a, b = _frames(case["lanes"], w, h, seed, "u8")
        st["video"] = [[f[i].cpu().pin_memory() for i in range(case["lanes"])] for f in (a, b)]
        st["flow"], st["views"] = _out(case["lanes"], h, w)
        st["image"] = torch.empty((case["lanes"], h, w, 3), dtype=torch.uint8, device="cuda")
        st["stream"] = oflow.FrameStream(w, h, "tvl1", case["lanes"], _tv_params(case), "u8", ctx)
        torch.cuda.synchronize()
        st["stream"].push(st["video"][0], out=st["views"])
        st["next"] = 1
        return st
    if kind == "lk":
        a, b = _value_noise(1, w, h, seed, "u8", peak=2.0)
        ring = [a[0], b[0]]
        g = torch.Generator(device="cuda")
        g.manual_seed(seed)
        while len(ring) < case["temp"]:
            n = torch.randn((h, w), generator=g, device="cuda")
            ring.append((0.5 * (ring[-1].float() + ring[-2].float()) + n).clamp(0, 255).round().to(torch.uint8))
        st["ring"] = ring
        st["params"] = oflow.LKParams(case["spac"], case["temp"], case["window"])
        st["flow"], st["views"] = _out(1, h, w)
        return st
    n = case["pairs"]
    a, b = _source(case)(n, w, h, seed, case.get("dtype", "u8"))
    st["flow"], st["views"] = _out(n, h, w)
    st["pairs"] = [(a[i], b[i]) for i in range(n)]
    if kind == "tvl1":
        st["params"] = _tv_params(case)
        st["host"] = case["host"]
        if case["host"]:
            st["pairs"] = [(x.cpu().numpy(), y.cpu().numpy()) for x, y in st["pairs"]]
    elif kind == "hs":
        st["params"] = oflow.HSParams(case["alpha"], case["levels"], case["warps"], case["sweeps"])
    elif kind == "pyrlk":
        st["params"] = oflow.LKParams(case["spac"], 2, case["window"], case["levels"], case["iters"])
    else:
        st["net"] = _net(w, h, n, ctx)
        st["params"] = oflow.TVL1Params(nscales=5, warps=case["warps"], max_iterations=case["iters"])
    key = (kind, w, h, n)
    if case.get("tuned") and key not in _shared["tuned"]:
        torch.cuda.synchronize()
        (oflow.tvl1_autotune if kind == "tvl1" else oflow.hs_autotune)(st["pairs"], st["params"], ctx)
        _shared["tuned"].add(key)
    return st


def run(st):
    kind, ctx = st["kind"], st["ctx"]
    if kind == "tvl1":
        if st["host"]:  # host frames in, host flows out
            return oflow.tvl1_batch(st["pairs"], st["params"])
        oflow.tvl1_batch(st["pairs"], st["params"], ctx, out=st["views"])
        return st["flow"]
    if kind == "hs":
        oflow.hs_batch(st["pairs"], st["params"], ctx, out=st["views"])
        return st["flow"]
    if kind == "pyrlk":
        oflow.pyrlk_batch(st["pairs"], st["params"], ctx, out=st["views"])
        return st["flow"]
    if kind == "lk":
        oflow.lk(st["ring"], len(st["ring"]) - 1, st["params"], ctx, out=st["views"][0])
        return st["flow"]
    if kind == "mixed":
        oflow.batch(st["jobs"], ctx, out=st["views"])
        return st["outs"]
    if kind == "stream":
        st["stream"].push(st["video"][st["next"]], out=st["views"])
        st["next"] ^= 1
        oflow.flow_to_color_batch(st["views"], ctx, out=list(st["image"]))
        return st["flow"], st["image"]
    if kind == "train":
        loss = st["net"].train_step(st["frames"], st["target"], 1e-4)
        return loss, st["net"].get_params()
    oflow.tvl1_warm(st["pairs"], st["net"], st["params"], None, ctx, out=st["views"])
    return st["flow"]


# ------------------------------------------------------------------ work
_CONVS = [(16, 32, 2), (32, 32, 2), (32, 64, 4), (64, 64, 4), (64, 96, 8), (96, 96, 8), (96, 128, 16), (224, 96, 8),
          (160, 64, 4), (64, 8, 4)]  # channels in, out, and the output's reduction against the half-resolution input


def _net_flops(case):
    px = case["w"] * case["h"] / 4 * case["pairs"]
    return sum(2 * 9 * c * k * px / r ** 2 for c, k, r in _CONVS)


def _tv_flops(px, warps=5, iters=15, coarse=4 / 3):
    """About 70 operations a pixel and inner iteration and 200 a pixel and warp; the stopping rule ends a warp after some
    15 iterations on these frames."""
    return px * coarse * warps * (70 * iters + 200)


def work(case):
    """Bytes: each frame read once, each flow written once.  Operations: of the iterations, sums and products."""
    kind = case["kind"]
    if kind == "mixed":
        s, n = case.get("shrink", 0), case["per_size"]
        px = sum((w - s) * (h - s) for w, h in MIXED_SIZES[: case["sizes"]]) * n
        return {"bytes": 2 * px * 10, "flops": px * 28 * 200 + _tv_flops(px)}
    px = case["w"] * case["h"] * case.get("pairs", case.get("lanes", 1))
    frame = 4 if case.get("dtype") == "f32" else 1
    if kind == "tvl1":
        return {"bytes": px * (2 * frame + 8), "flops": _tv_flops(px)}
    if kind == "stream":
        return {"bytes": px * (1 + 8 + 3), "flops": _tv_flops(px)}
    if kind == "hs":
        area = sum(0.25 ** k for k in range(case["levels"]))
        return {"bytes": px * (2 * frame + 8), "flops": px * area * case["warps"] * (28 * case["sweeps"] + 60)}
    if kind == "pyrlk":
        area = sum(0.25 ** k for k in range(case["levels"]))
        return {"bytes": px * (2 * frame + 8), "flops": px * area * case["iters"] * (5 * case["window"] ** 2 + 40)}
    if kind == "lk":
        return {"bytes": px * (case["temp"] + 8), "flops": px * (5 * case["window"] ** 2 + 5 + 4 * case["spac"] + 30)}
    if kind == "train":  # frames and targets in; weights and Adam moments in and out
        return {"bytes": px * (2 + 8 / 64) + 28 * 607e3, "flops": 3 * _net_flops(case)}
    return {"bytes": px * 10, "flops": _net_flops(case) + _tv_flops(px, case["warps"], min(15, case["iters"]), 85 / 64)}


# ------------------------------------------------------------------ 64-bit results
def _shift(a, dy, dx):
    """a at (y + dy, x + dx), coordinates clamped to the image."""
    h, w = a.shape[-2:]
    yi = (torch.arange(h, device=a.device) + dy).clamp(0, h - 1)
    xi = (torch.arange(w, device=a.device) + dx).clamp(0, w - 1)
    return a[..., yi[:, None], xi[None, :]]


def _gauss(a, sigma):
    """Separable Gaussian; mirrored without the edge sample before the start, with it past the end."""
    size = int(5.0 * sigma) + 1
    b = torch.tensor([math.exp(-i * i / (2 * sigma * sigma)) for i in range(size)], dtype=torch.float64)
    b = b / (2 * b.sum() - b[0])
    for dim in (-1, -2):
        n = a.shape[dim]
        i = torch.arange(n, device=a.device)
        out = b[0].item() * a
        for j in range(1, size):
            lo, hi = (i - j).abs(), i + j
            hi = torch.where(hi >= n, 2 * n - 1 - hi, hi)
            out = out + b[j].item() * (a.index_select(dim, lo) + a.index_select(dim, hi))
        a = out
    return a


def _half(n):
    return int(n * 0.5 + 0.5)


def _zoom_out(a):
    """Half size: blur, then the even rows and columns."""
    h, w = a.shape[-2:]
    s = _gauss(a, 0.6 * math.sqrt(3.0))
    return s[..., : 2 * _half(h) : 2, : 2 * _half(w) : 2].contiguous()


def _keys(v, t):
    return v[1] + 0.5 * t * (v[2] - v[0] + t * (2 * v[0] - 5 * v[1] + 4 * v[2] - v[3] + t * (3 * (v[1] - v[2]) + v[3] - v[0])))


def _bicubic(img, x, y, zero_outside):
    """Keys cubic samples of [n, h, w] at [n, h', w'], taps clamped (or the sample 0 where a tap leaves the image)."""
    n, h, w = img.shape
    flat = img.reshape(n, -1)
    xi, yi = x.trunc(), y.trunc()
    bad = (xi < 1) | (xi > w - 3) | (yi < 1) | (yi > h - 3) | (x < 0) | (y < 0)
    tx, ty = x - xi.clamp(0, w - 1), y - yi.clamp(0, h - 1)
    xi, yi = xi.clamp(-1e6, 1e6).long(), yi.clamp(-1e6, 1e6).long()
    cols = []
    for cx in range(-1, 3):
        c = (xi + cx).clamp(0, w - 1)
        v = [flat.gather(1, ((yi + cy).clamp(0, h - 1) * w + c).reshape(n, -1)).reshape(x.shape) for cy in range(-1, 3)]
        cols.append(_keys(v, ty))
    out = _keys(cols, tx)
    return torch.where(bad, torch.zeros_like(out), out) if zero_outside else out


def _bilinear(img, x, y):
    """Bilinear samples of [n, h, w], coordinates limited to [-1, size] and taps clamped to the edge."""
    n, h, w = img.shape
    flat = img.reshape(n, -1)
    x, y = x.clamp(-1, w), y.clamp(-1, h)
    x0, y0 = x.floor(), y.floor()
    fx, fy = x - x0, y - y0

    def at(dy, dx):
        return flat.gather(1, ((y0.long() + dy).clamp(0, h - 1) * w + (x0.long() + dx).clamp(0, w - 1)).reshape(n, -1)).reshape(x.shape)
    return (1 - fy) * ((1 - fx) * at(0, 0) + fx * at(0, 1)) + fy * ((1 - fx) * at(1, 0) + fx * at(1, 1))


def _mesh(n, h, w):
    yy, xx = torch.meshgrid(torch.arange(h, device="cuda", dtype=torch.float64),
                            torch.arange(w, device="cuda", dtype=torch.float64), indexing="ij")
    return xx.expand(n, h, w), yy.expand(n, h, w)


def _upscale(U, h, w):
    """Centre-aligned bilinear prolongation of a flow (u, v) to h x w, scaled by the size ratios."""
    n, ch, cw = U[0].shape
    xx, yy = _mesh(n, h, w)
    x, y = (xx + 0.5) * (cw / w) - 0.5, (yy + 0.5) * (ch / h) - 0.5
    return [_bilinear(U[0], x, y) * (w / cw), _bilinear(U[1], x, y) * (h / ch)]


def _div(a, b):
    """Backward-difference divergence of (a, b); a vanishes in the last column, b in the last row."""
    d = a.clone()
    d[..., :, 1:] -= a[..., :, :-1]
    d += b
    d[..., 1:, :] -= b[..., :-1, :]
    return d


def _tvl1_exact(I0, I1, nscales, iters, warps=5, start=None):
    """TV-L1 of [n, h, w] pairs; start: (scale, flow at that scale) instead of zero at the coarsest."""
    tau, lam, theta, eps = 0.25, 0.15, 0.3, 0.01
    I0, I1 = I0.double(), I1.double()
    n, h, w = I0.shape
    ns = min(nscales, int(1 + math.log(math.hypot(w, h) / 16.0) / math.log(2.0)))
    lo = torch.minimum(I0.amin((1, 2), True), I1.amin((1, 2), True))
    hi = torch.maximum(I0.amax((1, 2), True), I1.amax((1, 2), True))
    pyr = [[_gauss(255.0 * (I - lo) / (hi - lo), 0.8)] for I in (I0, I1)]
    for p in pyr:
        for _ in range(ns - 1):
            p.append(_zoom_out(p[-1]))
    s0 = ns - 1 if start is None else start[0]
    U = None if start is None else start[1]
    for s in range(s0, -1, -1):
        A, B = pyr[0][s], pyr[1][s]
        hh, ww = A.shape[1:]
        xx, yy = _mesh(n, hh, ww)
        if U is None:
            U = [torch.zeros_like(A), torch.zeros_like(A)]
        elif s < s0:
            ch, cw = U[0].shape[1:]
            U = [2.0 * _bicubic(c, xx / (ww / cw), yy / (hh / ch), False) for c in U]
        Bx, By = 0.5 * (_shift(B, 0, 1) - _shift(B, 0, -1)), 0.5 * (_shift(B, 1, 0) - _shift(B, -1, 0))
        P = [torch.zeros_like(A) for _ in range(4)]
        for _ in range(warps):
            Iw, Ix, Iy = (_bicubic(c, xx + U[0], yy + U[1], True) for c in (B, Bx, By))
            rc, g2 = Iw - Ix * U[0] - Iy * U[1] - A, Ix * Ix + Iy * Iy
            live = torch.ones((n, 1, 1), dtype=torch.bool, device="cuda")
            for _ in range(iters):
                rho = rc + Ix * U[0] + Iy * U[1]
                lt = lam * theta
                k = torch.where(rho < -lt * g2, torch.full_like(rho, lt),
                                torch.where(rho > lt * g2, torch.full_like(rho, -lt),
                                            torch.where(g2 < 1e-10, torch.zeros_like(rho), -rho / g2.clamp_min(1e-300))))
                V = [U[0] + k * Ix + theta * _div(P[0], P[1]), U[1] + k * Iy + theta * _div(P[2], P[3])]
                err = ((V[0] - U[0]) ** 2 + (V[1] - U[1]) ** 2).mean((1, 2), keepdim=True)
                Q = []
                for c in (0, 1):
                    fx, fy = _shift(V[c], 0, 1) - V[c], _shift(V[c], 1, 0) - V[c]
                    g = 1.0 + tau / theta * torch.sqrt(fx * fx + fy * fy)
                    Q += [(P[2 * c] + tau / theta * fx) / g, (P[2 * c + 1] + tau / theta * fy) / g]
                U = [torch.where(live, v, u) for v, u in zip(V, U)]
                P = [torch.where(live, q, p) for q, p in zip(Q, P)]
                live = live & (err > eps * eps)
                if not bool(live.any()):
                    break
    return torch.stack(U, 1)


def _hs_exact(I0, I1, alpha, levels, warps, sweeps):
    pyr = [[I0.double()], [I1.double()]]
    for p in pyr:
        for _ in range(levels - 1):
            a = p[0]
            h, w = a.shape[1] // 2 * 2, a.shape[2] // 2 * 2
            p.insert(0, F.avg_pool2d(a[:, None, :h, :w], 2)[:, 0])
    U = [torch.zeros_like(pyr[0][0]) for _ in range(2)]

    def deriv(a, dy, dx):
        t = [_shift(a, k * dy, k * dx) for k in (-2, -1, 1, 2)]
        return (t[0] - 8 * t[1] + 8 * t[2] - t[3]) / 12.0
    for lv in range(levels):
        A, B = pyr[0][lv], pyr[1][lv]
        n, h, w = A.shape
        xx, yy = _mesh(n, h, w)
        if lv:
            U = _upscale(U, h, w)
        for _ in range(warps):
            Bw = _bilinear(B, xx + U[0], yy + U[1])
            Ix, Iy = 0.5 * (deriv(A, 0, 1) + deriv(Bw, 0, 1)), 0.5 * (deriv(A, 1, 0) + deriv(Bw, 1, 0))
            Iz = Bw - A
            den = Ix * Ix + Iy * Iy + alpha
            d = torch.zeros((2,) + A.shape, dtype=torch.float64, device="cuda")
            for _ in range(sweeps):
                p = F.pad(d, (1, 1, 1, 1), mode="replicate")
                m = 0.25 * (p[..., 1:-1, :-2] + p[..., 1:-1, 2:] + p[..., :-2, 1:-1] + p[..., 2:, 1:-1])
                f = (Ix * m[0] + Iy * m[1] + Iz) / den
                d = torch.stack([m[0] - Ix * f, m[1] - Iy * f])
            U = [U[0] + d[0], U[1] + d[1]]
    return torch.stack(U, 1)


_TAPS = {1: [1.0], 2: [-1.0, 1.0], 3: [-1 / 2, 0, 1 / 2], 5: [1 / 12, -2 / 3, 0, 2 / 3, -1 / 12],
         7: [-1 / 60, 3 / 20, -3 / 4, 0, 3 / 4, -3 / 20, 1 / 60]}


def _fir(a, taps, dim):
    """Correlation along a dimension, taps outside the image dropped."""
    c = len(taps) // 2
    pad = (c, c, 0, 0) if dim == -1 else (0, 0, c, c)
    p = F.pad(a, pad)
    n = a.shape[dim]
    return sum(t * p.narrow(dim, k, n) for k, t in enumerate(taps))


def _lk_solve(gx, gy, gt, window):
    c = window // 2

    def box(a):
        a = sum(F.pad(a, (c, c, 0, 0)).narrow(-1, k, a.shape[-1]) for k in range(window))
        return sum(F.pad(a, (0, 0, c, c)).narrow(-2, k, a.shape[-2]) for k in range(window))
    xx, xy, yy, xt, yt = box(gx * gx), box(gx * gy), box(gy * gy), box(gx * gt), box(gy * gt)
    det = xx * yy - xy * xy
    inv = torch.where(det != 0, 1.0 / det, torch.zeros_like(det))
    inside = torch.zeros_like(det)
    inside[..., c : det.shape[-2] - c, c : det.shape[-1] - c] = 1.0
    return inside * inv * (xy * yt - yy * xt), inside * inv * (xy * xt - xx * yt)


def _pyrlk_exact(I0, I1, case):
    A, B = [I0.double()], [I1.double()]
    for p in (A, B):
        for _ in range(case["levels"] - 1):
            p.append(_zoom_out(p[-1]))
    U = None
    for lv in range(case["levels"] - 1, -1, -1):
        n, h, w = A[lv].shape
        U = [torch.zeros_like(A[lv]) for _ in range(2)] if U is None else _upscale(U, h, w)
        xx, yy = _mesh(n, h, w)
        gx, gy = _fir(A[lv], _TAPS[case["spac"]], -1), _fir(A[lv], _TAPS[case["spac"]], -2)
        for _ in range(case["iters"]):
            it = _bilinear(B[lv], xx + U[0], yy + U[1]) - A[lv]
            d = _lk_solve(gx, gy, it, case["window"])
            U = [U[0] + d[0], U[1] + d[1]]
    return torch.stack(U, 1)


def _net_exact(frames, params):
    """The warm-start network in 64 bits: [n, 2, h, w] frames -> [n, 8, h/8, w/8]."""
    f = frames.double()
    f = F.pad(f, (0, f.shape[3] % 2, 0, f.shape[2] % 2), mode="replicate")
    f = F.avg_pool2d(f, 2) / 255.0
    x = torch.cat([f - 0.5, 4 * (f[:, 1:] - f[:, :1])], 1)
    x = torch.cat([x, torch.zeros((x.shape[0], 13) + x.shape[2:], dtype=x.dtype, device=x.device)], 1)

    def conv(i, a):
        w, b = params[i]
        stride = 2 if i in (0, 2, 4, 6) else 1
        a = F.conv2d(a, w.permute(0, 3, 1, 2), b, stride=stride, padding=1)
        return a if i == 9 else a.relu()

    def up(a, skip):
        h, w = skip.shape[2:]
        yi = (torch.arange(h, device=a.device) // 2).clamp_max(a.shape[2] - 1)
        xi = (torch.arange(w, device=a.device) // 2).clamp_max(a.shape[3] - 1)
        return torch.cat([a[:, :, yi[:, None], xi[None, :]], skip], 1)
    c4 = conv(3, conv(2, conv(1, conv(0, x))))
    c6 = conv(5, conv(4, c4))
    c8 = conv(7, up(conv(6, c6), c6))
    return conv(9, conv(8, up(c8, c4)))


def _net_params(grad=False):
    flat = torch.from_numpy(np.asarray(_weights(), np.float64)).cuda()
    out, at = [], 0
    for c, k in warmstart.LAYERS:
        w = flat[at : at + 9 * c * k].reshape(k, 3, 3, c).clone().requires_grad_(grad)
        at += 9 * c * k
        out.append((w, flat[at : at + k].clone().requires_grad_(grad)))
        at += k
    return out


def _train_exact(case, seed):
    frames, target = _train_io(case, seed)
    params = _net_params(True)
    flow = _net_exact(frames, params)[:, :2].permute(0, 2, 3, 1)
    loss = torch.sqrt((flow - target.double()) ** 2 + 1e-6).mean()
    loss.backward()
    new = []
    for p in (q for wb in params for q in wb):  # Adam's first step
        new.append((p.detach() - 1e-4 * p.grad / (p.grad.abs() + 1e-8)).reshape(-1))
    return float(loss.detach()), torch.cat(new)


def exact(case, seed):
    kind = case["kind"]
    if kind == "train":
        return _train_exact(case, seed)
    if kind == "mixed":
        return [_hs_exact(a, b, 15.0, 1, 1, 200) if solver == "hs" else _tvl1_exact(a, b, 5, 50)
                for solver, a, b in _mixed_jobs(case, seed)]
    w, h = case["w"], case["h"]
    if kind == "lk":
        ring = [f.double() for f in prepare(case, seed)["ring"]]
        gt = sum(t * f for t, f in zip(_TAPS[case["temp"]], ring))  # the newest frame is in the last slot
        taps = _TAPS[case["spac"]]
        return torch.stack(_lk_solve(_fir(ring[0], taps, -1), _fir(ring[0], taps, -2), gt, case["window"]))[None]
    if kind == "stream":
        a, b = _frames(case["lanes"], w, h, seed, "u8")
        return _tvl1_exact(a, b, case["nscales"], case["iters"]), None  # the image is bytes
    a, b = _source(case)(case["pairs"], w, h, seed, case.get("dtype", "u8"))
    if kind == "tvl1":
        r = _tvl1_exact(a, b, case["nscales"], case["iters"])
        return [(r[i, 0], r[i, 1]) for i in range(len(r))] if case["host"] else r
    if kind == "hs":
        # repeated warps on coarse levels amplify rounding: no 64-bit value says how exact 32 bits are there
        if case["warps"] > 1 and (case["levels"] > 3 or case["levels"] > 1 and case["alpha"] < 15):
            return None
        return _hs_exact(a, b, case["alpha"], case["levels"], case["warps"], case["sweeps"])
    if kind == "pyrlk":
        return _pyrlk_exact(a, b, case)
    with torch.no_grad():
        flow = _net_exact(torch.stack([a, b], 1), _net_params())
    return _tvl1_exact(a, b, 5, case["iters"], case["warps"], (3, [flow[:, 0], flow[:, 1]]))
