"""Timed cases of the solver's public entry points.

One segmentation of a 4D volume is an edge detector (once per volume) and a
series of semi-implicit time steps; beside it stand the mean-curvature-flow
known-answer step, batches of small volumes, the step on host arrays and the
learned warm start (a step that uses it, a training step that makes it).  The
cases cover these from the 32^3 x 8 reference size to the 256 x 256 x 128 x 20
benchmark size, in the FP64 and the mixed form, with round and ragged extents.

listed() and draw() give cases, prepare() what a program holds before the
call, run() one pass, work() the bytes and operations a pass cannot do
without, exact() the result in plain 64-bit torch.
"""
from __future__ import annotations

import math
import os
import random
import sys

import numpy as np
import torch

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
PKG = os.path.join(ROOT, "4d-image-segmentation-algorithm_gb300")
if PKG not in sys.path:
    sys.path.insert(0, PKG)

import ss4d  # noqa: E402

BALL_RADIUS = 8.0
CROP_MARGIN = 4  # reach of the network's four 3x3x3 layers


# ---------------------------------------------------------------------------
# cases


def listed():
    return [
        # the reference's own volume size: one FP64 step, where latency and launches count
        {"name": "step fp64 32x32x32x8", "kind": "step", "form": "fp64", "nx": 32, "ny": 32, "nz": 32, "nt": 8,
         "h": 1.0, "balls": False},
        # an ordinary volume in the plain form (the two-sector workload's size)
        {"name": "step fp64 128x128x128x16", "kind": "step", "form": "fp64", "nx": 128, "ny": 128, "nz": 128,
         "nt": 16, "h": 1.0, "balls": False},
        # the known-answer test of the flow without an image: tight tolerance, h no power of two
        {"name": "mcf fp64 40^4", "kind": "mcf", "form": "fp64", "n": 40},
        # a small cell volume followed in time, the form the benchmark reports
        {"name": "series mixed 45x37x29x7", "kind": "series", "nx": 45, "ny": 37, "nz": 29, "nt": 7, "h": 1.0,
         "steps": 10},
        # the benchmark volume: the first steps of its time series
        {"name": "series mixed 256x256x128x20", "kind": "series", "nx": 256, "ny": 256, "nz": 128, "nt": 20,
         "h": 1.0, "steps": 5},
        # a step as the reference's main takes it, with centres and a mask, ragged extents
        {"name": "step mixed balls 161x143x61x9", "kind": "step", "form": "mixed", "nx": 161, "ny": 143, "nz": 61,
         "nt": 9, "h": 1.0, "balls": True},
        # the reference-named layer's step: u on the host before and after
        {"name": "host mixed 128x128x64x12", "kind": "host", "form": "mixed", "nx": 128, "ny": 128, "nz": 64,
         "nt": 12, "h": 1.0},
        # a step started from the network's prediction, at the size it is trained on
        {"name": "learned 128x128x64x12", "kind": "learned", "nx": 128, "ny": 128, "nz": 64, "nt": 12, "h": 1.0},
        # the front end of a plain-form segmentation: image and thresholded image, ragged extents
        {"name": "edge fp64 97x101x53x11", "kind": "edge", "form": "fp64", "nx": 97, "ny": 101, "nz": 53, "nt": 11,
         "h": 1.0, "images": 2},
        # the front end of the benchmark volume
        {"name": "edge mixed 256x256x128x20", "kind": "edge", "form": "mixed", "nx": 256, "ny": 256, "nz": 128,
         "nt": 20, "h": 1.0, "images": 2},
        # many small volumes together
        {"name": "batch mixed 48 of 24-48", "kind": "batch", "volumes": 48, "lo": 24, "hi": 48, "tlo": 4, "thi": 8,
         "steps": 3, "sizes": 1},
        # one optimiser step of the network (forward, backward, weight gradients, Adam)
        {"name": "train 8 crops 40x40x20", "kind": "train", "nx": 40, "ny": 40, "nz": 20, "crops": 8},
    ]


def _extents(rng: random.Random, lo: int, hi: int, least: int = 8):
    """ragged extents whose voxel count is log-uniform in [lo, hi]"""
    v = math.exp(rng.uniform(math.log(lo), math.log(hi)))
    nt = max(2, min(24, round(v ** 0.25 * rng.uniform(0.15, 0.35))))
    s = (v / nt) ** (1 / 3)
    nx = max(least, round(s * rng.uniform(0.8, 1.6)))
    ny = max(least, round(s * rng.uniform(0.8, 1.25)))
    nz = max(least, int(v / (nt * nx * ny)))
    return {"nx": nx, "ny": ny, "nz": nz, "nt": nt}


def draw(rng: random.Random):
    kind = rng.choice(["step", "step", "step", "series", "series", "edge", "edge", "mcf", "host", "learned",
                       "batch", "train"])
    h = rng.choice([1.0, 1.0, 0.5, 0.8])
    if kind == "step":
        form = rng.choice(["fp64", "mixed"])
        balls = rng.random() < 0.4
        return {"kind": kind, "form": form, **_extents(rng, 200_000, 40_000_000, 24 if balls else 8), "h": h,
                "balls": balls}
    if kind == "series":
        e = _extents(rng, 60_000, 80_000_000)
        return {"kind": kind, **e, "h": h, "steps": rng.randint(2, 8)}
    if kind == "edge":
        form = rng.choice(["fp64", "mixed"])
        return {"kind": kind, "form": form, **_extents(rng, 200_000, 20_000_000 if form == "fp64" else 120_000_000),
                "h": h, "images": rng.choice([1, 2])}
    if kind == "mcf":
        return {"kind": kind, "form": rng.choice(["fp64", "mixed"]), "n": round(math.exp(rng.uniform(math.log(11), math.log(64))))}
    if kind == "host":
        return {"kind": kind, "form": rng.choice(["fp64", "mixed"]), **_extents(rng, 200_000, 14_000_000), "h": h}
    if kind == "learned":
        return {"kind": kind, **_extents(rng, 200_000, 14_000_000, 16), "h": 1.0}
    if kind == "batch":
        lo = rng.randint(16, 40)
        return {"kind": kind, "volumes": rng.randint(4, 48), "lo": lo, "hi": lo + rng.randint(4, 30), "tlo": 3,
                "thi": rng.randint(4, 10), "steps": rng.randint(1, 4), "sizes": rng.randint(2, 1 << 20)}
    return {"kind": "train", "nx": rng.randint(16, 48), "ny": rng.randint(16, 48), "nz": rng.randint(10, 28),
            "crops": rng.randint(2, 16)}


# ---------------------------------------------------------------------------
# scenes, made on the GPU: deforming ellipsoids with erased boundary sectors,
# noise and 8-bit quantisation; u0 = 1 / (distance to the nearest centre + 1)


def _gen(seed):
    return torch.Generator(device="cuda").manual_seed(int(seed) & 0x7FFFFFFF)


def _scene(nx, ny, nz, nt, seed, nobj):
    r = random.Random(int(seed) * 7919 + 11)
    gen = _gen(seed)
    least = min(nx, ny, nz)
    objs = []
    for _ in range(nobj):
        rad = [r.uniform(0.16, 0.38) * least for _ in range(3)]
        m = 1.15 * max(rad) + 1.0
        c = [r.uniform(1.0 + m, n - m) if 1.0 + m < n - m else (n + 1) / 2.0 for n in (nx, ny, nz)]
        objs.append((c, rad, [r.uniform(0, 2 * math.pi) for _ in range(3)], r.uniform(150.0, 230.0)))
    i0 = torch.zeros((nt + 2, nz + 2, ny + 2, nx + 2), dtype=torch.float64, device="cuda")
    u0 = torch.zeros_like(i0)
    x = torch.arange(nx + 2, device="cuda", dtype=torch.float64)[None, None, :]
    y = torch.arange(ny + 2, device="cuda", dtype=torch.float64)[None, :, None]
    z = torch.arange(nz + 2, device="cuda", dtype=torch.float64)[:, None, None]
    for l in range(nt + 2):
        val = torch.full(i0.shape[1:], 50.0, device="cuda", dtype=torch.float32)
        for c, rad, ph, inten in objs:
            dx, dy, dz = x - c[0], y - c[1], z - c[2]
            d2 = dx * dx + dy * dy + dz * dz
            u0[l] = torch.maximum(u0[l], 1.0 / (torch.sqrt(d2 + (l - (nt + 1) / 2.0) ** 2) + 1.0))
            rr = [rad[a] * (1.0 + 0.15 * math.sin(2 * math.pi * (l - 1) / nt + ph[a])) for a in range(3)]
            rho2 = ((dx / rr[0]) ** 2 + (dy / rr[1]) ** 2 + (dz / rr[2]) ** 2).float()
            a0 = r.uniform(-math.pi, math.pi)
            rel = torch.remainder(torch.atan2(dy, dx) - a0, 2 * math.pi)
            inside = (rho2 <= 1.0) & ~((rho2 >= 0.49) & (rel < 2 * math.pi / 10))
            val = torch.where(inside, val.clamp(min=inten), val)
        if 1 <= l <= nt:
            drift = 1.0 + 0.1 * (2.0 * (l - 1) / (nt - 1) - 1.0 if nt > 1 else 0.0)
            val = val * drift + 25.0 * torch.randn(val.shape, device="cuda", generator=gen)
            q = torch.floor(val + 0.5).clamp(0, 255).double() / 255.0
            i0[l, 1:-1, 1:-1, 1:-1] = q[1:-1, 1:-1, 1:-1]
    return i0, u0


def _balls(nx, ny, nz, nt, seed, per_frame=5):
    """centres per frame, (frame, x, y, z), whose boxes stay in the volume"""
    r = random.Random(int(seed) * 31 + 5)
    m = BALL_RADIUS + 1.5
    return [(l, *(round(r.uniform(1 + m, n - m), 1) for n in (nx, ny, nz)))
            for l in range(1, nt + 1) for _ in range(per_frame)]


def _box(b):
    return tuple(slice(int(c - BALL_RADIUS - 0.5), int(c + BALL_RADIUS + 0.5) + 1) for c in b[:0:-1])  # z, y, x


def _dist(b, box):
    z, y, x = (torch.arange(s.start, s.stop, device="cuda", dtype=torch.float64) for s in box)
    return torch.sqrt(((x[None, None, :] - b[1]) ** 2 + (y[None, :, None] - b[2]) ** 2)
                      + (z[:, None, None] - b[3]) ** 2)


def _balls_init(shape, balls):
    """the reference's initial function and mask around the centres"""
    u, mask = (torch.zeros(shape, dtype=torch.float64, device="cuda") for _ in range(2))
    for b in balls:
        box = _box(b)
        r = _dist(b, box)
        near = r <= 12.0
        v, w = u[b[0]][box], mask[b[0]][box]
        v.copy_(torch.where(near, torch.maximum(v, (1.0 / (r + 0.5) - 1.0 / 12.5).abs()), v))
        w.masked_fill_(near, 1.0)
    return u, mask


# ---------------------------------------------------------------------------
# the same mathematics in plain 64-bit torch


def _at(v, off=(0, 0, 0, 0)):
    """interior of v shifted by off = (x, y, z, t)"""
    return v[tuple(slice(1 + o, n - 1 + o) for o, n in zip(reversed(off), v.shape))]


def _e(a, s):
    o = [0, 0, 0, 0]
    o[a] = s
    return tuple(o)


def _plus(p, q):
    return tuple(a + b for a, b in zip(p, q))


def _red(v):
    lM, kM, jM, iM = v.shape
    r = torch.arange(max(v.shape), device=v.device)
    s = (r[1:lM - 1, None, None, None] + r[None, 1:kM - 1, None, None] + r[None, None, 1:jM - 1, None]
         + r[None, None, None, 1:iM - 1])
    return s % 2 == 0


def _sum8(v):
    s = _at(v, _e(0, 1)) + _at(v, _e(0, -1))
    for a in range(1, 4):
        s += _at(v, _e(a, -1))
        s += _at(v, _e(a, 1))
    return s


def _presmooth(p, img):
    prev = _at(img).clone()
    for a in range(4):
        d = 3 - a
        n = img.shape[d]
        img.select(d, 0).copy_(img.select(d, 1))
        img.select(d, n - 1).copy_(img.select(d, n - 2))
    c, h4 = p.sigma / (p.h * p.h), p.h ** 4
    red = _red(img)
    z = 0
    while True:
        z += 1
        for m in (red, ~red):
            gs = (prev + c * _sum8(img)) / (1 + 8 * c)
            v = _at(img)
            v.copy_(torch.where(m, v + p.omega_sigma * (gs - v), v))
        r = _at(img) * (1 + 8 * c) - c * _sum8(img) - prev
        R = float((r * r).sum()) * h4
        if not (R > p.gsTol and z < p.maxNoGSIteration_sigma):
            return img


def _face_sq(v, f, h):
    """|grad v|^2 at face f (e, w, n, s, t, b, fw, bw) of every interior voxel"""
    d, nb = f >> 1, _e(f >> 1, -1 if f & 1 else 1)
    s = torch.zeros_like(_at(v))
    for a in range(4):
        if a == d:
            t = (_at(v, nb) - _at(v)) / h
        else:
            up, dn = _e(a, 1), _e(a, -1)
            t = ((_at(v, _plus(nb, up)) + _at(v, up)) - (_at(v, _plus(nb, dn)) + _at(v, dn))) / (4.0 * h)
        s += t * t
    return s


def _edges(p, i0, thr=None):
    g = []
    for f in range(8):
        s = p.theta_img * _face_sq(i0, f, p.h)
        if thr is not None:
            s = s + p.rho_thr * _face_sq(thr, f, p.h)
        out = torch.zeros_like(i0)
        _at(out).copy_(1.0 / (1.0 + p.K * s))
        g.append(out)
    return g


def _coefficients(p, u, g):
    nf = [torch.sqrt(_face_sq(u, f, p.h) + p.eps2) for f in range(8)]
    mean = sum(nf) / 8.0
    vc = torch.sqrt(mean * mean + p.eps2)
    return [vc / nf[f] if g is None else vc * _at(g[f]) / nf[f] for f in range(8)]


def _solve(p, u, prev, a, tol=None, omega=None):
    """red-black SOR in place on u; returns the iterations"""
    c, h4 = p.tau / (p.h * p.h), p.h ** 4
    tol, omega = p.gsTol if tol is None else tol, p.omega_c if omega is None else omega
    nbr = [_e(f >> 1, -1 if f & 1 else 1) for f in range(8)]
    ca = [c * x for x in a]
    diag = 1.0 + sum(ca)
    red = _red(u)

    def rhs():
        s = prev.clone()
        for f in range(8):
            s += ca[f] * _at(u, nbr[f])
        return s

    for z in range(1, p.maxNoGSIteration + 1):
        for m in (red, ~red):
            v = _at(u)
            v.copy_(torch.where(m, v + omega * (rhs() / diag - v), v))
        r = _at(u) * diag - rhs()
        if not float((r * r).sum()) * h4 > tol:
            break
    return z


def _rescale(p, u, mask, balls):
    last = -1
    for b in balls:
        box = _box(b)
        v = u[b[0]][box]
        inside = _dist(b, box) <= p.ballRadius
        lo = min(100000.0, float(v[inside].min()))
        q = 1.0 / (max(0.0, float(v[inside].max())) - lo)
        nv = q * v - lo * q
        v.copy_(torch.where(inside & ((v < nv) if b[0] == last else torch.ones_like(inside)), nv, v))
        last = b[0]
    _at(u).masked_fill_(_at(mask) == 0, 0.0)


def _exact_step(p, u, g, plain):
    """one time step in place; plain: stopped as the FP64 form stops, else to
    the limit of 64 bits (the solution every form approaches)"""
    a = _coefficients(p, u, g)
    prev = _at(u).clone()
    if plain:
        return _solve(p, u, prev, a)
    _solve(p, u, prev, a, tol=1e-24 * float((prev * prev).sum()) * p.h ** 4, omega=1.15)
    return None


# ---------------------------------------------------------------------------
# inputs


def _params(case, **over):
    return ss4d.scene_params(h=case["h"], ballRadius=BALL_RADIUS, **over)


def _dims(case):
    return case["nx"], case["ny"], case["nz"], case["nt"]


def _threshold_image(i0):
    hi = i0.max()
    return torch.where(i0 > 0.5 * hi, hi, torch.zeros_like(i0))


def _step_inputs(case, seed):
    p = _params(case)
    i0, u0 = _scene(*_dims(case), seed, 3)
    i0 = _presmooth(p, i0)
    g = _edges(p, i0)
    mask = balls = None
    if case.get("balls"):
        balls = _balls(*_dims(case), seed)
        u0, mask = _balls_init(tuple(u0.shape), balls)
    return p, i0, u0, g, mask, balls


def _edge_inputs(case, seed):
    two = case["images"] == 2
    p = _params(case, **({"theta_img": 0.5, "rho_thr": 0.5} if two else {}))
    i0, _ = _scene(*_dims(case), seed, 3)
    return p, i0, _threshold_image(i0) if two else None


def _batch_inputs(case, seed):
    r = random.Random(case["sizes"])  # the sizes belong to the case, the contents to the seed
    q = random.Random(seed)
    vols = []
    for v in range(case["volumes"]):
        dims = [r.randint(case["lo"], case["hi"]) for _ in range(3)] + [r.randint(case["tlo"], case["thi"])]
        p = ss4d.scene_params(K=q.uniform(500, 2000), tau=q.uniform(0.25, 1.0))
        i0, u0 = _scene(*dims, seed * 64 + v, 1)
        vols.append((p, u0, _edges(p, _presmooth(p, i0))))
    return vols


def _mcf_start(case, seed):
    """the known solution at t = 0 with a seeded perturbation of the interior"""
    n = case["n"]
    h = 2.5 / n
    c = (torch.arange(n + 2, device="cuda", dtype=torch.float64) - 1) * h + h / 2 - 1.25
    x2 = c * c
    u = (x2[:, None, None, None] + x2[None, :, None, None] + x2[None, None, :, None] + x2[None, None, None, :]
         - 1.0) / 6.0
    _at(u).add_(1e-3 * torch.randn(_at(u).shape, device="cuda", dtype=torch.float64, generator=_gen(seed)))
    return ss4d.mcf_params(n), u


def _train_inputs(case, seed):
    """crops of the network's features and targets: a residual field of unit
    RMS at three frames, its first Jacobi iterate, the couplings, 1/diag, the
    mean g, u and the image; the target a damped, smoothed residual"""
    gen = _gen(seed)
    f, nz, ny, nx = case["crops"], case["nz"], case["ny"], case["nx"]

    def rnd(n):
        return torch.randn((f, n, nz, ny, nx), device="cuda", generator=gen)

    def uni(n):
        return torch.rand((f, n, nz, ny, nx), device="cuda", generator=gen)

    def smooth(a):
        return torch.nn.functional.avg_pool3d(a, 3, 1, 1, count_include_pad=False)

    amp = torch.exp(0.8 * smooth(rnd(1)) * 3.0)
    res = amp * (rnd(3) + 2.0 * smooth(rnd(3)))
    inv = 0.2 + 0.7 * smooth(uni(1))
    coup = (1.0 - inv) * (0.06 + 0.13 * uni(8))
    x = torch.cat([res, res[:, :1] * inv, coup, inv, smooth(uni(1)), smooth(uni(1)), smooth(uni(1))], dim=1)
    target = (inv * res[:, :1] + 0.4 * smooth(res[:, :1]))[:, 0].contiguous()
    return x.to(torch.bfloat16), target.float()


LAYERS = ((16, 24), (24, 24), (24, 24), (24, 1))


def _net_params(seed):
    """a network at the start of its training: per layer weights [27][cout][cin], biases"""
    r = np.random.default_rng([int(seed), 3])
    return np.concatenate([np.concatenate([r.normal(0.0, math.sqrt(2.0 / (27 * cin)), 27 * cout * cin),
                                           r.normal(0.0, 0.01, cout)]) for cin, cout in LAYERS]).astype(np.float32)


# ---------------------------------------------------------------------------


class _State:
    pass


def prepare(case, seed):
    s = _State()
    s.kind = case["kind"]
    if s.kind in ("step", "series", "host", "learned"):
        p, i0, u0, g, mask, balls = _step_inputs(case, seed)
        s.p, s.u0, s.u, s.g, s.mask, s.balls = p, u0, u0.clone(), g, mask, balls
        form = case.get("form", "mixed")
        s.solver = ss4d.Solver.for_interior(*_dims(case), arith=form)
        s.steps = case.get("steps", 1)
        if s.kind == "learned":
            s.net = ss4d.Wsnet(seed=None)
            s.net.set_params(np.load(os.path.join(PKG, "weights", "wsnet_seg.npy")))
            s.i0 = i0
            s.solver.set_warm_start(s.net, i0)
        if s.kind == "host":
            s.h_u0 = u0.cpu().pin_memory()
            s.h_u = torch.empty_like(s.h_u0).pin_memory()
            s.h_view = s.h_u.numpy()
    elif s.kind == "edge":
        s.p, s.src, s.src_thr = _edge_inputs(case, seed)
        s.i0 = s.src.clone()
        s.thr = None if s.src_thr is None else s.src_thr.clone()
        s.g = [torch.zeros_like(s.i0) for _ in range(8)]
        s.solver = ss4d.Solver.for_interior(*_dims(case), arith=case["form"])
    elif s.kind == "mcf":
        s.p, s.u0 = _mcf_start(case, seed)
        s.u = s.u0.clone()
        s.solver = ss4d.Solver.for_interior(*(case["n"],) * 4, arith=case["form"])
    elif s.kind == "batch":
        vols = _batch_inputs(case, seed)
        s.ps, s.u0s, s.gs = ([v[k] for v in vols] for k in range(3))
        s.us = [u.clone() for u in s.u0s]
        s.steps = case["steps"]
        s.batch = ss4d.Batch([tuple(u.shape[::-1]) for u in s.us])
        s.batch.set_arith("mixed")
        s.batch.set_projection(True)
    else:
        x, s.t = _train_inputs(case, seed)
        s.x = ss4d.features_to_planar(x.permute(0, 2, 3, 4, 1))
        s.dims = (case["nx"], case["ny"], case["nz"], case["crops"])
        s.net = ss4d.Wsnet(seed=None)
        s.net.set_params(_net_params(seed))
        s.grad = torch.zeros(s.net.nparam, dtype=torch.float32, device="cuda")
    return s


def run(s):
    if s.kind == "step":
        s.u.copy_(s.u0)
        st = s.solver.seg_time_step(s.p, s.u, None, s.g, s.mask, s.balls)
        return {"u": s.u, "iterations": st["iterations"]}
    if s.kind == "series":
        # a new time series: its start, and a history that begins with it
        s.u.copy_(s.u0)
        s.solver.set_extrapolation(3)
        s.solver.set_projection(True)
        its = [s.solver.seg_time_step(s.p, s.u, None, s.g)["iterations"] for _ in range(s.steps)]
        return {"u": s.u, "iterations": np.array(its, dtype=np.int64)}
    if s.kind == "learned":
        s.u.copy_(s.u0)
        st = s.solver.seg_time_step(s.p, s.u, None, s.g)
        return {"u": s.u, "iterations": st["iterations"], "warm": st["warm_started"]}
    if s.kind == "host":
        s.h_u.copy_(s.h_u0)
        st = s.solver.seg_time_step_host(s.p, s.h_view, s.u, s.g)
        return {"u": s.h_u, "iterations": st["iterations"]}
    if s.kind == "edge":
        # the detector smooths its images in place
        s.i0.copy_(s.src)
        if s.thr is not None:
            s.thr.copy_(s.src_thr)
        s.solver.edge_detector(s.p, s.i0, s.thr, s.g)
        return {"i0": s.i0, "thr": s.thr, "g": s.g}
    if s.kind == "mcf":
        s.u.copy_(s.u0)
        st = s.solver.mcf_time_step(s.p, 1, s.u)
        return {"u": s.u, "iterations": st["iterations"]}
    if s.kind == "batch":
        for u, u0 in zip(s.us, s.u0s):
            u.copy_(u0)
        s.batch.set_extrapolation(3)
        its = [[st["iterations"] for st in s.batch.seg_time_step(s.ps, s.us, s.gs)] for _ in range(s.steps)]
        return {"u": s.us, "iterations": np.array(its, dtype=np.int64)}
    loss = s.net.train_step(s.x, s.t, *s.dims, margin=CROP_MARGIN, lr=1e-3, grad=s.grad)
    return {"loss": loss, "grad": s.grad}


def work(case):
    """Bytes: u (or the image) in and out, the 8 g faces in (or out).  Operations: the
    assembly's about 200 per voxel and 20 per voxel and iteration, with the iterations
    a step of that kind takes."""
    kind = case["kind"]
    if kind == "train":
        v = case["nx"] * case["ny"] * case["nz"] * case["crops"]
        macs = 27 * (16 * 24 + 24 * 24 + 24 * 24 + 24)
        return {"bytes": v * (32 + 4), "flops": 2.0 * macs * v * 3}
    if kind == "mcf":
        v = case["n"] ** 4
        return {"bytes": 16 * v, "flops": v * (200 + 20 * 40)}
    if kind == "batch":
        r = random.Random(case["sizes"])
        v = 0
        for _ in range(case["volumes"]):
            n = [r.randint(case["lo"], case["hi"]) for _ in range(3)] + [r.randint(case["tlo"], case["thi"])]
            v += math.prod(n)
        return {"bytes": 80 * v, "flops": v * case["steps"] * (200 + 20 * 15)}
    v = math.prod(_dims(case))
    if kind == "edge":
        return {"bytes": v * (16 * case["images"] + 64), "flops": v * (case["images"] * (10 * 22 + 90) + 32)}
    if kind == "series":
        return {"bytes": 80 * v, "flops": v * case["steps"] * (200 + 20 * 15)}
    if kind == "learned":
        return {"bytes": 88 * v, "flops": v * (200 + 20 * 20 + 84240)}
    return {"bytes": (80 + (8 if case.get("balls") else 0)) * v, "flops": v * (200 + 20 * 30)}


def _bf16(t):
    return t + (t.detach().to(torch.bfloat16).double() - t.detach())


def exact(case, seed):
    kind = case["kind"]
    if kind in ("step", "series", "host", "learned"):
        v = math.prod(_dims(case))
        if v * case.get("steps", 1) > 60_000_000:
            return None
        p, _, u, g, mask, balls = _step_inputs(case, seed)
        plain = case.get("form", "mixed") == "fp64"
        for _ in range(case.get("steps", 1)):
            _exact_step(p, u, g, plain)
            if balls:
                _rescale(p, u, mask, balls)
        return {"u": u}
    if kind == "edge":
        p, i0, thr = _edge_inputs(case, seed)
        i0 = _presmooth(p, i0)
        thr = None if thr is None else _presmooth(p, thr)
        return {"i0": i0, "thr": thr, "g": _edges(p, i0, thr)}
    if kind == "mcf":
        p, u = _mcf_start(case, seed)
        a = _coefficients(p, u, None)
        prev = _at(u).clone()
        n, h = case["n"], p.h
        c = (torch.arange(n + 2, device="cuda", dtype=torch.float64) - 1) * h + h / 2 - 1.25
        x2 = c * c
        full = (x2[:, None, None, None] + x2[None, :, None, None] + x2[None, None, :, None]
                + x2[None, None, None, :] - 1.0) / 6.0 + p.tau
        inner = _at(u).clone()
        u.copy_(full)  # the ghosts: the known solution at t = tau
        _at(u).copy_(inner)
        if case["form"] == "fp64":
            _solve(p, u, prev, a)
        else:
            _solve(p, u, prev, a, tol=1e-24 * float((prev * prev).sum()) * h ** 4, omega=1.3)
        return {"u": u}
    if kind == "batch":
        if work(case)["bytes"] / 80 * case["steps"] > 60_000_000:
            return None
        us = []
        for p, u, g in _batch_inputs(case, seed):
            for _ in range(case["steps"]):
                _exact_step(p, u, g, False)
            us.append(u)
        return {"u": us}
    # the network with its BF16 weights and activations (rounding passed by in the backward)
    w0 = torch.from_numpy(_net_params(seed)).cuda().double().requires_grad_(True)
    x, t = _train_inputs(case, seed)
    a, off = x.double(), 0
    for k, (cin, cout) in enumerate(LAYERS):
        w = _bf16(w0[off:off + 27 * cin * cout]).reshape(3, 3, 3, cout, cin).permute(3, 4, 0, 1, 2)
        off += 27 * cin * cout
        a = torch.nn.functional.conv3d(a, w, w0[off:off + cout], padding=1)
        off += cout
        if k < 3:
            a = _bf16(torch.relu(a))
    m = CROP_MARGIN
    inner = (slice(None),) + tuple(slice(m, n - m) for n in (case["nz"], case["ny"], case["nx"]))
    loss = ((a[:, 0] - t.double())[inner] ** 2).mean()
    loss.backward()
    return {"loss": float(loss.detach()), "grad": w0.grad}
