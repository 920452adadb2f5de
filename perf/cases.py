"""Performance cases of the AL-DIC library: the calls a user's program makes,
over the sizes, data types and options it meets.

Kinds of case (the field "kind"):

  frame     one deformed image of an image pair or sequence on the uniform
            grid, from the raw image to the ADMM result: Context images set,
            then set_images(g=...) and frame().  init "search" starts from the
            whole-field integer search, "given" from the program's own
            prediction of the displacement (the later frames of a sequence).
  quadtree  one frame of the quadtree path on a plate with a hole.
  search    funIntegerSearch, the whole-field integer search alone.
  mg        funIntegerSearchMg, the multigrid search for large displacements.
  icgn      local_icgn, the subset registration of every node alone.
  subpb2    Subpb2, the finite-element global step alone.
  smooth    funSmoothDisp, the displacement smoothing.
  interp    ba_interp2, the bicubic sampler.
  predict   the learned initial guess's network, forward.
  train     one training step of that network.
"""
from __future__ import annotations

import importlib
import math

import numpy as np
import torch

aldic = importlib.import_module("2d_aldic_b200")

DEV = "cuda"
F64 = torch.float64


# ------------------------------------------------------------------ the cases
def listed():
    return [
        # the ordinary frame: 2048^2 8-bit camera, dense grid (59 k subsets), the
        # default FP32 sampling, initial guess searched
        dict(name="frame_2048_u8", kind="frame", width=2048, height=2048, dtype="u8", subset=32, step=8,
             search=16, precision="fp32", init="search", smooth=False, subpb2="fe", tol=1e-2, admm=3),
        # a small image in double precision throughout (1849 subsets): launches and
        # latency count
        dict(name="frame_512_u8_fp64", kind="frame", width=512, height=512, dtype="u8", subset=20, step=10,
             search=20, precision="fp64", init="search", smooth=False, subpb2="fe", tol=1e-3, admm=3),
        # a later frame of a 4096^2 16-bit sequence: the displacement is predicted from
        # earlier frames, nothing is searched
        dict(name="frame_4096_u16_given", kind="frame", width=4096, height=4096, dtype="u16", subset=32,
             step=16, search=24, precision="fp32", init="given", smooth=False, subpb2="fe", tol=1e-2, admm=3),
        # plate with a hole, quadtree mesh refined to the hole's edge, element-sized subsets
        dict(name="quadtree_2048", kind="quadtree", width=2048, height=2048, subset=32, step=16, search=16,
             min_size=2, precision="fp32"),
        # the first frames of a 16-bit sequence: the whole-field search by itself
        dict(name="search_2048_u16", kind="search", width=2048, height=2048, dtype="u16", subset=32, step=16,
             search=24, qfactors=False),
        # displacements larger than a subset
        dict(name="mg_2048_u8", kind="mg", width=2048, height=2048, dtype="u8", subset=32, step=16),
        # registration alone, on a ragged image whose grid is no round number either
        dict(name="icgn_1531x1187_u8", kind="icgn", width=1531, height=1187, dtype="u8", subset=32, step=8,
             precision="fp32", tol=1e-2),
        # the smallest call: one global step on a small grid
        dict(name="subpb2_43x43", kind="subpb2", M=43, N=43, step=10),
        # smoothing of a dense displacement field
        dict(name="smooth_243x243", kind="smooth", M=243, N=243),
        # the sampler over every pixel of an image
        dict(name="interp_2048_f64", kind="interp", width=2048, height=2048, points=2048 * 2048, dtype="f64"),
        # the learned guess for every node of a sparse grid
        dict(name="predict_16384", kind="predict", batch=16384),
        # one training step at the training loop's batch size
        dict(name="train_256", kind="train", batch=256),
    ]


def _logint(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


# subset, step and search radius as the configurations, tests and the reference's examples set them
_GEOMETRY = [(32, 8, 16), (32, 16, 16), (32, 16, 24), (24, 8, 12), (16, 8, 10), (16, 4, 8), (20, 10, 20),
             (20, 10, 35), (40, 10, 16), (28, 7, 13), (50, 25, 30)]


def draw(rng):
    while True:
        c = _draw(rng)
        if _cost(c) <= 1.0:
            return c


def _draw(rng):
    kind = rng.choice(["frame", "frame", "frame", "frame", "quadtree", "search", "search", "mg", "icgn", "icgn",
                       "subpb2", "smooth", "interp", "predict", "train"])
    if kind in ("subpb2", "smooth"):
        c = dict(kind=kind, M=_logint(rng, 9, 300), N=_logint(rng, 9, 300))
        if kind == "subpb2":
            c["step"] = rng.choice([4, 8, 10, 16])
        return c
    if kind == "predict":
        return dict(kind=kind, batch=_logint(rng, 16, 20000))
    if kind == "train":
        return dict(kind=kind, batch=_logint(rng, 16, 1024))
    w, h = _logint(rng, 300, 4096), _logint(rng, 300, 4096)
    if kind == "interp":
        return dict(kind=kind, width=w, height=h, points=_logint(rng, 1000, 2 * w * h),
                    dtype=rng.choice(["f64", "f64", "f32"]))
    sub, step, search = rng.choice(_GEOMETRY)
    if kind == "quadtree":
        return dict(kind=kind, width=min(max(w, 512), 2048), height=min(max(h, 512), 2048), subset=32, step=16,
                    search=rng.choice([8, 13, 16]), min_size=rng.choice([2, 4]),
                    precision=rng.choice(["fp32", "fp32", "fp64"]))
    if kind == "mg":
        return dict(kind=kind, width=min(w, 2048), height=min(h, 2048), dtype=rng.choice(["u8", "u16"]),
                    subset=rng.choice([16, 32]), step=rng.choice([8, 16]))
    dtype = rng.choice(["u8", "u8", "u16"])
    if kind == "search":
        return dict(kind=kind, width=w, height=h, dtype=dtype, subset=sub, step=step, search=search,
                    qfactors=rng.random() < 0.25)
    prec = rng.choice(["fp32", "fp32", "fp32", "fp64"])
    tol = rng.choice([1e-2, 1e-2, 1e-3])
    if kind == "icgn":
        return dict(kind=kind, width=w, height=h, dtype=dtype, subset=sub, step=step, precision=prec, tol=tol)
    return dict(kind=kind, width=w, height=h, dtype=dtype, subset=sub, step=step, search=search, precision=prec,
                init=rng.choice(["search", "search", "given"]), smooth=rng.random() < 0.25,
                subpb2=rng.choice(["fe", "fe", "fe", "fd"]), tol=tol, admm=3)


def _cost(c):
    """Roughly the work of a case over that of the largest listed ones (1 at most is drawn)."""
    k = c["kind"]
    if k in ("frame", "search", "icgn"):
        M, N = _nodes(c)
        if M < 6 or N < 6:
            return 2.0
        taps = (c["subset"] + 1) ** 2
        cost = 0.0
        if k == "search" or (k == "frame" and c["init"] == "search"):
            shifts = (2 * c["search"] + 3) ** 2
            cost += M * N * taps * shifts / (13.5e10 if c["dtype"] == "u8" else 4.5e10)
            if c.get("qfactors"):
                cost += M * N * taps * (2 * c["subset"] + 2 * c["search"] + 1) ** 2 / 1.2e10
        if k in ("frame", "icgn"):
            cost += M * N * taps * (8 if c["precision"] == "fp64" else 1) / (1.1e8 if k == "frame" else 3.8e8)
        if c.get("smooth"):
            cost += 0.4 * M * N / 59049.0
        return max(cost, c["width"] * c["height"] / 4096 ** 2, M * N / 65536.0)
    if k == "mg":
        return c["width"] * c["height"] / 2048 ** 2 * (32 / c["subset"])
    if k in ("subpb2", "smooth"):
        return c["M"] * c["N"] / 65536.0
    if k == "interp":
        return c["points"] / 4.5e6
    return 1.0


# ------------------------------------------------------------------ inputs
def _gen(seed, salt):
    return torch.Generator(device=DEV).manual_seed(int(seed) * 977 + salt)


def _bicubic(img, X, Y):
    """Keys' cubic convolution (a = -1/2), clamped, at 1-based (X, Y); img[y, x]."""
    H, W = img.shape
    flat = img.reshape(-1)
    xf, yf = torch.floor(X), torch.floor(Y)
    tx, ty = X - xf, Y - yf

    def weights(t):
        return (0.5 * (-t + 2 * t * t - t ** 3), 0.5 * (2 - 5 * t * t + 3 * t ** 3),
                0.5 * (t + 4 * t * t - 3 * t ** 3), 0.5 * (-t * t + t ** 3))
    wx, wy = weights(tx), weights(ty)
    xi, yi = xf.long() - 1, yf.long() - 1
    out = torch.zeros_like(X)
    for a in range(4):
        row = (yi - 1 + a).clamp(0, H - 1) * W
        s = torch.zeros_like(X)
        for b in range(4):
            s += wx[b] * flat[row + (xi - 1 + b).clamp(0, W - 1)]
        out += wy[a] * s
    return out


def _speckle(W, H, seed):
    """Dots of radius 2, 3 and 4 px (profile A exp(-d^2 / r^2), A in 60..140), 0.031 dots a
    pixel, on a background of 20 grey levels: a well exposed speckle pattern."""
    g = _gen(seed, 1)
    img = torch.full((H, W), 20.0, dtype=F64, device=DEV)
    for r in (2.0, 3.0, 4.0):
        a = torch.rand((H, W), generator=g, device=DEV, dtype=torch.float32)
        dots = torch.where(a < 0.0103, 60 + 80 * torch.rand((H, W), generator=g, device=DEV), torch.zeros((), device=DEV))
        R = int(3 * r)
        for dim in (0, 1):
            n = dots.shape[dim]
            acc = dots.clone()
            for k in range(1, R + 1):
                c = math.exp(-k * k / (r * r))
                acc.narrow(dim, k, n - k).add_(dots.narrow(dim, 0, n - k), alpha=c)
                acc.narrow(dim, 0, n - k).add_(dots.narrow(dim, k, n - k), alpha=c)
            dots = acc
        img += dots
    return img


def _field(seed, u0, v0, amp, period):
    p = _gen_phase(seed)

    def at(X, Y):
        return (u0 + amp * torch.sin(2 * math.pi * Y / period + p[0]),
                v0 + 0.75 * amp * torch.cos(2 * math.pi * X / period + p[1]))
    return at


def _gen_phase(seed):
    return np.random.default_rng(seed + 5).uniform(0, 2 * math.pi, 2)


def _warped(f, field):
    H, W = f.shape
    y, x = torch.meshgrid(torch.arange(1, H + 1, dtype=F64, device=DEV), torch.arange(1, W + 1, dtype=F64, device=DEV),
                          indexing="ij")
    X, Y = x, y
    for _ in range(12):
        u, v = field(X, Y)
        X, Y = x - u, y - v
    return _bicubic(f, X, Y)


def _quantised(img, dtype):
    if dtype == "u16":
        return torch.clamp(torch.round(img * 257.0), 0, 65535).to(torch.int32).to(torch.uint16)
    return torch.clamp(torch.round(img), 0, 255).to(torch.uint8)


def _noisy(img, seed, salt, dtype):
    sigma = 30.0 / 257.0 if dtype == "u16" else 2.0
    return img + sigma * torch.randn(img.shape, generator=_gen(seed, salt), dtype=F64, device=DEV)


def _pair(c, seed, field=None):
    """(f, g, field): the reference image, the deformed one and its displacement."""
    dtype = c.get("dtype", "u8")
    base = _speckle(c["width"], c["height"], seed)
    field = field or _field(seed, 0.4, -0.3, 1.5, 256.0)
    f = _quantised(_noisy(base, seed, 2, dtype), dtype)
    g = _quantised(_noisy(_warped(base, field), seed, 3, dtype), dtype)
    return f, g, field


def _nodes(c):
    """M, N of the whole-field search grid (funIntegerSearch.m:14-25, :90-91)."""
    s = c.get("search", 8)
    lo = int(math.ceil(1 + s + 0.5 * c["subset"]))
    n = []
    for size in (c["width"], c["height"]):
        hi = int(math.floor(size - 1.5 * c["subset"] - s))
        n.append((hi - c["step"] - lo) // c["step"] + 1 if hi - c["step"] >= lo else 0)
    return n[0], n[1]


def _grid(c):
    """Node coordinates (n x 2, x fastest) of that grid."""
    M, N = _nodes(c)
    first = int(math.ceil(1 + c.get("search", 8) + 0.5 * c["subset"])) + 0.5 * c["subset"]
    x = first + c["step"] * torch.arange(M, dtype=F64, device=DEV)
    y = first + c["step"] * torch.arange(N, dtype=F64, device=DEV)
    yy, xx = torch.meshgrid(y, x, indexing="ij")
    return torch.stack([xx.reshape(-1), yy.reshape(-1)], 1)


def _guess(c, seed, field):
    """A prediction of the displacement at the nodes, good to about 0.1 px."""
    xy = _grid(c)
    u, v = field(xy[:, 0], xy[:, 1])
    U = torch.stack([u, v], 1)
    return (U + 0.1 * torch.randn(U.shape, generator=_gen(seed, 9), dtype=F64, device=DEV)).reshape(-1).contiguous()


def _node_fields(c, seed):
    """Displacement, gradient and dual fields of an M x N grid as an ADMM step leaves them."""
    M, N = c["M"], c["N"]
    g = _gen(seed, 11)
    n = M * N

    def smooth(k, amp, noise):
        j, i = torch.meshgrid(torch.arange(N, dtype=F64, device=DEV), torch.arange(M, dtype=F64, device=DEV), indexing="ij")
        ph = _gen_phase(seed)
        cols = [amp * torch.sin(0.05 * (q + 1) * i + 0.07 * j + ph[q % 2]).reshape(-1) for q in range(k)]
        return (torch.stack(cols, 1) + noise * torch.randn((n, k), generator=g, dtype=F64, device=DEV)).reshape(-1).contiguous()
    return smooth(2, 2.0, 0.02), smooth(4, 0.02, 0.002), smooth(4, 0.001, 0.001), smooth(2, 0.005, 0.005)


_COUT, _CIN = (128, 128, 256, 8), (64, 128, 4096, 256)


def _weights(seed):
    r = np.random.default_rng(seed + 17)
    parts = []
    for co, ci in zip(_COUT, _CIN):
        parts += [(r.standard_normal(co * ci) * math.sqrt(2.0 / ci)), 0.05 * r.standard_normal(co)]
    return np.concatenate(parts).astype(np.float32)


def _patches(c, seed):
    """Normalised 64 x 64 patch pairs of a speckle image, the deformed ones shifted by up to 8 px."""
    B = c["batch"]
    S = _speckle(1024, 1024, seed).to(torch.float32)
    S = (S - S.mean()) / S.std()
    g = _gen(seed, 21)
    xy = torch.randint(16, 1024 - 64 - 16, (B, 2), generator=g, device=DEV)
    sh = torch.randint(-8, 9, (B, 2), generator=g, device=DEV)
    r = torch.arange(64, device=DEV)

    def cut(p):
        return S[(p[:, 1, None, None] + r[None, :, None]), (p[:, 0, None, None] + r[None, None, :])]
    x = torch.stack([cut(xy), cut(xy + sh)], -1).to(torch.bfloat16).contiguous()
    t = torch.zeros((B, 6), dtype=torch.float32, device=DEV)
    t[:, :2] = -sh / 16.0
    t[:, 2:] = 0.3 * torch.randn((B, 4), generator=g, device=DEV)
    return x, t


def prepare(case, seed):
    c, k = case, case["kind"]
    if k == "frame":
        f, g, field = _pair(c, seed)
        al = aldic.ALDIC(c["subset"], c["step"], c["search"], tol=c["tol"], n_admm=c["admm"],
                         precision=aldic.FP64 if c["precision"] == "fp64" else aldic.FP32, smooth=c["smooth"],
                         subpb2=c["subpb2"], ctx=aldic.Context(0))
        s = dict(kind=k, al=al, g=g, init=aldic.INIT_SEARCH, U0=None)
        if c["init"] == "given":
            s["init"], s["U0"] = aldic.INIT_GIVEN, _guess(c, seed, field)
        # the program is in its loop over the images: it has processed one before (here the
        # undeformed specimen again, with other noise)
        al.set_images(f, _quantised(_noisy(_speckle(c["width"], c["height"], seed), seed, 4, c["dtype"]), c["dtype"]))
        if s["U0"] is not None:
            al.set_init(torch.zeros_like(s["U0"]))
        al.frame(device_out=True, stats=False, init=s["init"])
        return s
    if k == "quadtree":
        cx, cy, rad = 0.5 * c["width"], 0.5 * c["height"], 0.15 * min(c["width"], c["height"])

        def plate(X, Y):
            dx, dy = X - cx, Y - cy
            r2 = (dx * dx + dy * dy).clamp_min(1e-12)
            inside = r2 < rad * rad
            z = torch.zeros((), dtype=F64, device=DEV)
            return torch.where(inside, z, 0.002 * dx * (1.0 + rad * rad / r2)), torch.where(inside, z, -0.0006 * dy)
        f, g, _ = _pair(c, seed, plate)
        yy, xx = np.mgrid[1:c["height"] + 1, 1:c["width"] + 1]
        mask = ((xx - cx) ** 2 + (yy - cy) ** 2 >= rad * rad).astype(np.float64)
        qt = aldic.ALDICQuadtree(c["subset"], c["step"], c["search"], min_size=c["min_size"], subsets="element",
                                 precision=aldic.FP64 if c["precision"] == "fp64" else aldic.FP32, ctx=aldic.Context(0))
        qt.set_images(f, f, mask)
        qt.frame()      # the loop's earlier image: the mesh is there
        qt.g = g
        return dict(kind=k, qt=qt)
    if k == "search":
        f, g, _ = _pair(c, seed)
        return dict(kind=k, c=c, f=f, g=g)
    if k == "mg":
        f, g, _ = _pair(c, seed, _field(seed, 26.0, -21.0, 3.0, 1024.0))
        return dict(kind=k, c=c, f=f, g=g)
    if k == "icgn":
        f, g, field = _pair(c, seed)
        ctx = aldic.Context(0)
        ctx.set_ref(f)
        ctx.set_def(g)
        U0 = _guess(c, seed, field)
        return dict(kind=k, c=c, ctx=ctx, xy=_grid(c), U0=torch.round(U0 * 4) / 4)
    if k == "subpb2":
        U, F, ud, vd = _node_fields(c, seed)
        x = 20.0 + c["step"] * np.arange(c["M"])
        y = 20.0 + c["step"] * np.arange(c["N"])
        mesh = aldic.MeshSetUp(np.tile(x, (c["N"], 1)), np.tile(y[:, None], (1, c["M"])), {"ImgSize": (0, 0)})
        return dict(kind=k, mesh=mesh, beta=1e-2 * c["step"] ** 2 * 1e-3, U=U, F=F, ud=ud, vd=vd)
    if k == "smooth":
        return dict(kind=k, U=_node_fields(c, seed)[0], mesh={"M": c["M"], "N": c["N"]})
    if k == "interp":
        F, X, Y = _interp_inputs(c, seed)
        return dict(kind=k, F=F, X=X, Y=Y)
    if k in ("predict", "train"):
        net = aldic.InitNet(0, seed=1)
        net.set_params(_weights(seed))
        x, t = _patches(c, seed)
        return dict(kind=k, net=net, x=x, t=t)
    raise ValueError(k)


def _interp_inputs(c, seed):
    """An image and the points of a smooth deformation of it, in raster order."""
    dt = torch.float64 if c["dtype"] == "f64" else torch.float32
    F = _speckle(c["width"], c["height"], seed)
    n = c["points"]
    W, H = c["width"], c["height"]
    cols = max(1, int(round(math.sqrt(n * W / H))))
    k = torch.arange(n, dtype=F64, device=DEV)
    x = 1 + (k % cols) * ((W - 1) / max(1, cols - 1))
    y = 1 + torch.floor(k / cols) * ((H - 1) / max(1.0, math.ceil(n / cols) - 1))
    u, v = _field(seed, 0.4, -0.3, 1.5, 256.0)(x, y)
    # ba_interp2's X runs along the slow axis of the array it is given, Y along the fast one
    return F.to(dt), (y + v).to(dt), (x + u).to(dt)


# ------------------------------------------------------------------ one pass
def run(state):
    s, k = state, state["kind"]
    if k == "frame":
        al = s["al"]
        al.set_images(g=s["g"])
        if s["U0"] is not None:
            al.set_init(s["U0"])
        r = al.frame(device_out=True, stats=False, init=s["init"])
        return {q: r[q] for q in ("x0", "y0", "U", "F", "iters")}
    if k == "quadtree":
        r = s["qt"].frame()
        return {q: r[q] for q in ("coords", "U", "F", "U_icgn", "iters_icgn", "beta")}
    if k == "search":
        c = s["c"]
        x, y, u, v, cc = aldic.funIntegerSearch(s["f"], s["g"], c["search"], [1, c["width"]], [1, c["height"]],
                                                c["subset"], c["step"], 0, c["step"], qfactors=c["qfactors"])
        out = {"x": x, "y": y, "u": u, "v": v, "max": cc["max"]}
        if c["qfactors"]:
            out["qfactors"] = cc["qfactors"]
        return out
    if k == "mg":
        c = s["c"]
        x, y, u, v, cc = aldic.funIntegerSearchMg(s["f"], s["g"], [1, c["width"]], [1, c["height"]], c["subset"],
                                                  c["step"], c["step"])
        return {"x": x, "y": y, "u": u, "v": v, "max": cc["max"], "qfactors": cc["qfactors"]}
    if k == "icgn":
        c = s["c"]
        U, F, it, H = aldic.local_icgn(s["ctx"], s["xy"], s["U0"], c["subset"], c["tol"],
                                       aldic.FP64 if c["precision"] == "fp64" else aldic.FP32)
        return {"U": U, "F": F, "iters": it, "H": H}
    if k == "subpb2":
        return {"Uhat": aldic.Subpb2(s["mesh"], s["beta"], 1e-3, s["U"], s["F"], s["ud"], s["vd"])}
    if k == "smooth":
        return {"U": aldic.funSmoothDisp(s["U"], s["mesh"])}
    if k == "interp":
        return {"Z": aldic.ba_interp2(s["F"], s["X"], s["Y"])}
    if k == "predict":
        return {"out": s["net"].predict(s["x"])}
    loss, grads, out = s["net"].train_step(s["x"], s["t"], 3e-4, grads=True, outputs=True)
    return {"loss": loss, "grads": grads, "out": out}


# ------------------------------------------------------------------ what a pass cannot do without
_PX = {"u8": 1, "u16": 2, "f32": 4, "f64": 8}
_EVALS = 4      # subset evaluations of a registration, about


def _icgn_work(c, n):
    N = (c["subset"] + 1) ** 2
    real = 8 if c["precision"] == "fp64" else 4
    # per pixel: sampling 40 and residual sums 16 an evaluation, 50 for the Hessian and the
    # reference's sums; the images read once each, U, F and 21 entries of H written
    return {"bytes": 4 * real * c["width"] * c["height"] + n * 8 * 28, "flops": n * N * (56 * _EVALS + 50)}


def _solve_work(M, N, fields):
    """One direct solve by separation of variables."""
    return 4 * fields * M * N * (M + N)


def work(case):
    c, k = case, case["kind"]
    if k == "frame":
        M, N = _nodes(c)
        n = M * N
        w = _icgn_work(c, n)
        px = c["width"] * c["height"]
        w["bytes"] += px * _PX[c["dtype"]] * 2 + n * 8 * 9
        if c["init"] == "search":
            w["flops"] += 2 * px * (2 * c["search"] + 3) ** 2
        w["flops"] += c["admm"] * n * (c["subset"] + 1) ** 2 * 48 * 3 + (6 + c["admm"]) * _solve_work(M, N, 2)
        return w
    if k == "quadtree":
        n = c["width"] * c["height"] / c["step"] ** 2
        px = c["width"] * c["height"]
        w = _icgn_work(c, n)
        return {"bytes": w["bytes"] + 2 * px + n * 8 * 12, "flops": w["flops"] * 1.5 + 2 * px * (2 * c["search"] + 3) ** 2}
    if k == "search":
        px = c["width"] * c["height"]
        M, N = _nodes(c)
        shifts = (2 * c["search"] + 3) ** 2
        if c["qfactors"]:
            shifts = (2 * c["subset"] + 2 * c["search"] + 1) ** 2
        # each product of two pixels once, however many windows share it
        return {"bytes": 2 * px * _PX[c["dtype"]] + M * N * 8 * 5, "flops": 2 * px * shifts}
    if k == "mg":
        px = c["width"] * c["height"]
        # the whole-field correlation by transforms, then 13 x 14 shifts a level
        levels = math.ceil(math.log2(max(c["width"], c["height"]) / c["subset"]))
        n = px / c["step"] ** 2
        return {"bytes": 2 * px * _PX[c["dtype"]] + n * 8 * 7,
                "flops": 3 * 5 * 4 * px * math.log2(4 * px) + 2 * px * 182 * levels}
    if k == "icgn":
        M, N = _nodes(c)
        return _icgn_work(c, M * N)
    if k == "subpb2":
        n = c["M"] * c["N"]
        return {"bytes": 8 * 14 * n + 8 * (c["M"] ** 2 + c["N"] ** 2), "flops": _solve_work(c["M"], c["N"], 2)}
    if k == "smooth":
        n = c["M"] * c["N"]
        return {"bytes": 8 * 4 * n, "flops": 2 * 2 * n * (10 * 20 + 20)}
    if k == "interp":
        b = _PX[c["dtype"]]
        return {"bytes": b * (c["width"] * c["height"] + 3 * c["points"]), "flops": 60 * c["points"]}
    B = c["batch"]
    mac = B * (2 * 64 * (64 * 128 + 128 * 128) + 64 * 64 * 128 + 4096 * 256 + 256 * 8)
    params = sum(co * ci + co for co, ci in zip(_COUT, _CIN))
    if k == "predict":
        return {"bytes": B * (64 * 64 * 2 * 2 + 8 * 4) + 2 * params, "flops": 2 * mac}
    return {"bytes": B * (64 * 64 * 2 * 2 + 14 * 4) + params * 4 * 8, "flops": 6 * mac}


# ------------------------------------------------------------------ how far a correct answer may be off
def tolerance(case):
    c, k = case, case["kind"]
    fp32 = c.get("precision") == "fp32"
    if k in ("frame", "icgn", "quadtree") and not fp32:
        return {"rel": 1e-8, "max": 1e-6, "differ": 1e-3}
    # FP32: 1e-7 as long as every stopping test falls the same way; a subset whose test falls
    # the other way moves by one last step (0.01 px and 0.002 in the gradient)
    if k == "icgn":
        return {"rel": 2e-4, "max": 0.05, "differ": 2e-3}
    if k == "frame":
        return {"rel": 1e-3, "max": 0.3, "differ": 5e-3}
    if k == "quadtree":
        # the same, and its refined elements of 4 px magnify it: 1e-2 in F between FP32 and FP64
        return {"rel": 0.03, "max": 0.99, "differ": 5e-3}
    if k in ("search", "mg"):
        # u and v are rounded to 1e-3 px, the q-factors count histogram bins
        return {"rel": 2e-5, "max": 5e-3}
    if k == "subpb2":
        return {"rel": 1e-12, "max": 1e-11}
    if k == "smooth":
        # solved to a relative residual of 1e-11
        return {"rel": 5e-11, "max": 5e-10}
    if k == "interp":
        return {"rel": 1e-14, "max": 1e-12} if c["dtype"] == "f64" else {"rel": 1e-6, "max": 1e-5}
    # bf16 operands and activations: 3e-3 in the outputs and 8e-3 in the gradients against 64 bits
    return {"rel": 1.5e-2, "max": 0.3} if k == "predict" else {"rel": 0.03, "max": 0.5}


# ------------------------------------------------------------------ the same in 64 bits, plainly
def exact(case, seed):
    c, k = case, case["kind"]
    if k in ("quadtree", "mg"):
        return None     # region by region and element by element: far over 20 s in plain torch
    if k == "frame":
        return None if c["subpb2"] == "fd" else _exact_frame(c, seed)
    if k == "search":
        f, g, _ = _pair(c, seed)
        r = _exact_search(c, f, g, c["qfactors"])
        if c["qfactors"]:
            r["qfactors"] = torch.stack(r.pop("q"), 1)
        else:
            r.pop("q")
        return r
    if k == "icgn":
        f, g, field = _pair(c, seed)
        U0 = torch.round(_guess(c, seed, field) * 4) / 4
        fn, gn = _normalised(f), _normalised(g)
        r = _exact_icgn(fn, gn, *_gradient(fn), _grid(c), U0.reshape(-1, 2), c["subset"], c["tol"])
        return {"U": r["U"].reshape(-1), "F": r["F"].reshape(-1), "iters": None, "H": r["H21"]}
    if k == "subpb2":
        U, F, ud, vd = _node_fields(c, seed)
        return {"Uhat": _fe_solve(c["M"], c["N"], c["step"], 1e-2 * c["step"] ** 2 * 1e-3, 1e-3, U, F, ud, vd)}
    if k == "smooth":
        return {"U": _smoothed(c["M"], c["N"], _node_fields(c, seed)[0], 2)}
    if k == "interp":
        F, X, Y = (t.to(F64) for t in _interp_inputs(c, seed))
        return {"Z": _bicubic(F, Y, X)}
    p = torch.from_numpy(_weights(seed)).to(DEV, F64).requires_grad_(k == "train")
    x, t = _patches(c, seed)
    if k == "predict":
        return {"out": torch.cat([_net(p, x[i:i + 512].to(F64)) for i in range(0, c["batch"], 512)]).to(torch.float32)}
    out = _net(p, x.to(F64))
    e = out[:, :6] - t.to(F64)
    z = out[:, 6]
    near = (e[:, :2].abs().max(1).values * 16.0 < 0.5).to(F64).detach()
    loss = ((e ** 2).sum() + torch.nn.functional.binary_cross_entropy_with_logits(z, near, reduction="sum")) / c["batch"]
    loss.backward()
    return {"loss": float(loss.detach()), "grads": p.grad.cpu().numpy(), "out": out.detach().cpu().numpy()}


def _net(p, x):
    B, o, L = x.shape[0], 0, []
    for co, ci in zip(_COUT, _CIN):
        L.append((p[o:o + co * ci].view(co, ci), p[o + co * ci:o + co * ci + co]))
        o += co * ci + co

    def encode(y):
        cells = y.view(B, 8, 8, 8, 8).permute(0, 1, 3, 2, 4).reshape(B, 64, 64)
        return torch.relu(cells @ L[0][0].T + L[0][1]) @ L[1][0].T + L[1][1]
    corr = (encode(x[..., 0]) @ encode(x[..., 1]).transpose(1, 2)) / math.sqrt(128.0)
    h = torch.relu(corr.reshape(B, 4096) @ L[2][0].T + L[2][1])
    return h @ L[3][0].T + L[3][1]


def _normalised(img):
    a = img.to(F64)
    return (a - a.mean()) / a.std()


def _gradient(f):
    gx, gy = torch.zeros_like(f), torch.zeros_like(f)
    H, W = f.shape

    def d(a, k, dim):
        n = a.shape[dim]
        return a.narrow(dim, 3 + k, n - 6) - a.narrow(dim, 3 - k, n - 6)
    gx[:, 3:W - 3] = 0.75 * d(f, 1, 1) - 0.15 * d(f, 2, 1) + d(f, 3, 1) / 60
    gy[3:H - 3, :] = 0.75 * d(f, 1, 0) - 0.15 * d(f, 2, 0) + d(f, 3, 0) / 60
    gx[:3], gx[H - 3:], gy[:, :3], gy[:, W - 3:] = 0, 0, 0, 0
    return gx, gy


def _exact_search(c, f, g, qfactors):
    M, N = _nodes(c)
    w, s, step = c["subset"], c["search"], c["step"]
    tw, dw = w + 1, w + 1 + 2 * s
    n = dw + tw
    xy = (_grid(c) - 0.5 * w).long() - 1                       # 0-based template corner
    fa, ga = f.to(F64), g.to(F64)
    ga = ga - ga.mean()                                        # outside of the region reads the mean
    W = f.shape[1]
    ar = torch.arange
    res = []
    for i0 in range(0, M * N, 512):
        p = xy[i0:i0 + 512]
        tx, dx = ar(tw, device=DEV), ar(dw, device=DEV) - s
        T = fa.reshape(-1)[(p[:, 1, None, None] + tx[None, :, None]) * W + p[:, 0, None, None] + tx[None, None, :]]
        D = ga.reshape(-1)[(p[:, 1, None, None] + dx[None, :, None]) * W + p[:, 0, None, None] + dx[None, None, :]]
        T = T - T.mean((1, 2), keepdim=True)
        den_t = (T * T).sum((1, 2))
        num = torch.fft.irfft2(torch.fft.rfft2(D, (n, n)) * torch.fft.rfft2(T, (n, n)).conj(), (n, n))
        full = dw + w                                          # offsets -w .. dw - 1
        at = (ar(full, device=DEV) - w) % n
        num = num[:, at][:, :, at]

        def box(a):
            a = torch.nn.functional.pad(a, (w + 1, w, w + 1, w)).cumsum(1).cumsum(2)
            return a[:, tw:, tw:] - a[:, :-tw, tw:] - a[:, tw:, :-tw] + a[:, :-tw, :-tw]
        s1, s2 = box(D), box(D * D)
        var = s2 - s1 * s1 / tw ** 2
        ncc = torch.where(var > 0, num / torch.sqrt(den_t[:, None, None] * var.clamp_min(1e-300)), torch.zeros_like(num))
        ncc = torch.where(ncc.abs() > 1 + 1.5e-8, torch.zeros_like(ncc), ncc)
        crop = ncc[:, w - 1:w + 2 * s + 2, w - 1:w + 2 * s + 2]
        q = None
        if qfactors:
            v = (ncc - ncc.amin((1, 2), keepdim=True)).reshape(len(p), -1)
            pk = v.amax(1)
            b = (v / pk[:, None] * 30).floor().clamp(0, 29).long()
            prob = torch.zeros((len(p), 30), dtype=F64, device=DEV).scatter_add_(1, b, torch.ones_like(v)) / v.shape[1]
            ent = torch.where(prob > 0, -prob * torch.log(prob.clamp_min(1e-300)), torch.zeros_like(prob)).sum(1)
            q = (pk * pk / (v * v).mean(1), 1 / ent)
        res.append((*_peak(crop, s), *(q or ())))
    u, v, m = (torch.cat([r[i] for r in res]).view(N, M) for i in range(3))
    out = {"x": _grid(c)[:, 0].view(N, M), "y": _grid(c)[:, 1].view(N, M), "u": u, "v": v, "max": m, "q": None}
    if qfactors:
        qs = [torch.cat([r[i] for r in res]) for i in (3, 4)]
        out["q"] = [(a - a.min()) / (a - a.min()).max() for a in qs]
    return out


def _peak(crop, s):
    """u, v and height of each map's peak: a quadratic through the 3 x 3 entries about the
    largest, the position rounded to 1e-3 (findpeak.m)."""
    n, R, _ = crop.shape
    k = crop.reshape(n, -1).argmax(1)
    r, cl = k % R, k // R                                      # x and y shift
    inner = (r > 0) & (r < R - 1) & (cl > 0) & (cl < R - 1)
    rc, cc = r.clamp(1, R - 2), cl.clamp(1, R - 2)
    o = torch.arange(-1, 2, device=DEV)
    B = crop[torch.arange(n, device=DEV)[:, None, None], cc[:, None, None] + o[None, :, None], rc[:, None, None] + o[None, None, :]]
    yy, xx = torch.meshgrid(o.to(F64), o.to(F64), indexing="ij")   # yy: along y shifts, xx: along x shifts
    A = torch.stack([torch.ones(9, dtype=F64, device=DEV), yy.reshape(-1), xx.reshape(-1), (xx * yy).reshape(-1),
                     (yy * yy).reshape(-1), (xx * xx).reshape(-1)], 1)
    P = B.reshape(n, 9) @ torch.linalg.pinv(A).T
    a1, a2, a3, a4, a5, a6 = P.T
    den = a4 * a4 - 4 * a5 * a6
    yo = (-a3 * a4 + 2 * a6 * a2) / den
    xo = (-a2 * a4 + 2 * a5 * a3) / den
    ok = inner & (xo.abs() <= 1) & (yo.abs() <= 1)
    xo, yo = torch.round(1000 * xo) / 1000, torch.round(1000 * yo) / 1000
    top = a1 + a2 * yo + a3 * xo + a4 * xo * yo + a5 * yo * yo + a6 * xo * xo
    z = torch.zeros_like(xo)
    u = r + 1 + torch.where(ok, xo, z) - (s + 2)
    v = cl + 1 + torch.where(ok, yo, z) - (s + 2)
    return u, v, torch.where(ok, top, crop.reshape(n, -1).amax(1))


def _composed(P, d):
    """P after the inverse-compositional step d (both n x 6: F11-1, F21, F12, F22-1, u, v)."""
    def mat(q):
        m = torch.zeros((len(q), 3, 3), dtype=F64, device=DEV)
        m[:, 0, 0], m[:, 0, 1], m[:, 0, 2] = 1 + q[:, 0], q[:, 2], q[:, 4]
        m[:, 1, 0], m[:, 1, 1], m[:, 1, 2] = q[:, 1], 1 + q[:, 3], q[:, 5]
        m[:, 2, 2] = 1
        return m
    m = mat(P) @ torch.linalg.inv(mat(d))
    return torch.stack([m[:, 0, 0] - 1, m[:, 1, 0], m[:, 0, 1], m[:, 1, 1] - 1, m[:, 0, 2], m[:, 1, 2]], 1)


def _subsets(fn, gx, gy, xy, w):
    """Each subset's reference values, gradients and offsets from its centre, flattened."""
    W = fn.shape[1]
    o = torch.arange(w + 1, device=DEV)
    x0 = (xy - 0.5 * w).long()
    px = (x0[:, 0, None, None] + o[None, None, :]).expand(-1, w + 1, -1).reshape(len(xy), -1)
    py = (x0[:, 1, None, None] + o[None, :, None]).expand(-1, -1, w + 1).reshape(len(xy), -1)
    at = (py - 1) * W + px - 1
    return (fn.reshape(-1)[at], gx.reshape(-1)[at], gy.reshape(-1)[at], px.to(F64) - xy[:, :1], py.to(F64) - xy[:, 1:])


def _windows(fn, gx, xy, w):
    """The subset size each node ends with: half of it masked (zero gradient) gives up (status
    102), over a tenth makes it grow, which fails (-1) where it has no whole-pixel bounds."""
    H, W = fn.shape
    zero = torch.nn.functional.pad((gx == 0).to(F64), (1, 0, 1, 0)).cumsum(0).cumsum(1)
    x0, y0 = (xy - 0.5 * w).long().T
    n = w + 1
    cnt = zero[y0 - 1 + n, x0 - 1 + n] - zero[y0 - 1, x0 - 1 + n] - zero[y0 - 1 + n, x0 - 1] + zero[y0 - 1, x0 - 1]
    size = torch.full((len(xy),), w, dtype=torch.int64, device=DEV)
    big = int(math.floor(math.sqrt(2.0) * w + 0.5))
    lo, hi = xy - 0.5 * big, xy + 0.5 * big
    fits = (lo == lo.floor()).all(1) & (lo >= 4).all(1) & (hi[:, 0] <= W - 3) & (hi[:, 1] <= H - 3)
    size[cnt > 0.1 * n * n] = -1
    size[(cnt > 0.1 * n * n) & fits] = big
    size[cnt >= 0.5 * n * n] = 102
    return size, big


def _residual(gn, P, xy, X, Y, fbar, bf):
    u = (1 + P[:, :1]) * X + P[:, 2:3] * Y + xy[:, :1] + P[:, 4:5]
    v = P[:, 1:2] * X + (1 + P[:, 3:4]) * Y + xy[:, 1:] + P[:, 5:6]
    H, W = gn.shape
    out = ((u < 3) | (u > W - 2) | (v < 3) | (v > H - 2)).any(1)
    g = _bicubic(gn, u, v)
    g = g - g.mean(1, keepdim=True)
    return fbar / bf - g / g.norm(dim=1, keepdim=True), out


def _iterate(n, step):
    """The stopping rule of funICGN.m:249-261 around step(rows, count): (norm, apply)."""
    iters = torch.full((n,), 101, dtype=torch.int64, device=DEV)
    first = torch.ones(n, dtype=F64, device=DEV)
    live = torch.arange(n, device=DEV)
    for it in range(1, 102):
        if not len(live):
            break
        live = step(live, it, iters, first)
    return iters


def _stopped(live, it, iters, first, nrm, out, tol):
    if it == 1:
        first[live] = nrm
    rel = torch.where(first[live] > tol, nrm / first[live], torch.zeros_like(nrm))
    done = ((rel < tol) | (nrm < tol)) & ~out
    iters[live[done]] = it
    return ~(done | out)


def _chunks(size, big, w):
    """(rows, subset size) in pieces of at most 4096 subsets of one size."""
    for ww in dict.fromkeys((w, big)):
        for part in torch.nonzero(size == ww)[:, 0].split(4096):
            if len(part):
                yield part, ww


def _exact_icgn(fn, gn, gx, gy, xy, U0, w, tol):
    n = len(xy)
    size, big = _windows(fn, gx, xy, w)
    half = size == 102
    U, F = torch.full((n, 2), math.nan, dtype=F64, device=DEV), torch.full((n, 4), math.nan, dtype=F64, device=DEV)
    iters, H21 = torch.full((n,), -1, dtype=torch.int64, device=DEV), torch.zeros((n, 21), dtype=F64, device=DEV)
    U[half], F[half], iters[half] = U0[half], 0.0, 102
    rows, cols = np.array([(r, q) for q in range(6) for r in range(q, 6)]).T
    for sl, w in _chunks(size, big, w):
        f, fx, fy, X, Y = _subsets(fn, gx, gy, xy[sl], w)
        fbar = f - f.mean(1, keepdim=True)
        bf = fbar.norm(dim=1, keepdim=True)
        sd = torch.stack([X * fx, X * fy, Y * fx, Y * fy, fx, fy], 2)
        H = sd.transpose(1, 2) @ sd
        P = torch.zeros((len(f), 6), dtype=F64, device=DEV)
        P[:, 4:] = U0[sl]

        def step(live, it, its, first):
            r, out = _residual(gn, P[live], xy[sl][live], X[live], Y[live], fbar[live], bf[live])
            b = bf[live] * (sd[live].transpose(1, 2) @ r[:, :, None])[:, :, 0]
            go = _stopped(live, it, its, first, b.norm(dim=1), out, tol)
            at = live[go]
            P[at] = _composed(P[at], -torch.linalg.solve(H[at], b[go]))
            return at
        iters[sl] = _iterate(len(f), step)
        U[sl], F[sl], H21[sl] = P[:, 4:], P[:, :4], H[:, rows, cols]
    return {"U": U, "F": F, "iters": iters, "H21": H21}


def _exact_subpb1(fn, gn, gx, gy, xy, U2, F2, vd, H21, w, mu, tol):
    n = len(xy)
    size, big = _windows(fn, gx, xy, w)
    U = torch.full((n, 2), math.nan, dtype=F64, device=DEV)
    iters = torch.full((n,), -1, dtype=torch.int64, device=DEV)
    U[size == 102], iters[size == 102] = U2[size == 102], 102
    for sl, w in _chunks(size, big, w):
        f, fx, fy, X, Y = _subsets(fn, gx, gy, xy[sl], w)
        fbar = f - f.mean(1, keepdim=True)
        bf = fbar.norm(dim=1, keepdim=True)
        s2 = 2.0 / (bf * bf)[:, 0]
        A = torch.zeros((len(f), 2, 2), dtype=F64, device=DEV)
        A[:, 0, 0], A[:, 1, 1] = H21[sl, 18] * s2 + mu, H21[sl, 20] * s2 + mu
        A[:, 0, 1] = A[:, 1, 0] = H21[sl, 19] * s2
        A += 1e-3 * A.diagonal(dim1=1, dim2=2).amax(1)[:, None, None] * torch.eye(2, dtype=F64, device=DEV)
        P = torch.cat([F2[sl], U2[sl]], 1)

        def step(live, it, its, first):
            r, out = _residual(gn, P[live], xy[sl][live], X[live], Y[live], fbar[live], bf[live])
            img = torch.stack([(fx[live] * r).sum(1), (fy[live] * r).sum(1)], 1) * (bf[live] * s2[live, None])
            t = img + mu * (P[live, 4:] - U2[sl][live] - vd[sl][live])
            go = _stopped(live, it, its, first, t.norm(dim=1), out, tol)
            at = live[go]
            d = torch.zeros((len(at), 6), dtype=F64, device=DEV)
            d[:, 4:] = -torch.linalg.solve(A[at], t[go])
            P[at] = _composed(P[at], d)
            return at
        iters[sl] = _iterate(len(f), step)
        U[sl] = P[:, 4:]
    return U, iters


def _cg(apply, b, x):
    r = b - apply(x)
    p, rr = r.clone(), (r * r).sum((-2, -1), keepdim=True)
    stop = 1e-30 * (b * b).sum((-2, -1), keepdim=True)
    for it in range(20000):
        if it % 16 == 0 and bool((rr <= stop).all()):
            break
        q = apply(p)
        d = (p * q).sum((-2, -1), keepdim=True)
        a = torch.where(d > 0, rr / d.clamp_min(1e-300), torch.zeros_like(d))
        x, r = x + a * p, r - a * q
        new = (r * r).sum((-2, -1), keepdim=True)
        p = r + torch.where(rr > 0, new / rr.clamp_min(1e-300), torch.zeros_like(rr)) * p
        rr = new
    return x


def _laplacian(z, diagonals):
    """Springs between neighbours of a grid (..., N, M): axial, and the diagonals at half weight."""
    out = torch.zeros_like(z)

    def link(a, b, w):
        d = w * (a[0] - b[0])
        a[1].add_(d)
        b[1].sub_(d)
    v = lambda j, i: (z[..., j, i], out[..., j, i])     # noqa: E731
    lo, hi, al = slice(None, -1), slice(1, None), slice(None)
    link(v(al, lo), v(al, hi), 1.0)
    link(v(lo, al), v(hi, al), 1.0)
    if diagonals:
        link(v(lo, lo), v(hi, hi), 0.5)
        link(v(lo, hi), v(hi, lo), 0.5)
    return out


def _springs_fit(z):
    """gridfit 'springs' of data on the nodes (NaN: none), (k, N, M)."""
    known = ~torch.isnan(z)
    d = torch.where(known, z, torch.zeros_like(z))
    N, M = z.shape[1:]
    i, j = torch.arange(M, device=DEV), torch.arange(N, device=DEV)
    nx = (i > 0).to(F64) + (i < M - 1).to(F64)
    ny = (j > 0).to(F64) + (j < N - 1).to(F64)
    scale = 1.0 / float((nx[None, :] + ny[:, None] + ny[:, None] * nx[None, :] / math.sqrt(2.0)).max()) ** 2
    return _cg(lambda x: known * x + scale * _laplacian(x, True), d, d.clone())


def _filled(z):
    """inpaint_nans method 4 of (k, N, M)."""
    unk = torch.isnan(z)
    if not bool(unk.any()):
        return z
    d = torch.where(unk, torch.zeros_like(z), z)
    b = -(_laplacian(d, False)) * unk
    return d + _cg(lambda x: unk * _laplacian(x, False), b, torch.zeros_like(z))


def _smoothed(M, N, vals, nf):
    k = torch.tensor([math.exp(-2.0), 1.0, math.exp(-2.0)], dtype=F64, device=DEV)
    k = (k[:, None] * k[None, :])
    k = (k / k.sum())[None, None]
    z = vals.reshape(N, M, nf).permute(2, 0, 1).contiguous()
    wgt = torch.nn.functional.conv2d(torch.ones((1, 1, N, M), dtype=F64, device=DEV), k, padding=1)
    for _ in range(2):
        z = torch.nn.functional.conv2d(_springs_fit(z)[:, None], k, padding=1)[:, 0] / wgt[0]
    return z.permute(1, 2, 0).reshape(-1).contiguous()


def _lines(n, h):
    """1-D linear elements: stiffness, mass, integral of N', integral of N."""
    K, Mm = torch.zeros((n, n), dtype=F64, device=DEV), torch.zeros((n, n), dtype=F64, device=DEV)
    e = torch.arange(n - 1, device=DEV)
    for a, b, kk, mm in ((0, 0, 1, 2), (1, 1, 1, 2), (0, 1, -1, 1), (1, 0, -1, 1)):
        K.index_put_((e + a, e + b), torch.tensor(kk / h, dtype=F64, device=DEV), accumulate=True)
        Mm.index_put_((e + a, e + b), torch.tensor(mm * h / 6, dtype=F64, device=DEV), accumulate=True)
    d, m = torch.zeros(n, dtype=F64, device=DEV), torch.full((n,), h, dtype=F64, device=DEV)
    d[0], d[-1], m[0], m[-1] = -1, 1, h / 2, h / 2
    L = torch.linalg.cholesky(Mm)
    Li = torch.linalg.inv(L)
    lam, V = torch.linalg.eigh(Li @ K @ Li.T)
    return Mm, d, m, lam, Li.T @ V


def _fe_solve(M, N, h, beta, mu, U, F, ud, vd):
    """Subpb2 on the uniform Q4 mesh by separation of variables."""
    Mx, dx, mx, lx, Vx = _lines(M, float(h))
    My, dy, my, ly, Vy = _lines(N, float(h))
    FW = (F - ud).view(N, M, 4).permute(2, 0, 1)
    D = (U - vd).view(N, M, 2).permute(2, 0, 1)
    gxw, gyw = my[:, None] * dx[None, :], dy[:, None] * mx[None, :]
    b = torch.stack([beta * (FW[0] * gxw + FW[2] * gyw), beta * (FW[1] * gxw + FW[3] * gyw)]) + mu * (My @ D @ Mx)
    C = (Vy.T @ b @ Vx) / (beta * (ly[:, None] + lx[None, :]) + mu)
    return (Vy @ C @ Vx.T).permute(1, 2, 0).reshape(-1).contiguous()


def _nodal_strain(M, N, h, U):
    z = U.view(N, M, 2)

    def d(dim):
        n = z.shape[dim]
        e = (z.narrow(dim, 1, n - 1) - z.narrow(dim, 0, n - 1)) / h
        out = torch.zeros_like(z)
        out.narrow(dim, 0, n - 1).add_(e)
        out.narrow(dim, 1, n - 1).add_(e)
        out.narrow(dim, 1, n - 2).mul_(0.5)
        return out
    gx, gy = d(1), d(0)
    return torch.stack([gx[..., 0], gy[..., 0], gx[..., 1], gy[..., 1]], 2).reshape(-1)


def _exact_frame(c, seed):
    f, g, field = _pair(c, seed)
    M, N = _nodes(c)
    n, w, h, mu, tol = M * N, c["subset"], float(c["step"]), 1e-3, c["tol"]
    xy = _grid(c)
    if c["init"] == "given":
        U0 = _guess(c, seed, field).view(-1, 2)
    else:
        r = _exact_search(c, f, g, False)
        U0 = _filled(torch.stack([r["u"], r["v"]])).reshape(2, -1).T.contiguous()
    fn, gn = _normalised(f), _normalised(g)
    gx, gy = _gradient(fn)
    r = _exact_icgn(fn, gn, gx, gy, xy, U0, w, tol)
    it = r["iters"]
    good = (it >= 0) & (it <= 99)
    t = it[good].to(F64)
    bad = ~good | (it.to(F64) > t.mean() + 0.15 * t.std())
    z = torch.cat([r["U"], r["F"]], 1).masked_fill(bad[:, None], math.nan).T.reshape(6, N, M)
    z = _filled(z).reshape(6, -1)
    U1, F1 = z[:2].T.reshape(-1).contiguous(), z[2:].T.reshape(-1).contiguous()
    smooth = (lambda a, k: _smoothed(M, N, a, k)) if c["smooth"] else (lambda a, k: a)
    F1 = smooth(F1, 4)
    ud, vd = torch.zeros_like(F1), torch.zeros_like(U1)
    bs = np.array([1e-3, math.sqrt(1e-5), 1e-2, math.sqrt(1e-3), 1e-1, math.sqrt(1e-1)]) * h * h * mu
    err = []
    for beta in bs:
        U2 = _fe_solve(M, N, h, beta, mu, U1, F1, ud, vd)
        err.append((float((U1 - U2).norm()), float((F1 - _nodal_strain(M, N, h, U2)).norm())))
    e = np.array(err)
    es = ((e - e.mean(0)) / e.std(0, ddof=1)).sum(1)
    k = int(es.argmin())
    beta = bs[k]
    if 1 <= k <= 4:
        p = np.polyfit(np.log10(bs[k - 1:k + 2]), es[k - 1:k + 2], 2)
        beta = 10 ** (-p[1] / 2 / p[0])
    U2 = _fe_solve(M, N, h, beta, mu, U1, F1, ud, vd)
    F2 = smooth(_nodal_strain(M, N, h, U2), 4)
    ud, vd = F2 - F1, U2 - U1
    for _ in range(c["admm"]):
        u, its = _exact_subpb1(fn, gn, gx, gy, xy, U2.view(-1, 2), F2.view(-1, 4), vd.view(-1, 2), r["H21"], w, mu, tol)
        z = u.masked_fill(((its > 99) | (its < 0))[:, None], math.nan).T.reshape(2, N, M)
        U1, F1 = smooth(_springs_fit(z).reshape(2, -1).T.reshape(-1).contiguous(), 2), F2
        U2 = smooth(_fe_solve(M, N, h, beta, mu, U1, F1, ud, vd), 2)
        F2 = smooth(_nodal_strain(M, N, h, U2), 4)
        ud, vd = F2 - F1, U2 - U1
    return {"x0": xy[:, 0], "y0": xy[:, 1], "U": U2, "F": F2, "iters": None}
