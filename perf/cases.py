"""Performance cases of the cone-beam operators and reconstruction loops.

Each case is one pass through the public entry points, as a program that reconstructs calls
them: ``Context.project`` / ``backproject`` / ``fdk`` on a context with its defaults,
``Solver.iterate`` (the large one with the autotuner's choice, as the benchmark runs it) and
``Batch.iterate`` over uneven jobs. Inputs are seeded random ellipsoids and their cone-beam
line integrals (closed form) with 1% noise. ``exact`` restates every path in 64 bits.
"""
from __future__ import annotations

import math
import random

import numpy as np
import torch
import torch.nn.functional as F

import tomogpi_b200 as t
from tomogpi_b200 import autotune

DEV = "cuda:0"
DTYPES = {"f32": torch.float32, "bf16": torch.bfloat16, "f16": torch.float16}
LAMBDA = 0.01
MANY = 1 << 20  # iteration budget of a batch that is driven one pass after another


def _geo(n, nz, nu, nv, views, pitch, mag):
    return {"n": n, "nz": nz, "nu": nu, "nv": nv, "views": views, "pitch": pitch, "mag": mag}


def listed():
    return [
        # the smallest jobs of an uneven mix: a call's fixed costs and launches count
        dict(name="rs_f32_64", op="project", kind="RS", dtype="f32", **_geo(64, 64, 64, 64, 60, 2.0, 2.0)),
        dict(name="vi_f32_64", op="backproject", kind="VI", dtype="f32", **_geo(64, 64, 64, 64, 60, 2.0, 2.0)),
        # the plain 256^3 workload: project once, backproject once
        dict(name="rs_f32_256", op="project", kind="RS", dtype="f32", **_geo(256, 256, 256, 256, 256, 2.0, 2.0)),
        dict(name="vi_f32_256", op="backproject", kind="VI", dtype="f32", **_geo(256, 256, 256, 256, 256, 2.0, 2.0)),
        # a real scan's sizes: odd volume and detector, another magnification and pixel pitch
        dict(name="rs_f32_ragged", op="project", kind="RS", dtype="f32", **_geo(211, 173, 301, 259, 181, 1.4, 1.7)),
        dict(name="vi_f32_ragged", op="backproject", kind="VI", dtype="f32", **_geo(211, 173, 301, 259, 181, 1.4, 1.7)),
        # mixed precision: 16-bit storage of volume and sinogram, FP32 sums
        dict(name="rs_bf16_384", op="project", kind="RS", dtype="bf16", **_geo(384, 384, 384, 384, 360, 2.0, 2.0)),
        # the SIDDONVI pair's projector
        dict(name="siddon_f32_192", op="project", kind="SIDDON", dtype="f32", **_geo(192, 192, 192, 192, 128, 2.0, 2.0)),
        # filtered backprojection: ramp filter and weighted backprojection
        dict(name="fdk_f32_256", op="fdk", kind="FDK", dtype="f32", **_geo(256, 256, 256, 256, 256, 2.0, 2.0)),
        # the iterative benchmark: one gradient iteration at 512^3, autotuned
        dict(name="solve_f32_512", op="solve", dtype="f32", iters=1, tuned=True, reg="gg",
             **_geo(512, 512, 512, 512, 512, 2.0, 2.0)),
        # a small reconstruction, 16-bit operators on FP32 data, five iterations
        dict(name="solve_bf16_128", op="solve", dtype="bf16", iters=5, tuned=False, reg="gg",
             **_geo(128, 128, 128, 128, 128, 2.0, 2.0)),
        # uneven jobs advanced together, 16-bit operators on FP32 data, two iterations
        dict(name="batch_bf16_8", op="batch", dtype="bf16", iters=2, jobs=8, mix=3, lo=64, hi=192),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng: random.Random):
    """A case of the same ranges: 48..288 voxels a side, 40..300 views, odd sizes, pitches and
    magnifications of the job mixes, every storage type and operator variant in use."""
    what = rng.choice(["project", "project", "project", "backproject", "backproject", "fdk", "solve", "batch"])
    dtype = rng.choice(["f32", "f32", "bf16", "f16"])
    if what == "batch":
        return dict(op="batch", dtype=rng.choice(["bf16", "f32"]), iters=1, jobs=rng.randint(3, 9),
                    mix=rng.randrange(1 << 20), lo=48, hi=rng.randint(100, 192))
    n = _log(rng, 48, 288)
    nz = n if rng.random() < 0.5 else max(17, int(n * rng.uniform(0.4, 1.2)))
    nu = n if rng.random() < 0.4 else int(n * rng.uniform(0.8, 1.5))
    nv = nu if rng.random() < 0.5 else max(17, int(nz * rng.uniform(0.8, 1.5)))
    mag = round(rng.uniform(1.5, 2.5), 3)
    pitch = round(mag * rng.uniform(0.8, 1.1) * n / nu, 3)
    g = _geo(n, nz, nu, nv, _log(rng, 40, 300), pitch, mag)
    if what == "project":
        kind = rng.choice(["RS", "RS", "RS", "RS_UM", "SIDDON"])
        return dict(op="project", kind=kind, dtype="f32" if kind == "SIDDON" else dtype, **g)
    if what == "backproject":
        return dict(op="backproject", kind=rng.choice(["VI", "VI", "VI_UM"]), dtype=dtype, **g)
    if what == "fdk":
        return dict(op="fdk", kind="FDK", dtype="f32", **g)
    return dict(op="solve", dtype=dtype, iters=rng.randint(1, 3), tuned=False, reg=rng.choice(["gg", "huber"]), **g)


def _cfg(c):
    n, fod = c["n"], 2.0 * c["n"]
    return t.ConfigCT(fod=fod, fdd=c["mag"] * fod, projection_nb=c["views"],
                      u_detector_size=c["pitch"] * c["nu"], v_detector_size=c["pitch"] * c["nv"],
                      u_detector_pixel_nb=c["nu"], v_detector_pixel_nb=c["nv"],
                      x_volume_size=float(n), y_volume_size=float(n), z_volume_size=float(c["nz"]),
                      x_volume_pixel_nb=n, y_volume_pixel_nb=n, z_volume_pixel_nb=c["nz"])


def _jobs(c):
    """The jobs of a batch case: N a multiple of 16 or odd, views U[60, 200], magnification
    U[1.5, 2.5], an N x N detector of pitch 2."""
    rng = random.Random(c["mix"])
    out = []
    for j in range(c["jobs"]):
        n = c["hi"] if j == 0 else _log(rng, c["lo"], c["hi"])
        n = n if rng.random() < 0.3 else max(48, n // 16 * 16)
        out.append(_geo(n, n, n, n, rng.randint(60, 200), 2.0, round(rng.uniform(1.5, 2.5), 3)))
    return out


# --- inputs -------------------------------------------------------------------------------
def _ellipsoids(seed, g):
    """Eight axis-aligned ellipsoids inside the field of view: (value, semi-axes, centre), in
    voxels from the volume's centre."""
    r = np.random.default_rng(seed)
    out = []
    for _ in range(8):
        rad, ang = 0.3 * g["n"] * math.sqrt(r.uniform()), r.uniform(0, 2 * math.pi)
        ax = r.uniform(0.05, 0.2, 3) * np.array([g["n"], g["n"], g["nz"]])
        out.append((float(r.uniform(0.1, 1.0)), ax, np.array([rad * math.cos(ang), rad * math.sin(ang),
                                                              r.uniform(-0.3, 0.3) * g["nz"]])))
    return out


def _volume(seed, g):
    x = torch.arange(g["n"], device=DEV, dtype=torch.float32) - (g["n"] / 2 - 0.5)
    z = torch.arange(g["nz"], device=DEV, dtype=torch.float32) - (g["nz"] / 2 - 0.5)
    v = torch.zeros(g["nz"], g["n"], g["n"], device=DEV)
    for val, ax, c in _ellipsoids(seed, g):
        q = (((z - c[2]) / ax[2]) ** 2)[:, None, None] + (((x - c[1]) / ax[1]) ** 2)[None, :, None] \
            + (((x - c[0]) / ax[0]) ** 2)[None, None, :]
        v += val * (q <= 1.0)
    return v


def _sinogram(seed, g):
    """Line integrals of the ellipsoids over the rays of the scan, plus 1% noise."""
    fod, fdd = 2.0 * g["n"], 2.0 * g["n"] * g["mag"]
    u = (torch.arange(g["nu"], device=DEV, dtype=torch.float32) - (g["nu"] / 2 - 0.5)) * g["pitch"]
    v = (torch.arange(g["nv"], device=DEV, dtype=torch.float32) - (g["nv"] / 2 - 0.5)) * g["pitch"]
    out = torch.zeros(g["views"], g["nv"], g["nu"], device=DEV)
    ells = _ellipsoids(seed, g)
    for p in range(g["views"]):
        phi = p * 2.0 * math.pi / g["views"]
        ca, sa = math.cos(phi), math.sin(phi)
        dx, dy, dz = fdd * ca - u * sa, fdd * sa + u * ca, v[:, None]
        length = torch.sqrt((dx * dx + dy * dy)[None, :] + dz * dz)
        for val, ax, c in ells:
            ox, oy, oz = -fod * ca - float(c[0]), -fod * sa - float(c[1]), -float(c[2])
            a = ((dx / ax[0]) ** 2 + (dy / ax[1]) ** 2)[None, :] + (dz / ax[2]) ** 2
            b = (ox * dx / ax[0] ** 2 + oy * dy / ax[1] ** 2)[None, :] + oz * dz / ax[2] ** 2
            k = (ox / ax[0]) ** 2 + (oy / ax[1]) ** 2 + (oz / ax[2]) ** 2 - 1.0
            out[p] += val * 2.0 * torch.sqrt(torch.clamp(b * b - a * k, min=0.0)) / a * length
    gen = torch.Generator(device=DEV).manual_seed(int(seed))
    for p in range(g["views"]):
        out[p] += torch.randn(out[p].shape, device=DEV, generator=gen) * (0.01 * 0.5 * g["n"])
    return out


def prepare(case, seed):
    c = case
    if c["op"] == "batch":
        params = t.GradientParams(gradient_iteration_nb=MANY, optimal_step_iteration_nb=MANY + 1,
                                  regularization_parameter=LAMBDA, storage=c["dtype"], real_f32=True)
        b = t.Batch(params)
        vols = []
        for k, g in enumerate(_jobs(c)):
            vol = torch.zeros(g["nz"], g["n"], g["n"], device=DEV)
            b.add(_cfg(g), vol, _sinogram(seed * 131 + k, g))
            vols.append(vol)
        return {"case": c, "batch": b, "vols": vols}
    ctx = t.Context(_cfg(c))
    s = {"case": c, "ctx": ctx}
    if c["op"] == "project":
        s["in"] = _volume(seed, c).to(DTYPES[c["dtype"]])
    elif c["op"] in ("backproject", "fdk"):
        s["in"] = _sinogram(seed, c).to(DTYPES[c["dtype"]])
    else:
        if c["tuned"]:
            r = autotune.tune(ctx.cfg, c["dtype"])
            ctx.set_tuning(rs_layout=r["rs_layout"], vi_zc=r["vi_zc"], vi_layout=r["vi_layout"])
        s["in"] = _sinogram(seed, c)
        s["vol"] = torch.zeros(c["nz"], c["n"], c["n"], device=DEV)
        s["solver"] = t.Solver(ctx, t.GradientParams(
            gradient_iteration_nb=c["iters"], optimal_step_iteration_nb=c["iters"] + 1,
            regularization_parameter=LAMBDA, storage=c["dtype"], real_f32=True))
        if c["reg"] == "huber":
            s["solver"].set_regularizer("huber", huber_threshold=0.02)
    return s


def run(state):
    c = state["case"]
    if c["op"] == "project":
        return state["ctx"].project(c["kind"], state["in"])
    if c["op"] == "backproject":
        return state["ctx"].backproject(c["kind"], state["in"])
    if c["op"] == "fdk":
        return state["ctx"].fdk(state["in"])
    if c["op"] == "solve":
        state["vol"].zero_()
        return state["solver"].iterate(state["vol"], state["in"], first=1, count=c["iters"])
    for v in state["vols"]:
        v.zero_()
    state["batch"].iterate(c["iters"])
    return list(state["vols"])


# --- what a pass cannot do without ----------------------------------------------------------
def _samples(g):
    """Unit steps along the rays inside the volume's box, over all rays (from every fourth
    ray of 16 views)."""
    n, nz, fod = g["n"], g["nz"], 2.0 * g["n"]
    fdd = fod * g["mag"]
    u = (np.arange(0, g["nu"], 4) - (g["nu"] / 2 - 0.5)) * g["pitch"]
    v = ((np.arange(0, g["nv"], 4) - (g["nv"] / 2 - 0.5)) * g["pitch"])[:, None]
    tot = 0.0
    for p in range(16):
        phi = 2 * math.pi * p / 16 + 0.01
        ca, sa = math.cos(phi), math.sin(phi)
        d = np.stack(np.broadcast_arrays(fdd * ca - u * sa, fdd * sa + u * ca, v))
        d = d / np.sqrt((d * d).sum(0))
        o, half = np.array([-fod * ca, -fod * sa, 0.0]), np.array([n, n, nz]) / 2.0
        lo, hi = np.full(d[0].shape, -1e30), np.full(d[0].shape, 1e30)
        for k in range(3):
            with np.errstate(divide="ignore"):
                a, b = (-half[k] - o[k]) / d[k], (half[k] - o[k]) / d[k]
            lo, hi = np.maximum(lo, np.minimum(a, b)), np.minimum(hi, np.maximum(a, b))
        tot += np.maximum(hi - lo, 0.0).mean()
    return tot / 16 * g["nu"] * g["nv"] * g["views"]


def work(case):
    """Bytes: inputs read once, outputs written once. Operations: 16 per trilinear sample and
    8 per bilinear voxel update (interpolate and add), 4 per Siddon voxel visit."""
    c = case
    if c["op"] == "batch":
        by = fl = 0.0
        for g in _jobs(c):
            w = work(dict(op="solve", dtype=c["dtype"], iters=c["iters"], **g))
            by, fl = by + w["bytes"], fl + w["flops"]
        return {"bytes": by, "flops": fl}
    es = 4 if c["dtype"] == "f32" else 2
    vox, pix = c["n"] ** 2 * c["nz"], c["nu"] * c["nv"] * c["views"]
    if c["op"] == "project":
        return {"bytes": es * (vox + pix), "flops": (4 * 1.6 if c["kind"] == "SIDDON" else 16) * _samples(c)}
    if c["op"] == "backproject":
        return {"bytes": es * (vox + pix), "flops": 8.0 * vox * c["views"]}
    if c["op"] == "fdk":
        return {"bytes": 4.0 * (vox + pix), "flops": 14.0 * vox * c["views"] + 10.0 * pix * math.log2(2 * c["nu"])}
    return {"bytes": c["iters"] * 4.0 * (2 * vox + pix),
            "flops": c["iters"] * (32.0 * _samples(c) + 8.0 * vox * c["views"] + 40.0 * vox)}


def tolerance(case):
    """FP32 sums in another order: 1e-5. 16-bit results may round to the neighbouring value;
    a loop with 16-bit operators carries such roundings of the iterate through its
    projections."""
    c = case
    if c["op"] in ("solve", "batch"):
        return {"rel": 2e-5 if c["dtype"] == "f32" else 1e-3, "max": 2e-3 if c["dtype"] == "f32" else 0.1}
    return {"f32": {"rel": 1e-5, "max": 1e-3}, "bf16": {"rel": 2e-3, "max": 0.02},
            "f16": {"rel": 3e-4, "max": 3e-3}}[c["dtype"]]


# --- the same in 64 bits ---------------------------------------------------------------------
D = torch.float64


class _Geom:
    def __init__(self, g):
        self.n, self.nz, self.nu, self.nv, self.np = g["n"], g["nz"], g["nu"], g["nv"], g["views"]
        self.fod = 2.0 * g["n"]
        self.fdd = self.fod * g["mag"]
        self.du = g["pitch"]
        self.uc, self.vc = g["nu"] / 2 - 0.5, g["nv"] / 2 - 0.5
        self.xc, self.zc = g["n"] / 2 - 0.5, g["nz"] / 2 - 0.5
        self.phi = [p * 2.0 * math.pi / g["views"] for p in range(g["views"])]


def _f(x):
    return torch.as_tensor(x, dtype=D, device=DEV)


def _rs_rays(q, phi, um):
    """Entry points, unit steps and sample counts of a view's rays (the box-clipped form, or
    the cylinder form with um)."""
    al, be = math.cos(phi), math.sin(phi)
    uu = (torch.arange(q.nu, device=DEV, dtype=D) - q.uc)[None, :].expand(q.nv, q.nu)
    vv = (torch.arange(q.nv, device=DEV, dtype=D) - q.vc)[:, None].expand(q.nv, q.nu)
    ax = q.fdd * al - uu * be * q.du
    by = q.fdd * be + uu * al * q.du
    c = vv * q.du
    inv = 1.0 / torch.sqrt(ax * ax + by * by + c * c)
    sx, sy, sz = ax * inv, by * inv, c * inv
    a1 = by / ax
    b1 = -q.fod * be - a1 * (-q.fod * al)
    c1 = c / ax
    d1 = -c1 * (-q.fod * al)
    f = q.n * q.n / 2.0 * (a1 * a1 + 1.0) - b1 * b1 if not um else q.n * q.n / 4.0 * (a1 * a1 + 1.0) - b1 * b1
    hit = f >= 0
    e = torch.sqrt(torch.clamp(f, min=0.0))
    den = 1.0 + a1 * a1
    x1, x2 = (-a1 * b1 + e) / den, (-a1 * b1 - e) / den
    pt = lambda x: (x, a1 * x + b1, c1 * x + d1)  # noqa: E731
    p1, p2 = pt(x1), pt(x2)
    dist = lambda p: (p[0] + q.fod * al) ** 2 + (p[1] + q.fod * be) ** 2 + p[2] ** 2  # noqa: E731
    first = dist(p1) <= dist(p2)
    P = [torch.where(first, a, b) for a, b in zip(p1, p2)]
    E = [torch.where(first, b, a) for a, b in zip(p1, p2)]
    hi = q.xc  # the box [-xc, xc] about the centre
    if not um:
        for pts in (P, E):
            for lim in (-hi, hi):
                for k in (0, 1):
                    out = pts[k] < lim if lim < 0 else pts[k] > lim
                    x = torch.full_like(a1, lim) if k == 0 else (lim - b1) / a1
                    new = (x, a1 * x + b1 if k == 0 else torch.full_like(a1, lim), c1 * x + d1)
                    for m in range(3):
                        pts[m] = torch.where(out, new[m], pts[m])
    top = q.nz - q.zc if um else q.nz - 1 - q.zc
    hit &= (P[2] >= -q.zc) & ((P[2] < top) if um else (P[2] <= top))
    for lim in (-q.zc, q.nz - 1 - q.zc):
        out = E[2] < lim if lim < 0 else E[2] > lim
        x = (lim - d1) / c1
        new = (x, a1 * x + b1, torch.full_like(a1, lim))
        for m in range(3):
            E[m] = torch.where(out, new[m], E[m])
    length = torch.sqrt(sum((a - b) ** 2 for a, b in zip(P, E)))
    cnt = torch.where(hit, torch.floor(length), torch.zeros_like(length))
    return (P[0] + q.xc, P[1] + q.xc, P[2] + q.zc), (sx, sy, sz), cnt


def _rs(q, vol, um=False):
    v5 = vol.to(D)[None, None]
    out = torch.zeros(q.np, q.nv, q.nu, device=DEV, dtype=D)
    dims = (q.n, q.n, q.nz)
    step = max(1, 24_000_000 // (q.nu * q.nv))
    for p in range(q.np):
        P, S, cnt = _rs_rays(q, q.phi[p], um)
        most = int(cnt.max())
        for k in range(0, most, step):
            m = torch.arange(k, min(k + step, most), device=DEV, dtype=D)[:, None, None]
            grid = torch.stack([(P[i] + m * S[i]) * (2.0 / max(dims[i] - 1, 1)) - 1.0 for i in range(3)], -1)
            val = F.grid_sample(v5, grid[None], mode="bilinear", padding_mode="zeros", align_corners=True)[0, 0]
            out[p] += (val * (m < cnt)).sum(0)
    return out


def _vi(q, sino, weight=None):
    s = sino.to(D)
    x = torch.arange(q.n, device=DEV, dtype=D) - q.xc
    z = (torch.arange(q.nz, device=DEV, dtype=D) - q.zc)[:, None, None]
    out = torch.zeros(q.nz, q.n, q.n, device=DEV, dtype=D)
    zs = max(1, 32_000_000 // (q.n * q.n))
    for p in range(q.np):
        al, be = math.cos(q.phi[p]), math.sin(q.phi[p])
        w = al * x[None, :] + be * x[:, None] + q.fod
        u = (-be * x[None, :] + al * x[:, None]) * (q.fdd / q.du) / w
        a = q.fdd / q.du / w
        for k in range(0, q.nz, zs):
            v = a * z[k:k + zs]
            grid = torch.stack([((u + q.uc) * (2.0 / max(q.nu - 1, 1)) - 1.0).expand_as(v),
                                (v + q.vc) * (2.0 / max(q.nv - 1, 1)) - 1.0], -1).reshape(1, -1, q.n * q.n, 2)
            val = F.grid_sample(s[p][None, None], grid, mode="bilinear", padding_mode="zeros", align_corners=True)
            val = val.reshape(v.shape)
            out[k:k + zs] += val if weight is None else val * weight(w, u, v)
    return out


def _fdk(q, sino):
    nu, over = q.nu, 16
    M = over * nu
    nr = M - (M % 2)
    win = np.zeros(M)
    win[(M - nr) // 2:(M - nr) // 2 + nr] = 0.5 * (1.0 - np.cos(2.0 * np.pi * np.arange(nr) / (nr - 1)))
    k = np.arange(M)
    taps = np.fft.ifft(np.where(k <= M // 2, k, M - k) / (M // 2) * win[(k + M // 2) % M]).real / (2.0 * q.du)
    half, lo = math.floor(nu / 2 + 0.5), math.floor(3 * nu / 2 + 0.5) - 2 * nu
    lags = np.arange(max(-half, lo), half)
    L = 4 * nu
    h = np.zeros(L)
    h[lags % L] = taps[lags % M]
    f = torch.fft.irfft(torch.fft.rfft(sino.to(D), n=L) * torch.fft.rfft(_f(h)), n=L)[..., :nu]
    ac, bc = math.pi * q.fod * q.fdd / q.np, (q.fdd / q.du) ** 2
    return _vi(q, f, lambda w, u, v: ac * (q.fdd / q.du) / (w * w) / torch.sqrt(bc + u * u + v * v))


def _siddon(q, vol):
    """The exact-chord traversal: nearest crossing first, entry at the inscribed cylinder."""
    out = torch.zeros(q.np, q.nv, q.nu, device=DEV, dtype=D)
    flat = vol.to(D).reshape(-1)
    dims = (q.n, q.n, q.nz)
    s = ((torch.arange(q.nu, device=DEV, dtype=D) - q.uc) * q.du)[None, :].expand(q.nv, q.nu)
    tt = ((torch.arange(q.nv, device=DEV, dtype=D) - q.vc) * q.du)[:, None].expand(q.nv, q.nu)
    for p0 in range(0, q.np, 16):
        phi = _f(q.phi[p0:p0 + 16])[:, None, None]
        al, be = torch.cos(phi), torch.sin(phi)
        zero = torch.zeros_like(al * s)
        src = [q.xc - q.fod * al + zero, q.xc - q.fod * be + zero, q.zc + zero]
        det = [q.xc + al * (q.fdd - q.fod) - s * be, q.xc + be * (q.fdd - q.fod) + s * al, q.zc + tt + zero]
        L = torch.sqrt(q.fdd ** 2 + s * s + tt * tt) + zero
        A, B = (q.fdd ** 2 + s * s) / (L * L), -q.fod * q.fdd / L
        delta = B * B - A * (q.fod ** 2 - 0.25 * q.n * q.n)
        live = delta > 0
        sq = torch.sqrt(torch.clamp(delta, min=0.0))
        lam, lmax = (-B - sq) / A, (-B + sq) / A
        idx, cross, step, sign = [], [], [], []
        for k in range(3):
            d = det[k] - src[k]
            fwd = d >= 0
            pos = src[k] + lam * d / L
            i = torch.where(fwd, torch.floor(pos - 0.5), torch.ceil(pos + 0.5)).clamp(0, dims[k] - 1)
            c = L * (i + torch.where(fwd, 0.5, -0.5) - src[k]) / d
            idx.append(i.long())
            cross.append(torch.where(d.abs() > 1.0, c, L))
            step.append(L / d.abs())
            sign.append(torch.where(fwd, 1, -1))
        acc = zero.clone()
        while True:
            act = live & (lam <= lmax)
            if not bool(act.any()):
                break
            for _ in range(8):
                act = live & (lam <= lmax)
                lk = torch.minimum(torch.minimum(cross[0], cross[1]), cross[2])
                ok = act
                for k in range(3):
                    ok = ok & (idx[k] >= 0) & (idx[k] < dims[k])
                at = (idx[2].clamp(0, q.nz - 1) * q.n + idx[1].clamp(0, q.n - 1)) * q.n + idx[0].clamp(0, q.n - 1)
                acc += torch.where(ok, (lk - lam) * flat[at], zero)
                lam = torch.where(act, lk, lam)
                for k in range(3):
                    hit = act & (cross[k] <= lk)
                    cross[k] = torch.where(hit, cross[k] + step[k], cross[k])
                    idx[k] = torch.where(hit, idx[k] + sign[k], idx[k])
        out[p0:p0 + 16] = acc
    return out


def _lap(v):
    p = F.pad(v[None], (1, 1, 1, 1, 1, 1))[0]
    return 6.0 * v - p[1:-1, 1:-1, :-2] - p[1:-1, 1:-1, 2:] - p[1:-1, :-2, 1:-1] - p[1:-1, 2:, 1:-1] \
        - p[:-2, 1:-1, 1:-1] - p[2:, 1:-1, 1:-1]


def _gradient(q, data, iters, reg):
    f = torch.zeros(q.nz, q.n, q.n, device=DEV, dtype=D)
    thr = 0.02
    for _ in range(iters):
        dj = -2.0 * _vi(q, data.to(D) - _rs(q, f))
        lf = _lap(f)
        if reg == "gg":
            dj = dj + 2.0 * LAMBDA * _lap(lf)
            nr = 2.0 * float((_lap(dj) ** 2).sum())
        else:
            dj = dj + LAMBDA * _lap(torch.clamp(2.0 * lf, -2.0 * thr, 2.0 * thr))
            nr = float((_lap(_lap((lf.abs() <= thr) * dj)) * dj).abs().sum())
        den = 2.0 * float((_rs(q, dj) ** 2).sum()) + LAMBDA * nr
        f = f - float((dj ** 2).sum()) / den * dj
    return f


def exact(case, seed):
    c = case
    if c["op"] == "batch":
        return [_gradient(_Geom(g), _sinogram(seed * 131 + k, g), c["iters"], "gg") for k, g in enumerate(_jobs(c))]
    if c["op"] == "solve" and c["n"] ** 2 * c["nz"] * c["views"] * c["iters"] > 2.5e9:
        return None
    q = _Geom(c)
    if c["op"] == "project":
        vol = _volume(seed, c).to(DTYPES[c["dtype"]])
        return _siddon(q, vol) if c["kind"] == "SIDDON" else _rs(q, vol, c["kind"] == "RS_UM")
    if c["op"] == "solve":
        return _gradient(q, _sinogram(seed, c), c["iters"], c["reg"])
    sino = _sinogram(seed, c).to(DTYPES[c["dtype"]])
    return _fdk(q, sino) if c["op"] == "fdk" else _vi(q, sino)
