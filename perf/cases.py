"""Performance cases of the projection engine: what its users have it do on the GPU.

A time loop calls one of these once per time step, with a plan made once per grid:

  step     the projection step of the incompressible solver (divergence, Poisson solve,
           correction, boundary fill), FP64 or FP32 storage with FP64 refinement; with
           "stats" the step also returns its max|div u| record; with "rough" the predictor is
           first forced to the wall values inside a rough surface
  vd       the variable-density step
  poisson  the Poisson solve alone, in place on the right-hand side
  batch    many uneven Poisson solves in one launch

The grids are those of this repository's benchmark, tests and served mix, and ragged ones: sizes
that are products of 2, 3 and 5 as DNS grids often are, and odd sizes with larger primes.  The
host-buffer forms and the server run these same kernels behind copies and a queue.
"""
from __future__ import annotations

import importlib
import math
import random

import numpy as np
import torch

prj = importlib.import_module("dns-supercritical-ibm_b200.prj")

LX, LZ, BETA, DT, SIGMA = 2.0 * math.pi, math.pi, 2.0, 0.5, 0.1


def _grid(kind, nx, ny, nz, **options):
    return {"kind": kind, "nx": nx, "ny": ny, "nz": nz, **options}


def listed():
    return [
        # the smoke test's grid: a call that is all latency and launches
        {"name": "step 48x32x24", **_grid("step", 48, 32, 24)},
        # the reference's channel test, right-hand side given (the solver's own entry point)
        {"name": "poisson 128x96x64", **_grid("poisson", 128, 96, 64)},
        # an odd grid with primes above 5, as in the reference's randomised solver tests
        {"name": "poisson 135x60x77", **_grid("poisson", 135, 60, 77)},
        # a served request's grid, in a step that also reports its divergence
        {"name": "step+stats 256x128x128", **_grid("step", 256, 128, 128, stats=True)},
        # a production grid whose lengths are no powers of two
        {"name": "step 360x180x250", **_grid("step", 360, 180, 250)},
        # the largest of the served mix that still fits little more than L2
        {"name": "step 384x192x192", **_grid("step", 384, 192, 192)},
        # the headline channel, in both precisions
        {"name": "step 768x384x384", **_grid("step", 768, 384, 384)},
        {"name": "mixed 768x384x384", **_grid("step", 768, 384, 384, mixed=True)},
        # the mixed form on a ragged grid
        {"name": "mixed 240x120x150", **_grid("step", 240, 120, 150, mixed=True)},
        # the supercritical solver's own step
        {"name": "vd 512x256x256", **_grid("vd", 512, 256, 256)},
        # a parameter sweep: uneven independent grids in one launch
        {"name": "batch of 64", "kind": "batch", "count": 64, "sizes": 2},
        # the rough-wall run: the largest grid, its predictor forced inside the roughness
        {"name": "rough 1536x512x768", **_grid("step", 1536, 512, 768, rough=True)},
    ]


_PLANNED = (32, 48, 64, 96, 128, 192, 256, 384, 512, 768)


def _smooth(n, primes=(2, 3, 5)):
    for p in primes:
        while n % p == 0:
            n //= p
    return n == 1


def _length(rng, style, most):
    """A length of 32 .. most, spread over its logarithm."""
    while True:
        n = int(round(math.exp(rng.uniform(math.log(32), math.log(most)))))
        if style == "planned":
            return min(_PLANNED, key=lambda v: abs(math.log(v / n)))
        if style == "smooth":
            n += n % 2
            if _smooth(n):
                return n
        elif _smooth(n, (2, 3, 5, 7, 11, 13, 17, 19, 23, 29, 31)):
            return n


def draw(rng: random.Random):
    kind = rng.choices(("step", "mixed", "vd", "poisson", "batch"), (45, 10, 15, 20, 10))[0]
    if kind == "batch":
        return {"kind": "batch", "count": rng.randint(4, 64), "sizes": rng.randrange(1 << 20)}
    style = rng.choices(("planned", "smooth", "any"), (40, 40, 0 if kind == "mixed" else 20))[0]
    most = 256 if style == "any" else 800
    while True:
        nx, nz = _length(rng, style, most), _length(rng, style, most)
        ny = int(round(math.exp(rng.uniform(math.log(32), math.log(min(400, most))))))
        if nx * ny * nz <= 12e7:
            break
    options = {}
    if kind == "mixed":
        options = {"mixed": True}
    elif kind == "step" and rng.random() < 0.25:
        options = {"stats": True}
    return _grid("step" if kind == "mixed" else kind, nx, ny, nz, **options)


# ------------------------------------------------------------------ grids and inputs

def _faces(case):
    ny = case["ny"]
    if not case.get("rough"):
        j = np.arange(ny + 1, dtype=np.float64)
        return 1.0 + np.tanh(BETA * (2.0 * j / ny - 1.0)) / np.tanh(BETA)
    # uniform below y = 0.1, then 1.5% growth per cell toward the centre, mirrored
    lo, hi = 1e-9, 1.0
    for _ in range(100):
        first = 0.5 * (lo + hi)
        y, d, half = 0.0, first, [0.0]
        for _ in range(ny // 2):
            y += d
            half.append(y)
            d *= 1.015 if y >= 0.1 else 1.0
        lo, hi = (lo, first) if y > 1.0 else (first, hi)
    half = np.array(half) / half[-1]
    return np.concatenate([half, 2.0 - half[-2::-1]])


def _bands_name(case):
    # a step's divergence vanishes with the consistent bands; the reference's own bands leave a
    # divergence of order one, a value that two correct solvers agree on
    return "reference" if case["kind"] == "poisson" or case.get("stats") else "consistent"


def _batch_cases(case):
    r = random.Random(case["sizes"])
    n, m = (64, 96, 128, 192, 256), (48, 64, 96, 128)
    return [_grid("poisson", r.choice(n), r.choice(m), r.choice(n)) for _ in range(case["count"])]


def _generator(seed):
    return torch.Generator(device="cuda").manual_seed(seed)


def _rhs(case, gen):
    """Uniform noise on [-1, 1] without its volume-weighted mean."""
    yu = _faces(case)
    p = torch.rand((case["ny"], case["nz"], case["nx"]), generator=gen, device="cuda", dtype=torch.float64).mul_(2).sub_(1)
    w = torch.from_numpy(np.diff(yu)).cuda()
    p -= (p.mean(dim=(1, 2)) * w).sum() / w.sum()
    return p


def _halo(case, interior=None):
    """A halo'd field; its x and z halos periodic and its wall planes copies, when filled."""
    f = torch.zeros((case["ny"] + 2, case["nz"] + 2, case["nx"] + 2), device="cuda", dtype=torch.float64)
    if interior is not None:
        f[1:-1, 1:-1, 1:-1] = interior
        f[:, :, 0], f[:, :, -1] = f[:, :, -2].clone(), f[:, :, 1].clone()
        f[:, 0, :], f[:, -1, :] = f[:, -2, :].clone(), f[:, 1, :].clone()
        f[0], f[-1] = f[1], f[-2]
    return f


def _noise(case, gen, sigma):
    return torch.randn((case["ny"], case["nz"], case["nx"]), generator=gen, device="cuda", dtype=torch.float64).mul_(sigma)


def _predictor(case, gen):
    """Laminar profile plus normal noise; v = 0 on the bottom wall face."""
    yu = _faces(case)
    yp = torch.from_numpy((yu[1:] + yu[:-1]) / 2).cuda()
    fields = []
    for c in range(3):
        f, n = _halo(case), _noise(case, gen, SIGMA)
        if c == 0:
            n += (1.5 * (1.0 - (yp - 1.0) ** 2))[:, None, None]
        elif c == 1:
            n[0] = 0.0
        f[1:-1, 1:-1, 1:-1] = n
        fields.append(f)
    return fields


def _roughness(case, gen):
    """Column indices of a rough surface on both walls: a Gaussian random height field with
    spectrum k^-2 between 2 pi / 0.5 and 2 pi / 0.05, peak 0.08 and RMS 0.02."""
    nx, ny, nz = case["nx"], case["ny"], case["nz"]
    kx = 2 * math.pi * torch.fft.rfftfreq(nx, d=LX / nx, device="cuda", dtype=torch.float64)
    kz = 2 * math.pi * torch.fft.fftfreq(nz, d=LZ / nz, device="cuda", dtype=torch.float64)
    k = torch.hypot(kz[:, None], kx[None, :])
    amp = torch.where((k >= 2 * math.pi / 0.5) & (k <= 2 * math.pi / 0.05), 1.0 / k.clamp(min=1.0), torch.zeros_like(k))
    re, im = (torch.randn(k.shape, generator=gen, device="cuda", dtype=torch.float64) for _ in range(2))
    g = torch.fft.irfft2(torch.complex(amp * re, amp * im), s=(nz, nx))
    gap = (g.max() - g) / g.std()
    lo, hi = torch.zeros((), device="cuda", dtype=torch.float64), torch.ones((), device="cuda", dtype=torch.float64)
    for _ in range(40):  # the slope that gives the RMS height
        s = 0.5 * (lo + hi)
        low = (0.08 - s * gap).clamp(min=0.0).square().mean().sqrt() > 0.02
        lo, hi = torch.where(low, s, lo), torch.where(low, hi, s)
    h = (0.08 - lo * gap).clamp(min=0.0)
    yu = _faces(case)
    yp = torch.from_numpy((yu[1:] + yu[:-1]) / 2).cuda()
    inside = torch.searchsorted(yp, h)  # cells whose centre lies below the surface
    bot, top = (inside - 1).int().contiguous(), (ny - inside).int().contiguous()
    return {"%s_%s" % (c, w): t for c in "UVW" for w, t in (("bot", bot), ("top", top))}


def _inputs(case, seed):
    gen = _generator(seed)
    if case["kind"] == "batch":
        return {"rhs": torch.cat([_rhs(c, gen).reshape(-1) for c in _batch_cases(case)])}
    if case["kind"] == "poisson":
        return {"rhs": _rhs(case, gen)}
    d = {"hat": _predictor(case, gen)}
    if case.get("rough"):
        d["inds"] = _roughness(case, gen)
    if case["kind"] == "vd":
        # a light core between dense walls, and the pressures and divergence of earlier steps
        yu = _faces(case)
        yp = torch.from_numpy((yu[1:] + yu[:-1]) / 2).cuda()
        rho = (1.0 - 0.6 * (1.0 - (yp - 1.0) ** 2))[:, None, None] * (1.0 + _noise(case, gen, 0.05).clamp(-0.3, 0.3))
        d["fields"] = [_halo(case, rho)] + [_halo(case, _noise(case, gen, 0.01)) for _ in range(3)]
    return d


# ------------------------------------------------------------------ the measured calls

def _plan(case):
    return prj.Plan.from_yu(case["nx"], case["nz"], LX / case["nx"], LZ / case["nz"], _faces(case), _bands_name(case))


def prepare(case, seed):
    s = {"case": case, **_inputs(case, seed)}
    if case["kind"] == "batch":
        cases = _batch_cases(case)
        s["P"] = torch.empty_like(s["rhs"])
        parts = torch.split(s["P"], [c["nx"] * c["ny"] * c["nz"] for c in cases])
        s["plans"] = [_plan(c) for c in cases]
        s["batch"] = prj.Batch(s["plans"], [p.view(c["ny"], c["nz"], c["nx"]) for p, c in zip(parts, cases)])
        return s
    s["plan"] = _plan(case)
    s["P"] = torch.empty((case["ny"], case["nz"], case["nx"]), device="cuda", dtype=torch.float64)
    if case["kind"] != "poisson":
        s["out"] = [_halo(case) for _ in range(4 if case["kind"] == "vd" else 3)]
    return s


def run(s):
    case, P = s["case"], s["P"]
    if case["kind"] == "batch":
        P.copy_(s["rhs"])  # the right-hand sides, which the solve overwrites
        s["batch"].launch()
        return P
    if case["kind"] == "poisson":
        P.copy_(s["rhs"])
        return s["plan"].poisson_fp64(P)
    hat, out = s["hat"], s["out"]
    if case["kind"] == "vd":
        s["plan"].projection_step_vd(*hat, *s["fields"], *out[:3], P, out[3], DT, stats=False)
        return [*out, P]
    if case.get("rough"):
        prj.rough_force(*hat, s["inds"])
    mode = prj.MODE_FP32_REFINE if case.get("mixed") else prj.MODE_FP64
    record = s["plan"].projection_step(*hat, *out, P, DT, mode=mode, stats=bool(case.get("stats")))
    if case.get("stats"):
        return [*out, P, record["div_maxabs"], record["p_maxabs"]]
    return [*out, P, *hat] if case.get("rough") else [*out, P]


def work(case):
    if case["kind"] == "batch":
        parts = [work(c) for c in _batch_cases(case)]
        return {k: sum(w[k] for w in parts) for k in ("bytes", "flops")}
    nx, ny, nz = case["nx"], case["ny"], case["nz"]
    n, nh = nx * ny * nz, (nx + 2) * (ny + 2) * (nz + 2)
    # two transforms each way on half a spectrum, and two real Thomas sweeps per complex line
    flops = n * (5.0 * math.log2(nx * nz) + 14.0)
    if case["kind"] == "poisson":
        return {"bytes": 16 * n, "flops": flops}  # the right-hand side in, the solution out
    if case["kind"] == "vd":
        return {"bytes": 56 * n + 32 * nh + 8 * n, "flops": flops + 90.0 * n}
    # u_hat, v_hat, w_hat in; u, v, w with their halos and p out
    return {"bytes": 24 * n + 24 * nh + 8 * n, "flops": flops + 22.0 * n}


def tolerance(case):
    # about four times the largest error against exact() over the listed and drawn cases: FP64
    # transforms and sweeps reach 1.2e-13 (the corrected velocity of the variable-density step,
    # 6.6e-14 in the rough wall's pressure), one FP64 refinement of an FP32-storage solve 7.3e-14
    # at the headline size and 1e-13 against the FP64 path
    return {"rel": 1e-12 if case.get("mixed") else 5e-13}


# ------------------------------------------------------------------ the same in plain torch

def _bands(case):
    """Wall-normal bands a, b, c and those of the pinned mode."""
    yu = _faces(case)
    ny, yp = case["ny"], (yu[1:] + yu[:-1]) / 2
    if _bands_name(case) == "consistent":
        idy, gap = 1.0 / np.diff(yu), np.diff(yp)
        a = np.concatenate([[0.0], idy[1:] / gap])
        c = np.concatenate([idy[:-1] / gap, [0.0]])
        b = -(a + c)
        b00 = b.copy()
        b00[0] -= 2.0 * idy[0] / (2 * (yp[0] - yu[0]))
        return [(a, b, c), (a, b00, c)]
    ext = np.concatenate([[yu[0] - (yp[0] - yu[0])], yp, [yu[-1] + (yu[-1] - yp[-1])]])
    dy = 0.5 * (ext[2:] - ext[:-2])
    lo, up = 1.0 / ((ext[1:-1] - ext[:-2]) * dy), 1.0 / ((ext[2:] - ext[1:-1]) * dy)
    both = []
    for sign in (1.0, -1.0):  # zero gradient at both walls; the pinned mode is zero at the first
        a, b, c = lo.copy(), -(lo + up), up.copy()
        b[0] += sign * a[0]
        b[ny - 1] += c[ny - 1]
        a[0] = c[ny - 1] = 0.0
        both.append((a, b, c))
    return both


def _solve(case, rhs):
    nx, ny, nz = case["nx"], case["ny"], case["nz"]
    f = torch.fft.rfft2(rhs)
    sx = torch.sin(torch.arange(nx // 2 + 1, device="cuda", dtype=torch.float64) * math.pi / nx)
    sz = torch.sin(torch.arange(nz, device="cuda", dtype=torch.float64) * math.pi / nz)
    lam = -4 * (nz / LZ) ** 2 * sz.square()[:, None] - 4 * (nx / LX) ** 2 * sx.square()[None, :]
    (a, b, c), (a0, b0, c0) = _bands(case)

    def row(v, v0, k):
        r = torch.full_like(lam, float(v[k]))
        r[0, 0] = float(v0[k])
        return r

    up = torch.empty((ny, *lam.shape), device="cuda", dtype=torch.float64)
    for k in range(ny):
        low, d = row(a, a0, k), row(b, b0, k) + lam
        if k:
            d -= low * up[k - 1]
            f[k] -= low * f[k - 1]
        up[k] = row(c, c0, k) / d
        f[k] /= d
    for k in range(ny - 2, -1, -1):
        f[k] -= up[k] * f[k + 1]
    return torch.fft.irfft2(f, s=(nz, nx))


def _next(f, dim):
    return torch.roll(f, -1, dim)


def _before(f, dim):
    return torch.roll(f, 1, dim)


def _divergence(case, u, v, w):
    """Of interior fields with v on the lower faces: v = 0 on both walls."""
    idy = torch.from_numpy(1.0 / np.diff(_faces(case))).cuda()[:, None, None]
    d = (_next(u, 2) - u) * (case["nx"] / LX)
    d += (_next(w, 1) - w) * (case["nz"] / LZ)
    v = v.clone()
    v[0] = 0.0
    d += (torch.cat([v[1:], torch.zeros_like(v[:1])]) - v) * idy
    return d


def _wrapped(case, f):
    """Periodic halos in x and z, zero wall planes."""
    out = _halo(case, f)
    out[0] = out[-1] = 0.0
    return out


def exact(case, seed):
    d = _inputs(case, seed)
    if case["kind"] == "batch":
        cases = _batch_cases(case)
        parts = torch.split(d["rhs"], [c["nx"] * c["ny"] * c["nz"] for c in cases])
        return torch.cat([_solve(c, p.view(c["ny"], c["nz"], c["nx"])).reshape(-1) for c, p in zip(cases, parts)])
    if case["kind"] == "poisson":
        return _solve(case, d["rhs"])
    inner = (slice(1, -1),) * 3
    if case.get("rough"):
        k = torch.arange(case["ny"], device="cuda")[:, None, None]
        solid = (k <= d["inds"]["U_bot"]) | (k >= d["inds"]["U_top"])
        for f in d["hat"]:
            f[inner].masked_fill_(solid, 0.0)
    u, v, w = (f[inner] for f in d["hat"])
    idx, idz = case["nx"] / LX, case["nz"] / LZ
    yu = _faces(case)
    yp = (yu[1:] + yu[:-1]) / 2
    idy = torch.from_numpy(1.0 / np.diff(yu)).cuda()[:, None, None]
    idyp = torch.from_numpy(1.0 / np.diff(yp)).cuda()[:, None, None]
    div = _divergence(case, u, v, w)
    if case["kind"] == "step":
        P = _solve(case, div / DT)
        del div
        gx = gz = gy = P
        wx = wz = wy = 0.0
        ps = rmin = None
    else:
        rho, now, old, div_now = d["fields"]
        ps, half, rmin = 2.0 * now - old, 0.5 / rho, rho[inner].min()
        rhs = rmin / DT * (div - div_now[inner])

        def face(axis, at):  # (mean 1/rho, difference of ps) on the lower (0) or upper (1) faces
            hi, lo = list(inner), list(inner)
            hi[axis] = slice(2, None) if at else slice(1, -1)
            lo[axis] = slice(1, -1) if at else slice(0, -2)
            return half[tuple(hi)] + half[tuple(lo)], ps[tuple(hi)] - ps[tuple(lo)]

        pad = np.concatenate([[2 * yu[0] - yp[0]], yp, [2 * yu[-1] - yp[-1]]])
        ipad = torch.from_numpy(1.0 / np.diff(pad)).cuda()[:, None, None]
        for axis, scale in ((2, idx * idx), (1, idz * idz)):
            (r1, p1), (r0, p0) = face(axis, 1), face(axis, 0)
            rhs += ((1 - rmin * r1) * p1 - (1 - rmin * r0) * p0) * scale
        (r1, p1), (r0, p0) = face(0, 1), face(0, 0)
        rhs += ((1 - rmin * r1) * p1 * ipad[1:] - (1 - rmin * r0) * p0 * ipad[:-1]) * idy
        P = _solve(case, rhs)
        (rx, gx), (rz, gz), (ry, gy) = face(2, 0), face(1, 0), face(0, 0)
        wx, wz, wy = rx - 1 / rmin, rz - 1 / rmin, ry - 1 / rmin
    over = 1.0 if rmin is None else 1.0 / rmin
    un = u - DT * idx * ((P - _before(P, 2)) * over + wx * gx)
    wn = w - DT * idz * ((P - _before(P, 1)) * over + wz * gz)
    vn = torch.zeros_like(v)
    step = (P[1:] - P[:-1]) * over
    vn[1:] = v[1:] - DT * idyp * (step if rmin is None else step + wy[1:] * gy[1:])
    out = [_wrapped(case, f) for f in (un, vn, wn)]
    if case["kind"] == "vd":
        return [*out, _halo(case, P), P]
    if case.get("stats"):
        return [*out, P, float(_divergence(case, un, vn, wn).abs().max()), float(P.abs().max())]
    return [*out, P, *d["hat"]] if case.get("rough") else [*out, P]
