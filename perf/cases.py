"""The work that programs have this framework do, as timed cases through its public entry points.

Six kinds of call, each over a range of sizes (`draw` takes any of them):

  field    one realization of a planned field (`Plan.generate`): seeded device noise, or a noise
           buffer in the reference's draw order; 1D (the DFT pair), 2D and 3D, FP64 and FP32
  batch    several realizations of one 3D field with the log-normal value transform
           (`Plan.generate_batch`)
  ensemble one realization of each of many uneven 2D fields (`Ensemble.generate`)
  matvec   one product with the covariance matrix (`Plan.matvec`), FP64 and FP32
  inverse  one product with its inverse: conjugate gradients to a relative FP64 residual of 1e-12
           with FP32 or FP64 inner products (`Plan.multiply_inverse`); at that residual the
           solution is fixed to more digits than a change of rounding moves it, which the
           default mode's stagnation test does not give
  spectrum a new covariance: the eigenvalues of the torus and the first realization from them
           (`Plan.spectrum_build`, `Plan.generate`), as a loop over covariance parameters runs it

All buffers are on the device.  `exact` restates the same results with numpy and torch in 64 bits:
the covariance at the torus cells, its eigenvalues by an FFT, the counter-based noise
(Philox4x32-10 / 2x32-10 and Box-Muller) or the noise buffer scaled by their square roots, and
the backward transform; the matrix products by FFTs on the zero-padded field.
"""
import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "parafields-core_b200"))
import pfb200  # noqa: E402


def listed():
    return [
        # the smallest call: a coarse 2D map in the default precision, where launches and the
        # host path are the whole cost
        {"name": "field2d-64x48-f64", "kind": "field", "dim": 2, "n0": 64, "n1": 48, "n2": 1, "f64": True,
         "noise": False, "cov": "exponential", "ell": 0.1, "geo": False},
        # the 2D benchmark field (512^2, exponential, FP64), its noise drawn by the program
        {"name": "field2d-512-f64-noise", "kind": "field", "dim": 2, "n0": 512, "n1": 512, "n2": 1, "f64": True,
         "noise": True, "cov": "exponential", "ell": 0.1, "geo": False},
        # a 2D map whose sizes are round numbers, not powers of two
        {"name": "field2d-1000x600-f32", "kind": "field", "dim": 2, "n0": 1000, "n1": 600, "n2": 1, "f64": False,
         "noise": False, "cov": "matern32", "ell": 0.05, "geo": True},
        # the headline workload: a 256^3 Matern-3/2 field, FP32 realizations
        {"name": "field3d-256-f32", "kind": "field", "dim": 3, "n0": 256, "n1": 256, "n2": 256, "f64": False,
         "noise": False, "cov": "matern32", "ell": 0.1, "geo": False},
        # a 3D field of round sizes in the default precision
        {"name": "field3d-100-f64", "kind": "field", "dim": 3, "n0": 100, "n1": 100, "n2": 100, "f64": True,
         "noise": False, "cov": "exponential", "ell": 0.1, "geo": False},
        # a time series: both fields of one 1D noise draw (the DFT pair)
        {"name": "field1d-1000-f64", "kind": "field", "dim": 1, "n0": 1000, "n1": 1, "n2": 1, "f64": True,
         "noise": False, "cov": "exponential", "ell": 0.05, "geo": False},
        # log-normal realizations at 192^3 for a Monte Carlo run
        {"name": "batch3d-192-lognormal", "kind": "batch", "dim": 3, "n0": 192, "n1": 192, "n2": 192, "f64": False,
         "count": 4, "cov": "matern32", "ell": 0.1, "geo": False},
        # an ensemble of uneven 2D fields, sides log-uniform on [128, 1024]
        {"name": "ensemble2d-32", "kind": "ensemble", "count": 32, "lo": 128, "hi": 1024, "which": 20261203,
         "f64": False},
        # the covariance product of an inversion on a 128^3 grid with a rotated anisotropy
        {"name": "matvec3d-128-f64", "kind": "matvec", "dim": 3, "n0": 128, "n1": 128, "n2": 128, "f64": True,
         "cov": "exponential", "ell": 0.08, "geo": True},
        # the FP32 product on a grid with three different round sides
        {"name": "matvec3d-150x100x75-f32", "kind": "matvec", "dim": 3, "n0": 150, "n1": 100, "n2": 75, "f64": False,
         "cov": "exponential", "ell": 0.08, "geo": False},
        # timesInverseMatrix on a 128^3 grid, FP32 products inside FP64 residuals
        {"name": "inverse3d-128", "kind": "inverse", "dim": 3, "n0": 128, "n1": 128, "n2": 128, "f64": True,
         "inner32": True, "cov": "exponential", "ell": 0.05, "geo": False},
        # one step of a loop over covariance parameters on a 128 x 120 x 96 grid
        {"name": "spectrum3d-128x120x96", "kind": "spectrum", "dim": 3, "n0": 128, "n1": 120, "n2": 96, "f64": True,
         "noise": False, "cov": "exponential", "ell": 0.1, "geo": False},
    ]


def _side(rng, lo, hi):
    """A side length, log-uniform: a power of two, a round number, or any number, ragged ones too."""
    x = math.exp(rng.uniform(math.log(lo), math.log(hi)))
    how = rng.randrange(4)
    if how == 0:
        n = 2 ** round(math.log2(x))
    elif how == 1:
        n = 8 * round(x / 8)
    elif how == 2:
        n = 10 * round(x / 10)
    else:
        n = round(x)
    return max(lo, min(hi, n))


def draw(rng):
    kind = rng.choice(["field", "field", "field", "batch", "ensemble", "matvec", "matvec", "inverse", "spectrum"])
    if kind == "ensemble":
        return {"kind": kind, "count": rng.randint(4, 24), "lo": 128, "hi": 1024, "which": rng.randrange(1 << 30),
                "f64": False}
    f64 = kind in ("inverse", "spectrum") or (kind != "batch" and rng.random() < 0.5)
    dim = 3 if kind == "batch" else rng.choice([2, 3])
    if kind == "field" and rng.random() < 0.15:
        dim = 1
    lo, hi = {1: (16, 2000), 2: (24, 1500), 3: (16, 160)}[dim]
    if kind == "inverse":
        lo, hi = (24, 256) if dim == 2 else (12, 64)
    c = {"kind": kind, "dim": dim, "n0": _side(rng, lo, hi), "n1": _side(rng, lo, hi) if dim > 1 else 1,
         "n2": _side(rng, lo, hi) if dim > 2 else 1, "f64": f64}
    if kind == "inverse":
        c["inner32"] = rng.random() < 0.5
    if kind == "batch":
        c["count"] = rng.randint(2, 6)
    if kind in ("field", "spectrum"):
        c["noise"] = kind == "field" and rng.random() < 0.35
    c["cov"] = "exponential" if f64 or rng.random() < 0.5 else "matern32"
    c["ell"] = round(rng.uniform(0.03, 0.05 if kind == "inverse" else 0.15), 4)
    c["geo"] = dim > 1 and kind != "inverse" and rng.random() < 0.4
    return c


# ---------------------------------------------------------------------------
# descriptors
# ---------------------------------------------------------------------------
def _cells(c):
    return tuple(c["n%d" % i] for i in range(c["dim"]))


def _corr(c):
    """scalar, axiparallel or rotated (2D and 3D) correlation lengths"""
    d, ell = c["dim"], c["ell"]
    if not c["geo"]:
        return ell if d < 3 or c["kind"] == "inverse" else (2 * ell, ell, 0.5 * ell)
    t = 0.6
    r = np.eye(d)
    r[0, 0], r[0, 1], r[1, 0], r[1, 1] = math.cos(t), -math.sin(t), math.sin(t), math.cos(t)
    if d == 3:
        s = np.eye(3)
        s[1, 1], s[1, 2], s[2, 1], s[2, 2] = math.cos(t), -math.sin(t), math.sin(t), math.cos(t)
        r = r @ s
    return tuple((r @ np.diag([ell, 0.6 * ell, 0.4 * ell][:d])).ravel().tolist())


def _desc(c):
    return pfb200.make_desc(dim=c["dim"], cells=_cells(c), covariance=c["cov"], corr_length=_corr(c),
                            approximate=c["kind"] != "inverse",
                            precision=pfb200.PREC_F64 if c["f64"] else pfb200.PREC_F32,
                            transform="logNormal" if c["kind"] == "batch" else "none")


def _members(c):
    """the fields of an ensemble: (cells, covariance, variance, corr_length)"""
    rng = np.random.default_rng(c["which"])
    out = []
    for _ in range(c["count"]):
        n = [int(round(math.exp(rng.uniform(math.log(c["lo"]), math.log(c["hi"]))))) for _ in range(2)]
        cov = ["exponential", "gaussian", "spherical", "cubic"][int(rng.integers(4))]
        ell, var, t = rng.uniform(0.02, 0.3), rng.uniform(0.5, 2.0), rng.uniform(0, math.pi)
        co, si = math.cos(t), math.sin(t)
        out.append((tuple(n), cov, var, (ell * co, -ell * si, ell * si, ell * co)))
    return out


# ---------------------------------------------------------------------------
# inputs, passes
# ---------------------------------------------------------------------------
def _normal(n, seed, dtype=torch.float64):
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    return torch.randn(n, generator=g, device="cuda", dtype=dtype)


def prepare(case, seed):
    c = case
    ft = torch.float64 if c["f64"] else torch.float32
    if c["kind"] == "ensemble":
        descs = [pfb200.make_desc(dim=2, cells=n, covariance=cov, variance=var, corr_length=corr,
                                  anisotropy="geometric", approximate=True,
                                  precision=pfb200.PREC_F64 if c["f64"] else pfb200.PREC_F32)
                 for n, cov, var, corr in _members(c)]
        e = pfb200.Ensemble(descs, seed=seed)
        e.spectra()
        out = torch.empty(e.total, dtype=ft, device="cuda")
        e.generate(out)  # captures the graph that every later call replays
        return {"case": c, "ensemble": e, "out": out}
    plan = pfb200.Plan(_desc(c))
    s = {"case": c, "plan": plan, "seed": seed}
    n = plan.info.domain_size
    if c["kind"] != "spectrum":
        plan.spectrum_build()
    if c["kind"] in ("field", "spectrum"):
        s["noise"] = _normal(plan.info.noise_size, seed) if c["noise"] else None
        s["out"] = torch.empty(n, dtype=ft, device="cuda")
        if c["dim"] == 1:
            s["out2"] = torch.empty(n, dtype=ft, device="cuda")
    elif c["kind"] == "batch":
        s["out"] = torch.empty(n * c["count"], dtype=ft, device="cuda")
    else:
        s["x"] = _normal(n, seed, ft)
        s["out"] = torch.empty(n, dtype=ft, device="cuda")
    return s


def run(state):
    s, c = state, state["case"]
    if c["kind"] == "ensemble":
        return s["ensemble"].generate(s["out"])
    p = s["plan"]
    if c["kind"] == "field":
        first = p.generate(noise=s["noise"], seed=s["seed"], out=s["out"])
        if c["dim"] == 1:
            return first, p.generate(noise=s["noise"], seed=s["seed"], out=s["out2"])
        return first
    if c["kind"] == "spectrum":
        stats = p.spectrum_build()
        return stats, p.generate(seed=s["seed"], out=s["out"])
    if c["kind"] == "batch":
        return p.generate_batch(s["seed"], c["count"], out=s["out"], apply_transform=True)
    if c["kind"] == "matvec":
        return p.matvec(s["x"], precision=pfb200.PREC_F64 if c["f64"] else pfb200.PREC_F32, out=s["out"])
    return p.multiply_inverse(s["x"], x=s["out"], mode=pfb200.CG_RESIDUAL, tolerance=1e-12, max_iterations=2000,
                              inner_fp32=c["inner32"])[0]


# ---------------------------------------------------------------------------
# bytes and operations a pass cannot do without
# ---------------------------------------------------------------------------
def _field_work(cells, dct, f64, noise=False):
    """sqrt(eigenvalues) read (T/2+1 per axis where the axes mirror, the half spectrum otherwise), the
    noise buffer if any, the field written; the real transform of the torus, 2.5 N log2 N"""
    t = [2 * n for n in cells]
    big, es = math.prod(t), 8 if f64 else 4
    half = big // t[0] * (t[0] // 2 + 1)
    eig = math.prod(n // 2 + 1 for n in t) if dct else half
    return es * (eig + math.prod(cells)) + (16 * half if noise else 0), 2.5 * big * math.log2(big)


def work(case):
    c = case
    if c["kind"] == "ensemble":
        w = [_field_work(n, False, c["f64"]) for n, _, _, _ in _members(c)]
        return {"bytes": sum(x[0] for x in w), "flops": sum(x[1] for x in w)}
    cells, es = _cells(c), 8 if c["f64"] else 4
    n = math.prod(cells)
    if c["dim"] == 1:
        t = 2 * n
        return {"bytes": es * (t + 2 * n) + (16 * t if c["noise"] else 0), "flops": 5.0 * t * math.log2(t)}
    b, f = _field_work(cells, not c["geo"], c["f64"], c.get("noise", False))
    eig = b - es * n - (16 * (2 * cells[0] // 2 + 1) * 2 ** (c["dim"] - 1) * math.prod(cells[1:]) if c.get("noise") else 0)
    if c["kind"] == "batch":
        return {"bytes": eig + c["count"] * es * n, "flops": c["count"] * f}
    if c["kind"] == "matvec":
        return {"bytes": b + es * n, "flops": 2 * f}
    if c["kind"] == "inverse":  # 64 iterations, more or less: A d and the preconditioner
        return {"bytes": b + es * n, "flops": 256 * f}
    if c["kind"] == "spectrum":  # the eigenvalues written too; covariance evaluation not counted
        return {"bytes": b + eig, "flops": 2 * f}
    return {"bytes": b, "flops": f}


# ---------------------------------------------------------------------------
# the same results in 64 bits, with torch
# ---------------------------------------------------------------------------
M32 = 0xFFFFFFFF


def _mulhilo(a, m):
    """(high, low) words of the product of 32-bit words held in int64 with the 32-bit constant m"""
    p0, p1 = (a & 0xFFFF) * m, (a >> 16) * m
    return ((p1 + (p0 >> 16)) >> 16) & M32, (p0 + ((p1 & 0xFFFF) << 16)) & M32


def _philox4(x, y, z, w, seed):
    kx, ky = seed & M32, (seed >> 32) & M32
    for _ in range(10):
        h0, l0 = _mulhilo(x, 0xD2511F53)
        h1, l1 = _mulhilo(z, 0xCD9E8D57)
        x, y, z, w = h1 ^ y ^ kx, l1, h0 ^ w ^ ky, l0
        kx, ky = (kx + 0x9E3779B9) & M32, (ky + 0xBB67AE85) & M32
    return x, y, z, w


def _box_muller(a, b):
    r = torch.sqrt(-2.0 * torch.log((a.double() + 0.5) * 2.0 ** -32))
    t = math.pi * (b.double() * 2.0 ** -31 - 1.0)
    return torch.complex(r * torch.cos(t), r * torch.sin(t))


def _pair_noise(cells, seed, epoch):
    """complex noise of the half spectrum, shape (T_last, .., T0/2+1), natural order"""
    t = [2 * n for n in cells]
    c0 = t[0] // 2 + 1
    k0 = torch.arange(c0, device="cuda")
    if len(cells) == 2:
        si = k0 + c0 * torch.arange(t[1] // 2, device="cuda")[:, None]
    else:
        k1 = torch.arange(t[1], device="cuda")[:, None]
        k2 = torch.arange(t[2] // 2, device="cuda")[:, None, None]
        si = k0 + c0 * (k2 + t[2] * k1)
    full = torch.full_like(si, 0x70616972)
    a, b, g, h = _philox4(si & M32, si >> 32, full, torch.full_like(si, epoch), seed)
    return torch.cat([_box_muller(a, b), _box_muller(g, h)], 0)


def _covariance(dim, cells, cov, var, corr, aniso):
    """the covariance on the torus, shape (T_last, .., T0)"""
    x = []
    for i, n in enumerate(cells):
        v = torch.arange(2 * n, device="cuda", dtype=torch.float64) * (1.0 / n)
        v = torch.where(v > 1.0, v - 2.0, v)
        x.append(v.reshape([-1] + [1] * i))
    cl = np.atleast_1d(np.asarray(corr, dtype=np.float64)).ravel()
    if aniso == "geometric":
        g = np.linalg.inv(cl.reshape(dim, dim))
        y = [sum(float(g[i, k]) * x[k] for k in range(dim)) for i in range(dim)]
    else:
        y = [x[i] / float(cl[i if cl.size > 1 else 0]) for i in range(dim)]
    h = torch.sqrt(sum(v * v for v in y))
    if cov == "exponential":
        return var * torch.exp(-h)
    if cov == "gaussian":
        return var * torch.exp(-h * h)
    if cov == "matern32":
        return var * (1.0 + math.sqrt(3.0) * h) * torch.exp(-math.sqrt(3.0) * h)
    if cov == "spherical":
        hc = h.clamp(max=1.0)
        return var * (1.0 - 2.0 / math.pi * (hc * torch.sqrt(1.0 - hc * hc) + torch.asin(hc)))
    hc = h.clamp(max=1.0)  # cubic
    return torch.where(h > 1.0, torch.zeros_like(h), var * (1 - 7 * hc**2 + 8.75 * hc**3 - 3.5 * hc**5 + 0.75 * hc**7))


def _eigenvalues(dim, cells, cov, var, corr, aniso):
    """eigenvalues over N on the half spectrum (the whole one in 1D) before they are clamped"""
    c = _covariance(dim, cells, cov, var, corr, aniso)
    n = c.numel()
    return (torch.fft.fft(c) if dim == 1 else torch.fft.rfftn(c)).real / n


def _realization(cells, lam, z):
    t = [2 * n for n in cells]
    s = math.sqrt(0.5) * z
    ends = [[0, n] for n in cells]
    for i in ends[-1]:
        for j in (ends[1] if len(cells) == 3 else [0]):
            for k in ends[0]:
                at = (i, j, k) if len(cells) == 3 else (i, k)
                s[at] = z[at].real
    s = s * torch.sqrt(lam.clamp(min=0.0))
    for ax in range(len(cells) - 1):  # last field dimension first; the pruned part only
        s = torch.fft.ifft(s, dim=ax, norm="forward").narrow(ax, 0, cells[len(cells) - 1 - ax])
    s = s.contiguous()
    s[..., 0] = s[..., 0].real.to(s.dtype)
    s[..., -1] = s[..., -1].real.to(s.dtype)
    return torch.fft.irfft(s, n=t[0], dim=-1, norm="forward")[..., : cells[0]].reshape(-1)


def _product(cells, lam, x):
    shape = tuple(reversed(cells))
    t = tuple(2 * n for n in shape)
    y = torch.fft.irfftn(torch.fft.rfftn(x.reshape(shape), s=t) * lam, s=t)
    return y[tuple(slice(0, n) for n in shape)].reshape(-1)


def _solve(cells, lam, b):
    """A^-1 b by conjugate gradients preconditioned with the torus inverse, run far past convergence"""
    n2 = math.prod(2.0 * n for n in cells) ** 2
    inv = 1.0 / (lam * n2)
    x = torch.zeros_like(b)
    r = b.clone()
    z = _product(cells, inv, r)
    d = z.clone()
    rz = torch.dot(r, z)
    best, stall = float("inf"), 0
    for it in range(2000):
        q = _product(cells, lam, d)
        a = rz / torch.dot(d, q)
        x += a * d
        r = b - _product(cells, lam, x) if it % 20 == 19 else r - a * q
        z = _product(cells, inv, r)
        new = torch.dot(r, z)
        d = z + new / rz * d
        rz = new
        if it % 20 == 19:
            res = float(torch.linalg.vector_norm(r))
            stall = 0 if res < 0.5 * best else stall + 1
            best = min(best, res)
            if stall >= 3 or res == 0.0:
                break
    return x


def exact(case, seed):
    c = case
    if c["kind"] == "ensemble":
        out = []
        for i, (n, cov, var, corr) in enumerate(_members(c)):
            lam = _eigenvalues(2, n, cov, var, corr, "geometric")
            out.append(_realization(n, lam, _pair_noise(n, seed + i, 2)))  # the first pass is the second call
        return torch.cat(out)
    cells = _cells(c)
    aniso = "geometric" if c["geo"] else "axis"
    lam = _eigenvalues(c["dim"], cells, c["cov"], 1.0, _corr(c), aniso)
    if c["kind"] == "matvec":
        x = _normal(math.prod(cells), seed, torch.float64 if c["f64"] else torch.float32).double()
        return _product(cells, lam.clamp(min=0.0), x)
    if c["kind"] == "inverse":
        return _solve(cells, lam.clamp(min=0.0), _normal(math.prod(cells), seed))
    if c["dim"] == 1:
        t = 2 * cells[0]
        if c["noise"]:
            z = torch.view_as_complex(_normal(2 * t, seed).reshape(-1, 2))
        else:
            lo, hi, key = torch.arange(t, device="cuda"), torch.full((t,), seed >> 32, device="cuda"), seed & M32
            for _ in range(10):
                h, low = _mulhilo(lo, 0xD256D193)
                lo, hi, key = h ^ key ^ hi, low, (key + 0x9E3779B9) & M32
            z = _box_muller(lo, hi)
        f = torch.fft.ifft(torch.sqrt(lam.clamp(min=0.0)) * z, norm="forward")[: cells[0]]
        return f.real.contiguous(), f.imag.contiguous()
    if c["kind"] == "batch":
        return torch.cat([torch.exp(_realization(cells, lam, _pair_noise(cells, seed + r, 0)))
                          for r in range(c["count"])])
    if c["noise"]:
        t = [2 * n for n in cells]
        c0 = t[0] // 2 + 1
        z = torch.view_as_complex(_normal(2 * c0 * math.prod(t[1:]), seed).reshape(-1, 2))
        z = z.reshape(t[1], t[2], c0).transpose(0, 1).contiguous() if c["dim"] == 3 else z.reshape(t[1], c0)
    else:
        z = _pair_noise(cells, seed, 0)
    field = _realization(cells, lam, z)
    return (None, field) if c["kind"] == "spectrum" else field
