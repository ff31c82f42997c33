"""Workloads of the near-field-to-detector path, as a user's program runs them.

Every case is a scene with one call on it: a slice (`Context.simulate` and the
detector images read back), a spectral sweep, an extended source, or the Mie
coefficients alone.  Sizes come from the benchmark configurations
(`bimsim_gb300.scenes`), the command line's defaults and the test scenes;
spheres, refractive indices and Monte Carlo directions are drawn from the seed.

`exact` restates the path in plain torch / numpy double precision: tables,
bilinear lookups (or the direct order sums), full-size FFT band-pass.
"""
import ctypes
import math
import os
import sys

import numpy as np
import torch

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
sys.path.insert(0, os.path.join(ROOT, "bimsim-cuda_gb300"))

from bimsim_gb300 import (BS_FIELD_TOTAL, BS_IMG_ABSORBANCE, BS_IMG_INTENSITY, BS_PREC_FP64,  # noqa: E402
                          BS_PREC_MIXED, BimsimError, Context, abi, lib, scenes)

DEFAULTS = dict(kind="slice", precision="mixed", method="lut", res=64, fov=30.0, plane="xy", z=0.0, padding=1,
                supersample=1, lam=3.0, na_in=0.0, na_out=0.5, order=10, spheres=1, a_lo=1.0, a_hi=5.0, slab=0.0,
                waves=400, lut_uf=True, lut_r=0, lut_theta=0, uf_lut_r=0, bands=0, lam_hi=0.0, sources=0)


def case_of(name=None, **kw):
    c = dict(DEFAULTS, **kw)
    return dict(c, name=name) if name else c


def listed():
    return [
        # one small preview slice: two cells on a 16 x 16 detector; latency and launches are what it costs
        case_of("preview_16", res=16, fov=12.0, spheres=2, a_lo=1.0, a_hi=2.0, waves=48, lut_theta=256),
        # the command line's default setting for one sphere: tables of 2 R x 1000 samples, 400 directions
        case_of("one_sphere_256", res=256, fov=20.0, lam=2.5, spheres=1, a_lo=4.0, a_hi=5.0, lut_uf=False),
        # the plain method in double precision at its benchmark size: order sums, padding 2 (1280^2 near field)
        case_of("direct_fp64_256", precision="fp64", method="direct", res=256, fov=20.0, padding=2, lam=2.5,
                spheres=1, a_lo=4.9, a_hi=5.0, lut_uf=False),
        # the plain method in mixed precision on an odd grid in an xz plane, annular condenser, several spheres
        case_of("direct_xz_101", method="direct", res=101, fov=24.0, plane="xz", lam=2.2, na_in=0.1, na_out=0.45,
                spheres=5, a_lo=0.8, a_hi=2.5, slab=3.0, waves=200, lut_uf=False),
        # a double-precision table slice: what a user checks mixed results with
        case_of("lut_fp64_96", precision="fp64", res=96, fov=24.0, spheres=8, a_lo=0.8, a_hi=2.5, waves=200),
        # a served request of the smallest kind: coarse pixels, few directions; tables weigh most
        case_of("request_128", res=128, fov=100.0, lam=6.0, spheres=50, waves=200, lut_r=4096, lut_theta=1024,
                uf_lut_r=4096),
        # a served request of the middle kind: 120 spheres in a slab
        case_of("request_256", res=256, fov=100.0, lam=4.5, spheres=120, slab=30.0, waves=1000, lut_r=4096,
                lut_theta=1024, uf_lut_r=4096),
        # the benchmark's headline slice: 3072^2 near field, 50 spheres, 1000 directions
        case_of("slice_1024", res=1024, fov=100.0, spheres=50, waves=1000, lut_r=4096, lut_theta=1024,
                uf_lut_r=4096),
        # a short spectral sweep (the library chooses its kernels by its first bands)
        case_of("sweep_256", kind="sweep", res=256, fov=100.0, lam=2.5, lam_hi=12.5, bands=5, spheres=50, waves=1000,
                lut_r=4096, lut_theta=1024, uf_lut_r=4096),
        # extended illumination: point sources summed on the detector, tables built once
        case_of("sources_64", kind="sources", res=64, fov=30.0, spheres=12, a_lo=0.8, a_hi=2.5, sources=5),
        # a wide condenser, a plane above the spheres (forward angles), an odd supersampled grid, odd direction count
        case_of("wide_na_151", res=151, supersample=2, fov=40.0, z=3.0, lam=1.8, na_in=0.2, na_out=0.9, order=16,
                spheres=12, a_lo=0.5, a_hi=2.5, slab=2.0, waves=701),
        # Mie coefficients of many spheres into the caller's own device buffers
        case_of("mie_200", kind="mie", lam=2.0, spheres=200, a_lo=0.3, a_hi=12.0),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["slice"] * 5 + ["fp64", "direct", "direct64", "sweep", "sources", "mie"])
    if kind == "mie":
        return case_of(kind="mie", lam=round(rng.uniform(1.5, 6.0), 3), spheres=_log(rng, 2, 256), a_lo=0.3,
                       a_hi=round(rng.uniform(2.0, 15.0), 2))
    c = dict(res=_log(rng, 16, 400), fov=round(math.exp(rng.uniform(math.log(15), math.log(100))), 2),
             lam=round(rng.uniform(2.0, 10.0), 3), z=round(rng.choice([0.0, 0.0, rng.uniform(0.0, 4.0)]), 2),
             na_in=rng.choice([0.0, 0.0, 0.15]), na_out=rng.choice([0.5, 0.5, 0.35, 0.8]), spheres=_log(rng, 1, 100),
             waves=_log(rng, 40, 2000), slab=rng.choice([0.0, 3.0, 20.0]), lut_uf=rng.random() < 0.6)
    c["a_lo"] = round(0.01 * c["fov"] + 0.3, 3)
    c["a_hi"] = round(c["a_lo"] + 0.04 * c["fov"], 3)
    c["spheres"] = min(c["spheres"], 40 if c["slab"] == 0.0 else 100)
    if rng.random() < 0.5:
        c.update(lut_r=_log(rng, 512, 4096), lut_theta=_log(rng, 400, 1100), uf_lut_r=_log(rng, 512, 4096))
    cap = 4e10
    if kind == "fp64":
        c.update(precision="fp64", res=min(c["res"], 128), spheres=min(c["spheres"], 12))
        cap = 1.5e9
    elif kind in ("direct", "direct64"):
        c.update(method="direct", precision="fp64" if kind == "direct64" else "mixed", res=min(c["res"], 200),
                 spheres=min(c["spheres"], 8), plane=rng.choice(["xy", "xz"]), padding=rng.choice([1, 2]))
        cap = 4e9
    elif kind == "sweep":
        c.update(kind="sweep", bands=rng.randint(2, 6), lam=2.5, lam_hi=12.5, res=min(c["res"], 200), slab=0.0,
                 spheres=min(c["spheres"], 30))
        cap = 1e10
    elif kind == "sources":
        c.update(kind="sources", sources=rng.randint(2, 6), res=min(c["res"], 160))
        cap = 1e10
    R = c["res"] * (2 * c.get("padding", 1) + 1)
    c["waves"] = max(16, min(c["waves"], int(cap / (R * R * c["spheres"]))))
    return case_of(**c)


# ---------------------------------------------------------------------------
# The library's side
# ---------------------------------------------------------------------------
def params_of(c):
    s = c["fov"]
    geom = dict(xy=(s, c["z"])) if c["plane"] == "xy" else \
        dict(plane=((-s / 2, c["z"], -s / 2), (s / 2, c["z"], s / 2), (0.0, -1.0, 0.0)))
    return abi.make_params(lam=c["lam"], condenser=(c["na_in"], c["na_out"]), objective=(0.0, c["na_out"]),
                           resolution=c["res"], padding=c["padding"], supersample=c["supersample"],
                           field_order=c["order"], lut_us=c["method"] == "lut", lut_uf=c["lut_uf"],
                           us_lut_r=c["lut_r"], us_lut_theta=c["lut_theta"], uf_lut_r=c["uf_lut_r"], **geom)


def inputs_of(c, seed):
    """Spheres (x, y, z, a, n_re, n_im), directions, and what the kind needs beside them."""
    g = scenes.rng(seed * 1000003 + 17)
    if c["kind"] == "mie":
        a = np.exp(g.uniform(math.log(c["a_lo"]), math.log(c["a_hi"]), c["spheres"]))
        return dict(table=np.stack([a, g.uniform(1.2, 1.6, a.size), g.uniform(0.0, 0.05, a.size)], axis=1))
    sph = scenes.random_spheres(c["spheres"], c["fov"], c["a_lo"], c["a_hi"], seed=seed * 1009 + 2, z_slab=c["slab"])
    out = dict(spheres=sph, waves=scenes.mc_waves(c["waves"], c["na_in"], c["na_out"], seed=seed * 7919 + 1))
    if c["kind"] == "sweep":
        lam = np.linspace(c["lam"], c["lam_hi"], c["bands"])
        mats = [scenes.lorentz_material(lam, seed=seed * 31 + j) for j in range(3)]
        out.update(lambdas=lam, n_table=np.stack([mats[i % 3] for i in range(len(sph))], axis=1))
    if c["kind"] == "sources":
        xy = g.uniform(-0.25 * c["fov"], 0.25 * c["fov"], (c["sources"], 2))
        out["sources"] = np.column_stack([xy, np.full(c["sources"], c["z"]), g.uniform(0.3, 1.0, c["sources"])])
    return out


def mie_orders(a, lam):
    """Highest order of the series of a sphere (single precision, as the path counts it)."""
    f = np.float32
    ka = f(f(f(2) * f(3.14159)) * f(a)) / f(lam)
    return int(np.ceil(f(f(ka + f(f(4) * f(np.power(ka, f(1.0 / 3.0))))) + f(2))))


def prepare(case, seed):
    c, x = dict(DEFAULTS, **case), inputs_of(dict(DEFAULTS, **case), seed)
    if c["kind"] == "mie":
        dev = torch.device("cuda")
        nl = mie_orders(c["a_hi"], c["lam"])  # one order count for the caller's buffers; at most 127
        sph = torch.tensor(x["table"], dtype=torch.float64, device=dev)
        out = torch.empty((2, len(sph), nl + 1, 2), dtype=torch.float64, device=dev)
        return dict(kind="mie", lib=lib.library(), sph=sph, out=out, nl=nl, k=2 * float(np.float32(3.14159)) / c["lam"])
    ctx = Context(params_of(c))
    ctx.set_spheres(x["spheres"])
    ctx.set_waves(x["waves"])
    return dict(x, kind=c["kind"], ctx=ctx, prec=BS_PREC_FP64 if c["precision"] == "fp64" else BS_PREC_MIXED,
                field=c["precision"] == "fp64" and c["method"] == "lut")


def run(state):
    if state["kind"] == "mie":
        sph, out = state["sph"], state["out"]
        st = state["lib"].bs_mie_noalloc(ctypes.c_void_p(sph.data_ptr()), len(sph), state["nl"], state["k"],
                                         ctypes.c_void_p(out[0].data_ptr()), ctypes.c_void_p(out[1].data_ptr()),
                                         ctypes.c_void_p(torch.cuda.current_stream().cuda_stream))
        if st != 0:
            raise BimsimError(st, state["lib"].bs_last_error().decode())
        return dict(A=out[0], B=out[1])
    ctx, prec = state["ctx"], state["prec"]
    if state["kind"] == "sweep":
        return dict(intensity=ctx.sweep(state["lambdas"], state["n_table"], precision=prec))
    if state["kind"] == "sources":
        ctx.simulate_sources(state["sources"], prec)
    else:
        ctx.simulate(prec)
    f64 = prec == BS_PREC_FP64
    out = dict(intensity=ctx.image(BS_IMG_INTENSITY, f64=f64), absorbance=ctx.image(BS_IMG_ABSORBANCE, f64=f64))
    if state["field"]:
        out["field"] = ctx.field(BS_FIELD_TOTAL)
    return out


def work(case):
    """Inputs once, images once; the arithmetic of the slice's sums: 30 flop per (pixel, sphere, direction)
    lookup, 20 per (pixel, sphere, order pair) of the direct method, 26 per (pixel, order) of the incident
    field, 12 per (table entry, order)."""
    c = dict(DEFAULTS, **case)
    if c["kind"] == "mie":
        nl = mie_orders(c["a_hi"], c["lam"]) + 1
        return dict(bytes=c["spheres"] * (24.0 + 32.0 * nl), flops=c["spheres"] * nl * 300.0)
    R = c["res"] * c["supersample"] * (2 * c["padding"] + 1)
    slices = max(1, c["bands"], c["sources"])
    L = mie_orders(0.5 * (c["a_lo"] + c["a_hi"]), 0.5 * (c["lam"] + max(c["lam"], c["lam_hi"]))) + 1
    pairs = float(R) * R * c["spheres"]
    if c["method"] == "lut":
        tables = max(1, c["bands"]) * float(c["spheres"]) * (c["lut_r"] or 2 * R) * (c["lut_theta"] or 1000) * L
        us = slices * 30.0 * pairs * c["waves"] + 12.0 * tables
    else:
        us = slices * 20.0 * pairs * L * (L + 1) / 2
    es = 8 if c["precision"] == "fp64" else 4
    outs = c["res"] ** 2 * es * (max(1, c["bands"]) if c["kind"] == "sweep" else 2)
    if c["precision"] == "fp64" and c["method"] == "lut":
        outs += 16 * R * R
    return dict(bytes=48.0 * c["spheres"] + 24.0 * c["waves"] + outs,
                flops=us + slices * 26.0 * R * R * (c["order"] + 1))


# ---------------------------------------------------------------------------
# The path in plain double precision
# ---------------------------------------------------------------------------
PI_REF = 3.1415901184082031250   # the path's single-precision pi
CS = math.sqrt(3.14159 / math.pi)  # its scale of spherical Bessel values
EPS = 9.99999997475242707877e-07
F64, C128 = torch.float64, torch.complex128


def _dev():
    return torch.device("cuda" if torch.cuda.is_available() else "cpu")


def _bessel_j(N, z):
    """j_0 .. j_N of a real or complex array by Miller's downward recurrence; the values stay relative to
    1e-250 powers, so that small arguments do not overflow."""
    az = z.abs()
    top = max(float(N), float(az.max()))
    M = int(top + 20 + math.sqrt(70 * (top + 1)))
    fp, fc = torch.zeros_like(z), torch.full_like(z, 1e-300)
    scale = torch.zeros(z.shape, dtype=F64, device=z.device)
    kept = [None] * (N + 1)
    for l in range(M, 0, -1):
        fp, fc = fc, (2 * l + 1) / z * fc - fp
        big = fc.abs() > 1e200
        fc, fp = torch.where(big, fc * 1e-200, fc), torch.where(big, fp * 1e-200, fp)
        scale = scale + big
        if l - 1 <= N:
            kept[l - 1] = (fc, scale)
    s, c = torch.sin(z), torch.cos(z)
    j0, j1 = s / z, s / (z * z) - c / z
    f = [v * torch.pow(torch.tensor(1e-200, dtype=F64, device=z.device), scale - sc) for v, sc in kept]
    norm = j0 / f[0] if N < 1 else torch.where(j0.abs() >= j1.abs(), j0 / f[0], j1 / f[1])
    return torch.stack([v * norm for v in f]), j0, j1


def _bessel_y(N, z, y0, y1):
    y = [y0, y1]
    for l in range(2, N + 1):
        y.append((2 * l - 1) / z * y[-1] - y[-2])
    return torch.stack(y[: N + 1])


def _mie(a, n, k, N):
    """A_l, B_l (complex) of one sphere, orders 0..N."""
    ka, kna = torch.tensor([k * a], dtype=C128), torch.tensor([(n * k) * a], dtype=C128)
    l = torch.arange(N + 1, dtype=F64)[:, None]

    def primes(j, z):
        return torch.cat([-j[1:2], j[:-1] - (l[1:] + 1) * j[1:] / z])

    j, j0, _ = _bessel_j(N, ka)
    y0 = -torch.cos(ka) / ka
    if k * a > 12.0:  # the reference's y_0 slip above |z| = 12
        y0 = y0 + j0
    y = _bessel_y(N, ka, y0, -torch.cos(ka) / (ka * ka) - torch.sin(ka) / ka) * CS
    j = j * CS
    jn = _bessel_j(N, kna)[0] * CS
    jp, yp, jnp_ = primes(j, ka), primes(y, ka), primes(jn, kna)
    h, hp = j + 1j * y, jp + 1j * yp
    f = (2 * l + 1) * torch.tensor([1, 1j, -1, -1j], dtype=C128)[l.long() % 4]
    an, bn, cn = j * hp - jp * h, jn * hp - h * jnp_ * n, j * jnp_ * n - jn * jp
    return (f * an / bn)[:, 0], (f * cn / bn)[:, 0]


def _vec(v):
    return np.array(v, dtype=np.float64)


def _tri_dist(A, B, C, p):
    """Distance to a triangle by the region test of the path (regions 2, 4, 6 snap to a vertex)."""
    e0, e1, w = B - A, C - A, A - p
    a, b, c, d, e = e0 @ e0, e0 @ e1, e1 @ e1, e0 @ w, e1 @ w
    det, s, t = a * c - b * b, b * e - c * d, b * d - a * e
    if s + t <= det:
        if s < 0:
            s, t = 0.0, 0.0 if t < 0 or e >= 0 else min(1.0, -e / c)
        elif t < 0:
            s, t = (0.0 if d >= 0 else min(1.0, -d / a)), 0.0
        else:
            s, t = s / det, t / det
    elif s < 0:
        s, t = 0.0, 1.0
    elif t < 0:
        s, t = 1.0, 0.0
    else:
        num, den = c + e - b - d, a - 2 * b + c
        s = 0.0 if num <= 0 else min(1.0, num / den)
        t = 1 - s
    return float(np.linalg.norm(p - (A + e0 * s + e1 * t)))


class _Slice:
    """Geometry and incident field of one slice."""

    def __init__(self, p, waves, dev):
        self.p, self.dev = p, dev
        a, b, n = _vec(p.plane_min[:]), _vec(p.plane_max[:]), _vec(p.plane_normal[:])
        diag, side = b - a, np.cross(b - a, n)
        A, X, Y = a, diag * 0.5 + side * 0.5, diag * 0.5 - side * 0.5
        s = 2 * p.padding + 1
        mid = A + X * 0.5 + Y * 0.5
        self.X, self.Y = X * s, Y * s
        self.A = mid - self.X * 0.5 - self.Y * 0.5
        self.crop = p.resolution * p.supersample
        self.off = p.padding * self.crop
        self.R = self.crop * s
        self.k = 2 * PI_REF / p.lambda_
        self.cos_a, self.cos_b = (math.cos(math.asin(v)) for v in p.condenser[:])
        self.focus = _vec(p.focus[:])
        self.waves = torch.tensor(np.asarray(waves), dtype=F64, device=dev)
        sub = 2 * PI_REF * p.amplitude * ((1 - self.cos_b) - (1 - self.cos_a))
        self.amp = float(np.float32(1) / np.float32(len(waves))) * sub
        t = torch.arange(self.R, dtype=F64, device=dev) / self.R
        v, u = torch.meshgrid(t, t, indexing="ij")
        self.pos = torch.stack([self.A[i] + self.X[i] * u + self.Y[i] * v for i in range(3)], dim=-1).reshape(-1, 3)

    def dist(self, c):
        A, AX, AY = self.A, self.A + self.X, self.A + self.Y
        return min(_tri_dist(A, AX, AY, c), _tri_dist(AX + self.Y, AX, AY, c))

    def dist_max(self, c):
        return max(float(np.linalg.norm(q - c)) for q in (self.A, self.A + self.X, self.A + self.Y,
                                                           self.A + self.X + self.Y))

    def rel(self, c):
        r = self.pos - torch.tensor(c, dtype=F64, device=self.dev)
        return r, torch.sqrt((r * r).sum(-1))

    def incident(self):
        p, m = self.p, self.p.field_order
        r, d = self.rel(self.focus)
        center = d == 0 if p.lut_uf else d < EPS
        ds = torch.where(center, torch.ones_like(d), d)
        cth = (r @ torch.tensor(p.k_dir[:], dtype=F64, device=self.dev)) / ds
        if p.lut_uf:
            n = p.uf_lut_r or 2 * self.R
            lo, hi = self.dist(self.focus), self.dist_max(self.focus)
            kd = self.k * (torch.arange(n, dtype=F64, device=self.dev) * ((hi - lo) / (n - 1)) + lo)
            tab = _bessel_j(m, torch.where(kd < 1e-15, torch.ones_like(kd), kd))[0] * CS
            tab[:, kd < 1e-15] = 0.0
            tab[0, kd == 0] = 1.0
            y = ((ds - lo) / (hi - lo) * (n - 1)).clamp(0.0, n - 1.0)
            i0 = y.floor().long()
            be, i1 = y - i0, (i0 + 1).clamp(max=n - 1)
            jl = [(1 - be) * tab[l][i0] + be * tab[l][i1] for l in range(m + 1)]
        else:
            jl = _clamped_j(m, self.k * ds)
        w, pa, pb = [], [1.0, self.cos_a], [1.0, self.cos_b]
        for l in range(2, m + 2):
            for q, x in ((pa, self.cos_a), (pb, self.cos_b)):
                q.append(((2 * l - 1) * x * q[-1] - (l - 1) * q[-2]) / l)
        for l in range(m + 1):
            w.append(pa[l + 1] - pb[l + 1] - ((pa[l - 1] - pb[l - 1]) if l else 0.0))
        P0, P1, total = torch.ones_like(cth), cth, torch.zeros(d.shape, dtype=C128, device=self.dev)
        for l in range(m + 1):
            if l > 1:
                P0, P1 = P1, ((2 * l - 1) * cth * P1 - (l - 1) * P0) / l
            total = total + (1j ** l) * w[l] * jl[l] * (P0 if l == 0 else P1)
        scale = 2 * PI_REF * p.amplitude
        return torch.where(center, torch.full_like(total, scale * (self.cos_a - self.cos_b)), total * scale)

    def detector(self, U):
        """|band-passed crop|^2 binned to the detector."""
        p, R, C = self.p, self.R, self.crop
        i = torch.arange(R, device=self.dev)
        step = torch.where(i <= R // 2, i, -(R - 1 - i)).to(F64)
        fu, fv = step / float(np.linalg.norm(self.X)), step / float(np.linalg.norm(self.Y))
        f = torch.sqrt(fu[None, :] ** 2 + fv[:, None] ** 2)
        keep = (f >= p.objective[0] / p.lambda_) & (f <= p.objective[1] / p.lambda_)
        F = torch.fft.ifft2(torch.fft.fft2(U.reshape(R, R)) * keep)[self.off:self.off + C, self.off:self.off + C]
        I = F.real ** 2 + F.imag ** 2
        ss, res = p.supersample, p.resolution
        return I.reshape(res, ss, res, ss).mean(dim=(1, 3))


def _clamped_j(m, x):
    """j_0 .. j_m by the path's upward recurrence with its convergence clamp."""
    s, c = torch.sin(x), torch.cos(x)
    j = [s / x]
    j.append(j[0] / x - c / x)
    for l in range(2, m + 1):
        v = (2 * l - 1) * j[-1] / x - j[-2]
        re, xr = (v.real, x.real) if v.is_complex() else (v, x)
        j.append(torch.where((l > xr) & ((re < 0.0145) | (re > 0.4)), torch.zeros_like(v), v))
    return j[: m + 1]


def _clamped_y(m, x):
    s, c = torch.sin(x), torch.cos(x)
    y = [-c / x]
    y.append(y[0] / x - s / x)
    b0, b1 = y[0], y[1]
    for l in range(2, m + 1):
        v = (2 * l - 1) * b1 / x - b0
        cut = (v < -1e33) | ((v > 0) & (l > x))
        b0, b1 = torch.where(cut, torch.zeros_like(v), b1), torch.where(cut, torch.zeros_like(v), v)
        y.append(b1)
    return y[: m + 1]


def _scatter_lut(g, sph, phase):
    """Scattered field of one sphere from its two tables (bilinear in radius and angle)."""
    p, dev, R = g.p, g.dev, g.R
    ctr, a, n = _vec(sph[:3]), sph[3], complex(sph[4], sph[5])
    N = mie_orders(a, p.lambda_)
    A, B = (v.to(dev) for v in _mie(a, n, g.k, N))
    dmin, dmax = g.dist(ctr), g.dist_max(ctr)
    inter = math.sqrt(a - dmin) if dmin < a else 0.0
    aR = int(1 + 2.0 * R * inter / float(np.linalg.norm(g.X + g.Y)))
    dR, tR, r0 = p.us_lut_r or 2 * R, p.us_lut_theta or 1000, max(a, dmin)
    step = float(np.float32(3.14159) / np.float32(tR - 1))
    ct = torch.cos(step * torch.arange(tR, dtype=F64, device=dev))
    P = [torch.ones_like(ct), ct]
    for l in range(2, N + 1):
        P.append(((2 * l - 1) * ct * P[-1] - (l - 1) * P[-2]) / l)
    P = torch.stack(P).to(C128)
    x = g.k * (torch.arange(dR, dtype=F64, device=dev) * ((dmax - r0) / (dR - 1)) + r0)
    h = _bessel_j(N, x)[0] + 1j * _bessel_y(N, x, -torch.cos(x) / x, -torch.cos(x) / (x * x) - torch.sin(x) / x)
    tabs = [(B[:, None] * h * CS).T @ P]
    D = torch.zeros((aR, N + 1), dtype=C128, device=dev)
    D[0, 0] = A[0]
    if aR > 1:
        z = (n * g.k) * (torch.arange(1, aR, dtype=F64, device=dev) * (a / (aR - 1)))
        D[1:] = (A[:, None] * _bessel_j(N, z)[0] * CS).T
    tabs.append(D @ P)
    r, d = g.rel(ctr)
    inside = d < a
    rn = r / torch.where(d == 0, torch.ones_like(d), d)[:, None]
    out = torch.zeros(d.shape, dtype=C128, device=dev)
    for tab, sel, xs in ((tabs[0], ~inside, (d - r0) / (dmax - r0) * (dR - 1)),
                         (tabs[1], inside, (d - dmin) / (a - dmin) * (aR - 1) if a > dmin else d)):
        idx = sel.nonzero()[:, 0]
        rows, flat = tab.shape[0], tab.reshape(-1)
        for q in idx.split(max(1, (1 << 24) // len(g.waves))):
            y = xs[q].clamp(0.0, rows - 1.0)
            i0 = y.floor().long()
            al = (y - i0)[:, None]
            lo, hi = (i0 * tR)[:, None], ((i0 + 1).clamp(max=rows - 1) * tR)[:, None]
            c = torch.where((d[q] == 0)[:, None], torch.ones((), dtype=F64, device=dev), rn[q] @ g.waves.T)
            t = (torch.acos(c.clamp(-1.0, 1.0)) * (1.0 / PI_REF) * (tR - 1)).clamp(max=tR - 1.0)
            t0 = t.floor().long()
            be, t1 = t - t0, (t0 + 1).clamp(max=tR - 1)
            v = (1 - be) * ((1 - al) * flat[lo + t0] + al * flat[hi + t0]) + \
                be * ((1 - al) * flat[lo + t1] + al * flat[hi + t1])
            out[q] = v @ phase
    return out


def _scatter_direct(g, sph, phase):
    """Scattered field of one sphere by the order sums, each direction's Legendre series on its own."""
    ctr, a, n = _vec(sph[:3]), sph[3], complex(sph[4], sph[5])
    N = mie_orders(a, g.p.lambda_)
    A, B = (v.to(g.dev) for v in _mie(a, n, g.k, N))
    r, d = g.rel(ctr)
    ds = torch.where(d == 0, torch.ones_like(d), d)
    rn, inside = r / ds[:, None], d <= a
    kd = g.k * ds
    knd = torch.complex(kd * n.real, kd * n.imag)
    small = inside & (g.k * d * n.real < EPS)
    ji, jo, yo = _clamped_j(N, knd), _clamped_j(N, kd), _clamped_y(N, kd)
    coef = [torch.where(inside, A[l] * ji[l], B[l] * torch.complex(jo[l], yo[l])) for l in range(N + 1)]
    coef = [torch.where(small, (A[0] if l == 0 else 0 * A[0]).expand_as(c), c) for l, c in enumerate(coef)]
    out = torch.zeros(d.shape, dtype=C128, device=g.dev)
    for q in torch.arange(len(d), device=g.dev).split(max(1, (1 << 24) // len(g.waves))):
        x = rn[q] @ g.waves.T
        P0, P1 = torch.ones_like(x), x
        ph = torch.stack([phase.real, phase.imag], dim=1)
        for l in range(N + 1):
            if l > 1:
                P0, P1 = P1, ((2 * l - 1) * x * P1 - (l - 1) * P0) / l
            Q = (P0 if l == 0 else P1) @ ph
            out[q] = out[q] + coef[l][q] * torch.complex(Q[:, 0], Q[:, 1])
    return out


def _exact_slice(p, spheres, waves):
    """(D, Di, U) of one slice, double precision."""
    g = _Slice(p, waves, _dev())
    Uf = g.incident()
    U, outside = torch.zeros_like(Uf), torch.ones(Uf.shape, dtype=torch.bool, device=g.dev)
    for s in spheres:
        arg = g.k * (g.waves @ torch.tensor(_vec(s[:3]) - g.focus, dtype=F64, device=g.dev))
        phase = torch.polar(torch.full_like(arg, g.amp), arg)
        U = U + (_scatter_lut if p.lut_us else _scatter_direct)(g, s, phase)
        outside &= ~(g.rel(_vec(s[:3]))[1] < s[3])
    U = U + torch.where(outside, Uf, torch.zeros_like(Uf))
    return g.detector(U), g.detector(Uf), U.reshape(g.R, g.R)


def exact(case, seed):
    c, x = dict(DEFAULTS, **case), inputs_of(dict(DEFAULTS, **case), seed)
    if c["kind"] == "mie":
        nl = mie_orders(c["a_hi"], c["lam"])
        out = torch.zeros((2, len(x["table"]), nl + 1), dtype=C128)
        for i, (a, nr, ni) in enumerate(x["table"]):
            N = min(nl, mie_orders(a, c["lam"]))
            out[:, i, :N + 1] = torch.stack(_mie(a, complex(nr, ni), 2 * float(np.float32(3.14159)) / c["lam"], N))
        out = torch.view_as_real(out)
        return dict(A=out[0], B=out[1])
    p = params_of(c)
    R = p.resolution * p.supersample * (2 * p.padding + 1)
    slices = max(1, c["bands"], c["sources"])
    cost = float(R) * R * c["spheres"] * c["waves"] * slices
    if cost > 1.2e10 or (c["method"] == "direct" and cost > 2e9):
        return None
    if c["kind"] == "sweep":
        imgs = []
        for lam, row in zip(x["lambdas"], x["n_table"]):
            p.lambda_ = lam
            sph = [s[:4] + (n.real, n.imag) for s, n in zip(x["spheres"], row)]
            imgs.append(_exact_slice(p, sph, x["waves"])[0].cpu())
        return dict(intensity=torch.stack(imgs))
    if c["kind"] == "sources":
        D = Di = 0
        for s in x["sources"]:
            p.focus[:], p.amplitude = list(s[:3]), s[3]
            d, di, _ = _exact_slice(p, x["spheres"], x["waves"])
            D, Di = D + d, Di + di
        return dict(intensity=D.cpu(), absorbance=-torch.log10(D / Di).cpu())
    D, Di, U = _exact_slice(p, x["spheres"], x["waves"])
    out = dict(intensity=D.cpu(), absorbance=-torch.log10(D / Di).cpu())
    if c["precision"] == "fp64" and c["method"] == "lut":
        out["field"] = U.cpu()
    return out
