"""Timed cases: what a user of this framework has it compute, through its public entry points.

Every case is one call (or one sequence of calls) of the Python mirror of the toolbox's functions on arrays that
are resident on the GPU.  Volumes are torch tensors of shape (nz, ny, nx), C-contiguous, which is MATLAB's layout.
Inputs are synthetic and made on the GPU from the seed: ellipsoid susceptibility phantoms and their dipole fields
inside an ellipsoidal brain mask, sums of Gaussians for the Poisson problems, a harmonic background for the
background-removal functions.  Sizes are those of the repository's benchmark and test configurations, and odd,
anisotropic ones.

``exact`` restates each call in 64-bit torch: the finite-difference operators, the primal-dual iterations, the ADMM
loop and the spherical-mean-value filter step by step; a Poisson solve by its discrete solution (conjugate gradients
run to 1e-13), which the solvers reach to their tolerance.
"""
from __future__ import annotations

import math
import struct

import numpy as np
import torch

import qsm_gb300 as q

PI = math.pi
F64 = torch.float64


def _dev():
    return "cuda" if torch.cuda.is_available() else "cpu"


def _dt(case):
    return torch.float64 if case["dtype"] == "float64" else torch.float32


def _shape(case):
    return (case["nz"], case["ny"], case["nx"])


def _h(case):
    return (case["hx"], case["hy"], case["hz"])


def _vox(case):
    return case["nx"] * case["ny"] * case["nz"]


ELLIPSOID = 4.0 / 3.0 * PI * 0.42 ** 3  # share of the grid inside the brain mask


# ---------------------------------------------------------------------------
# the cases
# ---------------------------------------------------------------------------

def _case(kind, n, **kw):
    h = kw.pop("h", (1.0, 1.0, 1.0))
    c = dict(kind=kind, nx=n[0], ny=n[1], nz=n[2], hx=h[0], hy=h[1], hz=h[2])
    c.update(kw)
    return c


def listed():
    out = []

    def add(name, *a, **kw):
        c = _case(*a, **kw)
        c["name"] = name
        out.append(c)

    # One gradient of a small volume: the smallest call a script makes, inside loops of its own (latency).
    add("gradf f32 64x64x40", "fd", (64, 64, 40), op="gradf", dtype="float32")
    # Laplacian of a wrapped high-resolution phase volume, MATLAB's default class: the first step of sstgv.m and
    # unwrapLaplacian.m, on its own.
    add("lapw f64 320x320x192", "fd", (320, 320, 192), op="lapw", dtype="float64", h=(0.7, 0.7, 0.7))
    # The headline inversion: single-step TGV, whole head, mixed-precision path, 1000 iterations.
    add("tgv fused f32 224x224x128", "tgv", (224, 224, 128), dtype="float32", fused=True, iters=1000)
    # A small inversion (the 64^3 test configuration) on the same path: many short dependent iterations.
    add("tgv fused f32 64x64x64", "tgv", (64, 64, 64), dtype="float32", fused=True, iters=1000)
    # The same gateway with MATLAB's default class and the reference's own arithmetic (the default path of
    # pd_tgv_mex), on an anisotropic volume of odd size.
    add("tgv plain f64 181x217x91", "tgv", (181, 217, 91), dtype="float64", fused=False, iters=100,
        h=(1.0, 1.0, 2.0))
    # A study: several TV inversions of uneven size advanced together.
    add("tv batch f32 8 volumes", "tv_batch", (256, 256, 176), dtype="float32", iters=300,
        sizes="96x96x64,208x240x160,144x112x96,256x256x176,160x192x128,128x224x80,240x176x144,112x144x112")
    # Laplacian boundary value problem on a whole head, all FP64 (bit-exact multigrid PCG).
    add("mgpcg f64 256x256x256", "mgpcg", (256, 256, 256), mixed=False)
    # The same solver with its FP32 V-cycle on an odd, anisotropic volume.
    add("mgpcg mixed 181x217x155", "mgpcg", (181, 217, 155), mixed=True, h=(0.9, 0.9, 1.2))
    # lbv.m with its defaults, two echoes: crop, Laplacian and a Poisson solve on lbv.m's shallow hierarchy.
    add("lbv f64 224x224x128x2", "lbv", (224, 224, 128), dtype="float64", echoes=2, mixed=False)
    # vsharp.m with its defaults (radii 9:-2:2), one echo, MATLAB's default class.
    add("vsharp f64 224x224x128", "vsharp", (224, 224, 128), dtype="float64", echoes=1)
    # tv.m's ADMM inversion in single precision.
    add("tv admm f32 224x224x128", "tv_admm", (224, 224, 128), dtype="float32", iters=50, tv=1)
    # Loading a 4-echo int16 series into GPU memory: byte order, scaling, reorientation.
    add("nifti int16 224x224x128x4", "nifti", (224, 224, 128), echoes=4, stored="int16", orient="LPS")
    return out


def draw(rng):
    def log(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    def dims(lo, hi, limit):
        while True:
            n = (log(lo, hi), log(lo, hi), log(max(24, lo * 3 // 4), max(lo, hi * 3 // 4)))
            if n[0] * n[1] * n[2] <= limit:
                return n

    h = rng.choice([(1.0, 1.0, 1.0), (1.0, 1.0, 1.0), (0.8, 0.8, 0.8), (1.0, 1.0, 2.0), (0.9, 0.95, 1.3)])
    kind = rng.choice(["fd", "fd", "tgv", "tgv", "tgv", "tv_batch", "mgpcg", "mgpcg", "lbv", "vsharp", "tv_admm",
                       "nifti"])
    dt = rng.choice(["float32", "float64"])
    if kind == "fd":
        return _case(kind, dims(32, 320, 19_000_000), op=rng.choice(["gradf", "gradfm_adj", "lap1", "lapw"]),
                     dtype=dt, h=h)
    if kind == "tgv":
        fused = rng.random() < 0.6
        if fused:
            n = dims(48, 224, 6_400_000)
            return _case(kind, n, dtype=dt, fused=True, iters=rng.randrange(200, 801), h=h)
        n = dims(48, 192, 3_500_000)
        return _case(kind, n, dtype=dt, fused=False, iters=rng.randrange(40, 101), h=h)
    if kind == "tv_batch":
        sz = [dims(64, 224, 5_000_000) for _ in range(rng.randrange(3, 8))]
        return _case(kind, tuple(max(s[a] for s in sz) for a in range(3)), dtype="float32",
                     iters=rng.randrange(100, 301), h=h, sizes=",".join("%dx%dx%d" % s for s in sz))
    if kind == "mgpcg":
        return _case(kind, dims(96, 240, 10_000_000), mixed=rng.random() < 0.5, h=h)
    if kind == "lbv":
        mixed = rng.random() < 0.4
        return _case(kind, dims(96, 200, 5_000_000), dtype="float64" if mixed else dt, echoes=1, mixed=mixed)
    if kind == "vsharp":
        return _case(kind, dims(80, 224, 6_000_000), dtype=dt, echoes=rng.randrange(1, 3))
    if kind == "tv_admm":
        return _case(kind, dims(64, 224, 6_000_000), dtype=dt, iters=rng.randrange(20, 50), tv=rng.choice([1, 1, 2]),
                     h=h)
    return _case(kind, dims(48, 224, 6_000_000), echoes=rng.randrange(1, 5),
                 stored=rng.choice(["int16", "uint16", "float32"]), orient=rng.choice(["LPS", "RAS", "sagittal"]))


# ---------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------

def _axes(shape):
    return [torch.arange(n, dtype=F64, device=_dev()).reshape([-1 if a == b else 1 for b in range(3)])
            for a, n in enumerate(shape)]


def _brain(shape, rng):
    """Ellipsoidal mask with semi-axes 0.42 of the grid, its centre off by up to a voxel."""
    q2 = 0.0
    for g, n in zip(_axes(shape), shape):
        c = (n - 1) / 2 + rng.uniform(-1.0, 1.0) * min(1.0, n / 64)
        q2 = q2 + ((g - c) / (0.42 * n)) ** 2
    return (q2 <= 1.0).to(torch.uint8).contiguous()


def _phantom(shape, rng, count, lim):
    """Ellipsoids of susceptibility U[-lim, lim] (ppm), later ones over earlier ones."""
    g = _axes(shape)
    chi = torch.zeros(shape, dtype=F64, device=_dev())
    for _ in range(count):
        c = [n * rng.uniform(0.22, 0.78) for n in shape]
        a = [rng.uniform(4.0, 16.0) for _ in shape]
        inside = sum(((g[i] - c[i]) / a[i]) ** 2 for i in range(3)) <= 1.0
        chi = torch.where(inside, torch.full_like(chi, rng.uniform(-lim, lim)), chi)
    return chi


def _freq2(shape, h):
    """k-space coordinates (z, y, x order) of a volume."""
    return [torch.fft.fftfreq(n, d=d, dtype=F64, device=_dev()).reshape([-1 if a == b else 1 for b in range(3)])
            for a, (n, d) in enumerate(zip(shape, (h[2], h[1], h[0])))]


def _dipole(shape, h):
    kz, ky, kx = _freq2(shape, h)
    k2 = kx * kx + ky * ky + kz * kz
    k2[0, 0, 0] = 1.0
    D = 1.0 / 3.0 - kz * kz / k2
    D[0, 0, 0] = 0.0
    return D


def _local_field(shape, h, rng, gen, count=20, lim=0.1, noise=0.01):
    chi = _phantom(shape, rng, count, lim)
    phi = torch.fft.ifftn(_dipole(shape, h) * torch.fft.fftn(chi)).real
    return phi + noise * torch.randn(shape, dtype=F64, device=_dev(), generator=gen)


def _background(shape, h, rng):
    """Harmonic field of four point sources outside the grid."""
    g = _axes(shape)
    ext = [n * d for n, d in zip(shape, (h[2], h[1], h[0]))]
    step = (h[2], h[1], h[0])
    bg = 0.0
    for _ in range(4):
        ax = int(rng.integers(0, 3))
        c = [rng.uniform(0.2, 0.8) * e for e in ext]
        c[ax] = -0.25 * ext[ax] if rng.random() < 0.5 else 1.25 * ext[ax]
        r = torch.sqrt(sum((g[i] * step[i] - c[i]) ** 2 for i in range(3)))
        bg = bg + rng.uniform(0.5, 1.5) / r
    return bg


def _lapw64(u, h):
    """Laplacian of a wrapped phase on the interior, 0 on the faces."""
    d = torch.zeros_like(u)
    core = (slice(1, -1),) * 3
    acc = 0.0
    for ax, step in ((2, h[0]), (1, h[1]), (0, h[2])):
        up, dn = list(core), list(core)
        up[ax], dn[ax] = slice(2, None), slice(0, -2)
        f = u[tuple(up)] - u[core]
        b = u[core] - u[tuple(dn)]
        acc = acc + (_wrap(f) - _wrap(b)) / (step * step)
    d[core] = acc
    return d


def _wrap(x):
    y = x + PI
    y = torch.where(y < 0, torch.fmod(y, 2 * PI) + PI, torch.fmod(y, 2 * PI) - PI)
    return torch.where((x < -PI) | (x > PI), y, x)


def _lap7(u, h):
    """7-point Laplacian on the interior, 0 on the faces."""
    d = torch.zeros_like(u)
    core = (slice(1, -1),) * 3
    acc = 0.0
    for ax, step in ((2, h[0]), (1, h[1]), (0, h[2])):
        up, dn = list(core), list(core)
        up[ax], dn[ax] = slice(2, None), slice(0, -2)
        acc = acc + (u[tuple(up)] - 2.0 * u[core] + u[tuple(dn)]) / (step * step)
    d[core] = acc
    return d


def _seeded(seed):
    gen = torch.Generator(device=_dev())
    gen.manual_seed(int(seed))
    return np.random.default_rng(int(seed)), gen


def _levels(n):
    """The depth mgpcg.m and lbv.m choose."""
    return max(1, int(math.floor(math.log2(min(n)))) - 3)


def _sizes(case):
    return [tuple(int(x) for x in s.split("x")) for s in case["sizes"].split(",")]


def _tgv_input(shape, h, rng, gen):
    """(d2f, mask) of an inversion: minus the Laplacian of a local field (ppm), and the brain mask."""
    m = _brain(shape, rng)
    return -_lapw64(_local_field(shape, h, rng, gen), h), m


def _inputs(case, seed):
    """The arrays a call takes, in its dtype."""
    rng, gen = _seeded(seed)
    shape, h, kind = _shape(case), _h(case), case["kind"]
    if kind == "fd":
        dt = _dt(case)
        m = _brain(shape, rng)
        u = _local_field(shape, h, rng, gen, count=8) + _background(shape, h, rng) * 40.0
        if case["op"] == "lapw":
            u = _wrap(u * 20.0)
        if case["op"] == "gradfm_adj":
            xyz = [(u * s + 0.1 * torch.randn(shape, dtype=F64, device=_dev(), generator=gen)).to(dt)
                   for s in (1.0, -0.5, 0.25)]
            return dict(xyz=xyz, m=m)
        return dict(u=u.to(dt), m=m)
    if kind == "tgv":
        d2f, m = _tgv_input(shape, h, rng, gen)
        return dict(f=d2f.to(_dt(case)), m=m)
    if kind == "tv_batch":
        pairs = [_tgv_input((n[2], n[1], n[0]), h, rng, gen) for n in _sizes(case)]
        return dict(fs=[d.to(_dt(case)) for d, _ in pairs], ms=[m for _, m in pairs])
    if kind == "mgpcg":
        m = _brain(shape, rng)
        g = _axes(shape)
        u = torch.zeros(shape, dtype=F64, device=_dev())
        for _ in range(12):
            s = rng.uniform(5.0, 30.0)
            e = [torch.exp(-((g[i] - rng.uniform(0, shape[i] - 1)) ** 2) / (2 * s * s)) for i in range(3)]
            u = u + rng.uniform(-1.0, 1.0) * e[0] * e[1] * e[2]
        return dict(f=-_lap7(u, h) * m, m=m)
    if kind in ("lbv", "vsharp"):
        m = _brain(shape, rng)
        loc = _local_field(shape, h, rng, gen)
        bg = _background(shape, h, rng)
        bg = bg * (10.0 * loc.abs().max() / bg.abs().max())
        f = torch.stack([(t + 1) * (loc + bg) * m for t in range(case["echoes"])])
        return dict(f=(f[0] if case["echoes"] == 1 else f).to(_dt(case)).contiguous(), m=m)
    if kind == "tv_admm":
        m = _brain(shape, rng)
        return dict(f=(_local_field(shape, h, rng, gen) * m).to(_dt(case)), m=m)
    if kind == "nifti":
        n = case["echoes"] * _vox(case)
        stored = case["stored"]
        if stored == "float32":
            raw = torch.randn(n, dtype=torch.float32, device=_dev(), generator=gen)
        else:
            lo, hi = (-32768, 32768) if stored == "int16" else (0, 65536)
            raw = torch.randint(lo, hi, (n,), dtype=torch.int32, device=_dev(), generator=gen)
            raw = (raw if stored == "int16" else raw - (raw >= 32768).to(torch.int32) * 65536).to(torch.int16)
        slope, inter = float(np.float32(rng.uniform(1e-4, 1e-3))), float(np.float32(rng.uniform(-1.0, 1.0)))
        return dict(raw=raw, slope=slope, inter=inter, hdr=_nifti_header(case, slope, inter))
    raise ValueError(kind)


_SFORM = {"LPS": ((-1, 0, 0), (0, -1, 0), (0, 0, 1)), "RAS": ((1, 0, 0), (0, 1, 0), (0, 0, 1)),
          "sagittal": ((0, 0, -1), (1, 0, 0), (0, 1, 0))}  # rows: x, y, z of the stored axes


def _nifti_header(case, slope, inter):
    b = bytearray(352)
    code, bits = {"int16": (4, 16), "uint16": (512, 16), "float32": (16, 32)}[case["stored"]]
    struct.pack_into("<i", b, 0, 348)
    struct.pack_into("<8h", b, 40, 4, case["nx"], case["ny"], case["nz"], case["echoes"], 1, 1, 1)
    struct.pack_into("<hh", b, 70, code, bits)
    struct.pack_into("<8f", b, 76, 1, 1, 1, 1, 1, 1, 1, 1)
    struct.pack_into("<fff", b, 108, 352.0, slope, inter)
    b[123] = 2
    struct.pack_into("<h", b, 254, 1)
    for r, row in enumerate(_SFORM[case["orient"]]):
        struct.pack_into("<4f", b, 280 + 16 * r, *row, 0.0)
    b[344:348] = b"n+1\0"
    return bytes(b)


def prepare(case, seed):
    s = _inputs(case, seed)
    if case["kind"] == "fd":  # the operators write into the caller's arrays
        like = s["xyz"][0] if "xyz" in s else s["u"]
        s["out"] = [torch.zeros_like(like) for _ in range(3 if case["op"] == "gradf" else 1)]
    if case["kind"] == "nifti":
        s["payload"] = s.pop("raw").view(torch.uint8)
    s["case"] = case
    return s


# ---------------------------------------------------------------------------
# one pass
# ---------------------------------------------------------------------------

def run(s):
    c = s["case"]
    h, kind = _h(c), c["kind"]
    if kind == "fd":
        o, op = s["out"], c["op"]
        if op == "gradf":
            q.gradf_mex(o[0], o[1], o[2], s["u"], h)
        elif op == "gradfm_adj":
            q.gradfm_adj_mex(o[0], *s["xyz"], s["m"], h)
        elif op == "lap1":
            q.lap1_mex(o[0], s["u"], s["m"], h)
        else:
            q.lapw_mex(o[0], s["u"], h)
        return o
    if kind == "tgv":
        return q.pd_tgv_mex(s["f"], s["m"], h, 0.003, 2.0, 0.0, c["iters"], fused=c["fused"])
    if kind == "tv_batch":
        return q.pd_tv_batch(s["fs"], s["ms"], h, 1e-3, 0.0, c["iters"])
    if kind == "mgpcg":
        return q.mgpcg_mex(None, s["f"], s["m"], h, 1e-8, 100, -1.0, 2, 1, 2, 2, 2,
                           _levels((c["nx"], c["ny"], c["nz"])), mixed=c["mixed"])
    if kind == "lbv":
        return q.lbv(s["f"], s["m"], h, mixed=c["mixed"])
    if kind == "vsharp":
        return q.vsharp(s["f"], s["m"], h)
    if kind == "tv_admm":
        return q.tv(s["f"], s["m"], h, opts=dict(maxit=c["iters"], rtol=0.0, atol=0.0, tv=c["tv"]))
    img, _ = q.nifti.decode(s["hdr"], s["payload"], device=True)
    return img


# ---------------------------------------------------------------------------
# work
# ---------------------------------------------------------------------------

def work(case):
    """Bytes and operations of one pass.  An iterative solver's state is larger than the caches: it is read and
    written once an iteration, on the mask's voxels alone."""
    kind, n = case["kind"], _vox(case)
    b = 8 if case.get("dtype", "float64") == "float64" else 4
    if kind == "fd":
        arrays, ops = {"gradf": (4, 6), "gradfm_adj": (4, 8), "lap1": (2, 14), "lapw": (2, 25)}[case["op"]]
        mask = 1 if case["op"] in ("gradfm_adj", "lap1") else 0
        return {"bytes": n * (arrays * b + mask), "flops": n * ops}
    if kind == "tgv":
        vox, sb = n * ELLIPSOID, (4 if case["fused"] else b)
        # 15 state arrays of the iterates and duals read, 15 written, the previous iterates and f read
        return {"bytes": case["iters"] * vox * 36 * sb + n * (2 * b + 1), "flops": case["iters"] * vox * 160}
    if kind == "tv_batch":
        n = sum(x * y * z for x, y, z in _sizes(case))
        return {"bytes": case["iters"] * n * ELLIPSOID * 15 * 4 + n * 9, "flops": case["iters"] * n * ELLIPSOID * 65}
    if kind in ("mgpcg", "lbv"):
        # per PCG iteration two V-cycles of 4 sweeps (3 arrays), a residual and transfers on 8/7 of the voxels, and
        # the recurrence (10 arrays); about 10 iterations to 1e-8 on the deep hierarchy, 7 on lbv.m's
        vb, it = (4 if case["mixed"] else b), (10 if kind == "mgpcg" else 7 * case["echoes"])
        vox = n * ELLIPSOID
        return {"bytes": it * vox * (2 * 16 * vb * 8 / 7 + 10 * b) + n * (2 * b + 1), "flops": it * vox * 140}
    if kind == "vsharp":
        # forward transform, one complex inverse per pair of radii, one deconvolution; each transform reads and
        # writes its array once per axis
        t = 2 + 2 * 2
        return {"bytes": case["echoes"] * n * b * 2 * 3 * t, "flops": case["echoes"] * n * t * 2.5 * math.log2(n)}
    if kind == "tv_admm":
        return {"bytes": case["iters"] * n * (13 + 7 + 12) * b, "flops": case["iters"] * n * (90 + 5 * math.log2(n))}
    n *= case["echoes"]
    return {"bytes": n * ((4 if case["stored"] == "float32" else 2) + 4), "flops": 2 * n}


# ---------------------------------------------------------------------------
# 64-bit restatements
# ---------------------------------------------------------------------------

def _fd64(case, s):
    op, h, m = case["op"], _h(case), s["m"] != 0
    if op == "lapw":
        return [_lapw64(s["u"].to(F64), h)]
    ax = ((2, h[0]), (1, h[1]), (0, h[2]))
    if op == "gradf":
        u, out = s["u"].to(F64), []
        for a, d in ax:
            g = torch.diff(u, dim=a) / d
            out.append(torch.cat([g, g.narrow(a, g.shape[a] - 1, 1)], dim=a))
        return out
    if op == "gradfm_adj":
        acc = 0.0
        for (a, d), v in zip(ax, s["xyz"]):
            v = v.to(F64)
            lo, hi = _shifted(m, a, -1), _shifted(m, a, 1)
            back, fwd = v - _shifted(v, a, -1), _shifted(v, a, 1) - v
            zero = torch.zeros_like(v)
            acc = acc + torch.where(lo, back, torch.where(hi, fwd, zero)) * (-1.0 / d)
        return [torch.where(m, acc, torch.zeros_like(acc))]
    return [_lap1_64(s["u"].to(F64), m, h)]


def _shifted(v, ax, k):
    """v at the neighbour k steps along an axis, 0 (False) beyond the grid."""
    out = torch.zeros_like(v)
    n = v.shape[ax]
    if abs(k) < n:
        out.narrow(ax, max(0, -k), n - abs(k)).copy_(v.narrow(ax, max(0, k), n - abs(k)))
    return out


def _lap1_64(u, m, h):
    """lap1_mex for a mask that touches no face: central where both neighbours are inside, else one-sided with as
    many points as the mask holds."""
    acc = torch.zeros_like(u)
    for a, d in ((2, h[0]), (1, h[1]), (0, h[2])):
        u1, u2, u3 = (_shifted(u, a, k) for k in (1, 2, 3))
        v1, v2, v3 = (_shifted(u, a, -k) for k in (1, 2, 3))
        m1, m2, m3 = (_shifted(m, a, k) for k in (1, 2, 3))
        l1, l2, l3 = (_shifted(m, a, -k) for k in (1, 2, 3))
        fwd = torch.where(m2 & m3, 2 * u - 5 * u1 + 4 * u2 - u3, torch.where(m2, u - 2 * u1 + u2, u1 - u))
        bwd = torch.where(l2 & l3, 2 * u - 5 * v1 + 4 * v2 - v3, torch.where(l2, u - 2 * v1 + v2, v1 - u))
        val = torch.where(m1 & l1, v1 - 2 * u + u1, torch.where(m1, fwd, torch.where(l1, bwd, torch.zeros_like(u))))
        acc = acc + val / (d * d)
    return torch.where(m, acc, torch.zeros_like(acc))


def _box(m, margin):
    """Slices of the mask's bounding box grown by a margin, clamped."""
    out = []
    for a in range(3):
        i = torch.nonzero(m.amax(dim=tuple(b for b in range(3) if b != a)))[:, 0]
        out.append(slice(max(0, int(i[0]) - margin), min(m.shape[a], int(i[-1]) + 1 + margin)))
    return tuple(out)


def _pd64(f_in, mask, h, lam, alpha, iters, tgv):
    """pd_tgv_mex / pd_tv_mex (tol 0) in FP64 on the mask's box."""
    box = _box(mask, 2)
    f0 = f_in.to(F64)[box]
    m = (mask[box] != 0).to(F64)
    core = (slice(1, -1),) * 3
    hx, hy, hz = h
    ih = (1 / hx ** 2, 1 / hy ** 2, 1 / hz ** 2)
    K2 = (4 * sum(ih)) ** 2 + (6 * (ih[0] + ih[1] + 2 * ih[2]) / 3) ** 2
    tau = 1 / math.sqrt(K2)
    sg = 1 / (tau * K2)
    mi = torch.zeros_like(m)
    mi[core] = m[2:, 1:-1, 1:-1] * m[:-2, 1:-1, 1:-1] * m[1:-1, 2:, 1:-1] * m[1:-1, :-2, 1:-1] * \
        m[1:-1, 1:-1, 2:] * m[1:-1, 1:-1, :-2]
    mc, mic = m[core], mi[core]

    def sl(v, ax, k):
        i = list(core)
        i[ax] = slice(2, None) if k > 0 else slice(0, -2)
        return v[tuple(i)]

    AX = (2, 1, 0)
    lw = ih
    ww = (-ih[0] / 3, -ih[1] / 3, 2 * ih[2] / 3)

    def sten(v, w):
        return -2 * sum(w) * v[core] + sum(w[a] * (sl(v, AX[a], -1) + sl(v, AX[a], 1)) for a in range(3))

    def d(v, a):  # forward difference of axis a (x, y, z)
        return sl(v, AX[a], 1) - v[core]

    def b(v, a):  # backward difference
        return v[core] - sl(v, AX[a], -1)

    Z = lambda: torch.zeros_like(f0)  # noqa: E731
    f = (sg * f0)[core]
    chi, eta, chib, etab, nu = Z(), Z(), Z(), Z(), Z()
    p = [Z() for _ in range(3)]
    nw = 3 if tgv else 0
    w, wb, qq = [Z() for _ in range(nw)], [Z() for _ in range(nw)], [Z() for _ in range(2 * nw)]
    a1, a0 = lam, alpha * lam
    for _ in range(iters):
        nu[core] += mic * (sg * (sten(etab, lw) - sten(chib, ww)) + f)
        g = []
        for a in range(3):
            t = p[a][core] + sg / h[a] * d(chib, a)
            g.append(t - sg * wb[a][core] if tgv else t)
        s = a1 / torch.sqrt(g[0] ** 2 + g[1] ** 2 + g[2] ** 2).clamp_min(a1)
        for a in range(3):
            p[a][core] = mic * g[a] * s
        if tgv:
            e = [qq[0][core] + sg / hx * d(wb[0], 0),
                 qq[1][core] + 0.5 * sg * (d(wb[1], 0) / hx + d(wb[0], 1) / hy),
                 qq[2][core] + 0.5 * sg * (d(wb[2], 0) / hx + d(wb[0], 2) / hz),
                 qq[3][core] + sg / hy * d(wb[1], 1),
                 qq[4][core] + 0.5 * sg * (d(wb[2], 1) / hy + d(wb[1], 2) / hz),
                 qq[5][core] + sg / hz * d(wb[2], 2)]
            s = e[0] ** 2 + e[3] ** 2 + e[5] ** 2 + 2 * (e[1] ** 2 + e[2] ** 2 + e[4] ** 2)
            s = a0 / torch.sqrt(s).clamp_min(a0)
            for a in range(6):
                qq[a][core] = mic * e[a] * s
        e1 = (eta[core] - tau * sten(nu, lw)) / (1 + tau)
        c1 = chi[core] + tau * sum(b(p[a], a) / h[a] for a in range(3)) + tau * sten(nu, ww)
        upd = [(eta, etab, e1), (chi, chib, c1)]
        if tgv:
            rows = ((0, 1, 2), (1, 3, 4), (2, 4, 5))
            for a in range(3):
                # one voxel size per component, as the reference has it
                div = sum(b(qq[rows[a][k]], k) for k in range(3)) / h[a]
                upd.append((w[a], wb[a], w[a][core] + tau * (p[a][core] + div)))
        for old, bar, new in upd:
            new = mc * new
            bar[core] = 2 * new - old[core]
            old[core] = new
    out = torch.zeros(f_in.shape, dtype=F64, device=f_in.device)
    out[box] = chi
    return out


def _solve64(f, mask, h):
    """v with -Laplacian(v) = f inside the mask and v = 0 outside: conjugate gradients."""
    box = _box(mask, 2)
    m = (mask[box] != 0).to(F64)
    m[0], m[-1], m[:, 0], m[:, -1], m[:, :, 0], m[:, :, -1] = 0, 0, 0, 0, 0, 0
    r = f.to(F64)[box] * m
    x, p = torch.zeros_like(r), r.clone()
    rho = torch.sum(r * r)
    stop = float(rho) * 1e-26
    for it in range(4000):
        ap = -_lap7(p, h) * m
        a = rho / torch.sum(p * ap)
        x = x + a * p
        r = r - a * ap
        new = torch.sum(r * r)
        p = r + (new / rho) * p
        rho = new
        if it % 25 == 24 and float(rho) <= stop:
            break
    out = torch.zeros(f.shape, dtype=F64, device=f.device)
    out[box] = x
    return out


def _next_fast(n):
    while True:
        k = n
        for p in (2, 3, 5, 7):
            while k % p == 0:
                k //= p
        if k == 1:
            return n
        n += 1


def _vsharp64(f, mask, h):
    """vsharp.m with its default radii: the local field (the eroded mask is None here: it is compared as it is)."""
    hm = max(h)
    rs = [r for r in np.arange(9.0, 2 * hm - 1e-12, -2 * hm) if r >= 2 * hm]
    pad = int(math.ceil(max(rs) / min(h)))
    box = _box(mask, 0)
    sz = [b.stop - b.start for b in box]
    full = [_next_fast(s + 2 * pad) for s in sz]
    pre = [(t - s) // 2 + ((t - s) & 1 & s) for s, t in zip(sz, full)]
    inner = tuple(slice(p, p + s) for p, s in zip(pre, sz))

    def grow(v):
        o = torch.zeros(full, dtype=F64, device=v.device)
        o[inner] = v.to(F64)[box]
        return o

    def spectrum(r):
        g = []
        for a, (n, d) in enumerate(zip(full, (h[2], h[1], h[0]))):
            x = torch.fft.fftfreq(n, d=1.0 / n, dtype=F64, device=f.device) * d
            g.append(x.reshape([-1 if a == b else 1 for b in range(3)]))
        k = (g[0] ** 2 + g[1] ** 2 + g[2] ** 2 <= r * r).to(F64)
        return torch.fft.fftn(k / k.sum()).real

    M = torch.fft.fftn(grow(mask != 0))
    H = [spectrum(r) for r in rs]
    masks = [(torch.fft.ifftn(s * M).real > 0.999).to(F64) for s in H]
    ih = 1.0 / (1.0 - H[0])
    ih[(1.0 - H[0]).abs() < 0.05] = 0.0
    out = torch.zeros(f.shape, dtype=F64, device=f.device)
    for t in range(1 if f.dim() == 3 else f.shape[0]):
        F = torch.fft.fftn(grow(f if f.dim() == 3 else f[t]))
        acc, prev = 0.0, 0.0
        for s, mk in zip(H, masks):
            acc = acc + (mk - prev) * torch.fft.ifftn((1.0 - s) * F).real
            prev = mk
        u = masks[-1] * torch.fft.ifftn(ih * torch.fft.fftn(acc)).real
        (out if f.dim() == 3 else out[t])[box] = u[inner]
    return out


def _admm64(f, mask, h, iters, tv):
    """tv.m's ADMM loop with rtol = atol = 0 and its other defaults."""
    f = f.to(F64)
    mu, rho, alpha, rtau, stau, gamma = 7.5e3, 9.0, 1.5, 0.7, 1e2, 3.0
    D = _dipole(f.shape, h)
    L = 0.0
    for k, d in zip(_freq2(f.shape, h), (h[2], h[1], h[0])):
        L = L + (2.0 - 2.0 * torch.cos(2 * PI * k * d)) / (d * d)
    L[0, 0, 0] = 0.0
    F = mu * D * torch.fft.fftn(f)

    def inverse(r):
        A = mu * D * D + r * L
        A[0, 0, 0] = math.inf
        return 1.0 / A

    def grad(u):
        return [(torch.roll(u, -1, a) - u) / d for a, d in ((2, h[0]), (1, h[1]), (0, h[2]))]

    def adj(v):
        return sum((torch.roll(x, 1, a) - x) / d for x, (a, d) in zip(v, ((2, h[0]), (1, h[1]), (0, h[2]))))

    def size(v):
        return float(torch.sqrt(v[0] ** 2 + v[1] ** 2 + v[2] ** 2).sum())

    u, iA = f, inverse(rho)
    ls = [torch.zeros_like(f) for _ in range(3)]
    vs = grad(u)
    nr, flag = size(vs), 0
    for _ in range(iters):
        u = torch.fft.ifftn(iA * (F + torch.fft.fftn(adj([rho * v - l for v, l in zip(vs, ls)])))).real
        old, g = vs, grad(u)
        mix = [alpha * d + (1 - alpha) * v for d, v in zip(g, old)]
        r = [x + l / rho for x, l in zip(mix, ls)]
        if tv == 1:
            vs = [torch.sign(x) * (x.abs() - 1 / rho).clamp_min(0.0) for x in r]
        else:
            s = torch.sqrt(r[0] ** 2 + r[1] ** 2 + r[2] ** 2)
            s = torch.where(s > 1 / rho, (s - 1 / rho) / s, torch.zeros_like(s))
            vs = [x * s for x in r]
        ls = [l + rho * (x - v) for l, x, v in zip(ls, mix, vs)]
        before, nr = nr, size([d - v for d, v in zip(g, vs)])
        ns = float((rho * adj([v - o for v, o in zip(vs, old)])).norm())
        if nr > stau * ns or (nr > rtau * before and flag < 3):
            rho, flag = gamma * rho, 0 if flag > 5 else flag
            iA = inverse(rho)
        elif nr < ns / stau:
            rho, flag = rho / gamma ** 2, flag + 1
            iA = inverse(rho)
    return mask.to(F64) * u


def exact(case, seed):
    kind, h = case["kind"], _h(case)
    s = _inputs(case, seed)
    if kind == "fd":
        return _fd64(case, s)
    if kind == "tgv":
        return _pd64(s["f"], s["m"], h, 0.003, 2.0, case["iters"], True)
    if kind == "tv_batch":
        return [_pd64(f, m, h, 1e-3, 0.0, case["iters"], False) for f, m in zip(s["fs"], s["ms"])]
    if kind == "mgpcg":
        return _solve64(s["f"], s["m"], h)
    if kind == "lbv":
        echoes = [s["f"]] if case["echoes"] == 1 else list(s["f"])
        out = [_solve64(-_lap1_64(f.to(F64), s["m"] != 0, h), s["m"], h) for f in echoes]
        return out[0] if case["echoes"] == 1 else torch.stack(out)
    if kind == "vsharp":
        return [_vsharp64(s["f"], s["m"], h), None]
    if kind == "tv_admm":
        return _admm64(s["f"], s["m"], h, case["iters"], case["tv"])
    raw = s["raw"].to(F64)
    if case["stored"] == "uint16":
        raw = torch.where(raw < 0, raw + 65536.0, raw)
    img = (raw * s["slope"] + s["inter"]).reshape(case["echoes"], case["nz"], case["ny"], case["nx"])
    if case["echoes"] == 1:
        img = img[0]
    # loaded axis i (x, y, z) is the stored axis of row i's entry, reversed where that is -1
    e = img.dim() - 3
    order, flips = [], []
    for i, row in enumerate(_SFORM[case["orient"]]):
        j = next(k for k in range(3) if row[k])
        order.append(e + 2 - j)
        if row[j] < 0:
            flips.append(e + 2 - i)
    img = img.permute(*range(e), *reversed(order))
    return torch.flip(img, flips).contiguous() if flips else img.contiguous()
