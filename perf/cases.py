"""The work that users of this framework have it do, as cases to be timed.

A case is a call of the public Python mirror of the C ABI (``Context``,
``Group``): a few SCF iterations of ``converge`` (residual read back after
each, the free energy at the end), iterations of a sweep, the stress, the
adjoint, an Anderson update.  Fields are synthetic (no data set exists for this path):
ordered-phase patterns plus noise, as in the benchmark and the tests.

Result types.  FP64 and double-float contexts give 64-bit results.  An FP32
context keeps its fields in FP64 containers, but they carry single-precision
propagation, so a program that runs in FP32 takes them as float32 tensors
(converted on the context's own stream); that is what ``run`` returns there.
"""
from __future__ import annotations

import ctypes
import math

import numpy as np
import torch

from __graft_entry__ import load_package

pkg = load_package()

PREC = {"fp64": pkg.PREC_FP64, "fp32": pkg.PREC_FP32, "df": pkg.PREC_DF}
PI_REF = 3.1415926535            # the reference's value in the wave numbers
WOPT, WCMP = 0.05, 0.10          # the reference's simple-mixing constants
ANDERSON_LAMBDA = 0.5
SWEEP_ITS = 2


def scf(name, grid, box, prec, ds, f, chi, phase, batch=1, its=4):
    c = {"kind": "scf", "its": its, "nx": grid[0], "ny": grid[1], "nz": grid[2], "lx": box[0], "ly": box[1],
         "lz": box[2], "prec": prec, "ds": ds, "f": f, "chi": chi, "phase": phase,
         "batch": batch}
    return dict(c, name=name) if name else c


def listed():
    hexbox = (4.2, 4.2 * math.sqrt(3.0), 2.0)
    return [
        # a thin 2-D film, the quickest phase scans: launches and latency
        scf("film_64x64_fp64", (64, 64, 1), (4.0, 4.0, 1.0), "fp64", 0.01, 0.5, 20.0, "lamellar"),
        # the lamellar validation run at the reference's own precision
        scf("lamellar_32_fp64", (32, 32, 32), (4.0, 4.0, 4.0), "fp64", 0.01, 0.5, 20.0, "lamellar"),
        # the double-gyroid candidate at the reference's own precision
        scf("gyroid_64_fp64", (64, 64, 64), (3.8, 3.8, 3.8), "fp64", 0.005, 0.36, 18.0, "gyroid"),
        # the same in mixed precision: the bulk of a production solve
        scf("gyroid_64_fp32", (64, 64, 64), (3.8, 3.8, 3.8), "fp32", 0.005, 0.36, 18.0, "gyroid"),
        # the headline benchmark
        scf("gyroid_128_fp32", (128, 128, 128), (3.8, 3.8, 3.8), "fp32", 0.005, 0.36, 18.0,
            "gyroid"),
        # the double-float polish that ends a mixed-precision solve
        scf("gyroid_64_df", (64, 64, 64), (3.8, 3.8, 3.8), "df", 0.005, 0.36, 18.0, "gyroid"),
        # an orthorhombic box meshed at equal spacing: sizes with factors 3 and 5
        scf("ortho_100x80x60_fp32", (100, 80, 60), (5.0, 4.0, 3.0), "fp32", 0.005, 0.4, 20.0,
            "gyroid"),
        # the large single solve (200 contour steps: with 400 the single-precision
        # rounding of the densities grows to about 2e-5)
        scf("mixture_256_fp32", (256, 256, 256), (8.0, 8.0, 8.0), "fp32", 0.005, 0.45, 22.0,
            "mixture", its=1),
        # a phase-diagram sweep: instances of uneven grids and parameters, one group
        {"name": "sweep_16_fp32", "kind": "sweep", "n32": 6, "n48": 5, "n64": 5, "prec": "fp32"},
        # the box stress that drives a unit-cell relaxation, at 64-bit level
        {"name": "hexagonal_stress_df", "kind": "stress", "nx": 128, "ny": 128, "nz": 64,
         "lx": hexbox[0], "ly": hexbox[1], "lz": hexbox[2], "prec": "df", "ds": 0.005, "f": 0.3,
         "chi": 25.0, "phase": "hexagonal", "batch": 1},
        # the gradient of a function of the densities with respect to the fields
        {"name": "gyroid_adjoint_fp32", "kind": "adjoint", "nx": 64, "ny": 64, "nz": 64, "lx": 3.8,
         "ly": 3.8, "lz": 3.8, "prec": "fp32", "ds": 0.005, "f": 0.36, "chi": 18.0,
         "phase": "gyroid", "batch": 1},
        # the Anderson field update with a full history
        {"name": "anderson_128", "kind": "anderson", "nx": 128, "ny": 128, "nz": 128, "hist": 20,
         "chi": 18.0, "batch": 1},
    ]


# -- drawn cases --------------------------------------------------------------

def _sizes(lo, hi, primes=(2, 3, 5, 7)):
    def smooth(n):
        for p in primes:
            while n % p == 0:
                n //= p
        return n == 1
    return [n for n in range(lo, hi + 1, 2) if smooth(n)]


def _axis(rng, lo, hi):
    """An axis length: half the time one of the usual meshes, else any even
    number with small factors, spread over the logarithm of the range."""
    usual = [n for n in (16, 32, 48, 64, 96, 128, 192) if lo <= n <= hi]
    if rng.random() < 0.5:
        return rng.choice(usual)
    target = math.exp(rng.uniform(math.log(lo), math.log(hi)))
    return min(_sizes(lo, hi), key=lambda n: abs(n - target))


def draw(rng):
    kind = rng.choice(["scf", "scf", "scf", "scf", "scf", "sweep", "stress", "adjoint",
                       "anderson"])
    chi, f = round(rng.uniform(12.0, 30.0), 3), round(rng.uniform(0.25, 0.5), 3)
    ds = 1.0 / rng.choice([100, 120, 150, 160, 200])
    if kind == "sweep":
        return {"kind": kind, "n32": rng.randint(2, 8), "n48": rng.randint(1, 5),
                "n64": rng.randint(1, 3), "prec": "fp32"}
    if kind == "anderson":
        n = [_axis(rng, 16, 128) for _ in range(3)]
        return {"kind": kind, "nx": n[0], "ny": n[1], "nz": n[2], "hist": rng.randint(4, 30),
                "chi": chi, "batch": 1}
    prec = rng.choice(["fp32", "fp32", "fp64", "df"] if kind == "scf" else ["fp64", "df"]
                      if kind == "stress" else ["fp32", "fp64"])
    if prec == "df":                 # double-float contexts take these axes only
        n = [rng.choice([32, 64, 128]) for _ in range(3)]
    else:
        lo, hi = (16, 192) if prec == "fp32" and kind == "scf" else (16, 72)
        n = [_axis(rng, lo, hi) for _ in range(3)]
        if kind == "scf" and rng.random() < 0.15:
            n[2] = 1                 # a film
    h = rng.uniform(0.03, 0.12)      # mesh spacing in Rg
    box = [round(min(9.0, max(1.0, m * h)), 4) for m in n]
    batch = rng.choice([1, 1, 1, 2, 4]) if n[0] * n[1] * n[2] <= 1 << 17 else 1
    c = scf("", n, box, prec, ds, f, chi, rng.choice(["lamellar", "gyroid", "hexagonal"]), batch)
    if kind != "scf":
        del c["its"]
    c["kind"] = kind
    return c


# -- inputs -------------------------------------------------------------------

def _device():
    return torch.device("cuda" if torch.cuda.is_available() else "cpu")


def _gen(seed):
    return torch.Generator(device=_device()).manual_seed(int(seed))


def _pattern(case):
    """The ordered phase's level-set function on the mesh, [nz, ny, nx]."""
    dev, dt = _device(), torch.float64
    ax = lambda n: 2 * math.pi * torch.arange(n, device=dev, dtype=dt) / n
    X = ax(case["nx"])[None, None, :]
    Y = ax(case["ny"])[None, :, None]
    Z = ax(case["nz"])[:, None, None]
    g = X.sin() * Y.cos() + Y.sin() * Z.cos() + Z.sin() * X.cos()
    phase = case.get("phase", "gyroid")
    if phase == "lamellar":
        g = X.cos() + 0 * g
    elif phase == "hexagonal":
        g = -((2 * Y).cos() + (X + Y).cos() + (X - Y).cos()) / 3 + 0 * g
    elif phase == "mixture":
        g = 0.5 * (X.cos() + g)
    return g


def _fields(case, seed):
    """wA, wB: +-chi*0.2*pattern plus N(0, 0.02) noise, [batch, nz, ny, nx]."""
    g = _pattern(case) * (0.2 * case["chi"])
    r = torch.randn((2, case["batch"]) + tuple(g.shape), generator=_gen(seed), device=_device(),
                    dtype=torch.float64) * 0.02
    return g + r[0], -g + r[1]


def _context(case, **kw):
    return pkg.Context(nx=case["nx"], ny=case["ny"], nz=case["nz"], lx=case["lx"], ly=case["ly"],
                       lz=case["lz"], hAB=case["chi"], fA=case["f"], ds0=case["ds"],
                       batch=case["batch"], precision=PREC[case["prec"]], wopt=WOPT, wcmp=WCMP,
                       **kw)


def _views(ctx, w, fields):
    """Puts wA, wB into the context; torch views of its fields, and its stream."""
    ctx.field_view(pkg.FIELD_WA).copy_(w[0])
    ctx.field_view(pkg.FIELD_WB).copy_(w[1])
    p = ctypes.c_void_p()
    ctx.lib.scft_get_stream(ctx.h, ctypes.byref(p))
    torch.cuda.synchronize()
    views = [ctx.field_view(f) for f in fields]
    for v in views:
        v.owner = ctx                # the memory behind a view is the context's
    return views, torch.cuda.ExternalStream(p.value)


ALL_FIELDS = (pkg.FIELD_WA, pkg.FIELD_WB, pkg.FIELD_PHA, pkg.FIELD_PHB)


def _members(case):
    """The sweep's instances: grids and parameters fixed by the case."""
    out = []
    grids = [32] * case["n32"] + [48] * case["n48"] + [64] * case["n64"]
    for i, n in enumerate(grids):
        u = [math.modf((i + 1) * a)[0] for a in (0.618034, 0.414214, 0.732051, 0.236068)]
        L = round(3.0 + 2.0 * u[0], 4)
        out.append({"nx": n, "ny": n, "nz": n, "lx": L, "ly": L, "lz": L, "prec": case["prec"],
                    "ds": 1.0 / int(100 + 100 * u[1]), "f": round(0.25 + 0.25 * u[2], 4),
                    "chi": round(12 + 18 * u[3], 4), "phase": ("gyroid", "lamellar")[i % 2],
                    "batch": 1})
    return out


def _anderson_inputs(case, seed):
    """Start fields and hist+1 density pairs, as a solve in progress has them."""
    c = dict(case, phase="gyroid")
    w = _fields(c, seed)
    g = _pattern(c)
    gen, shape = _gen(seed + 1), w[0].shape

    def densities():
        r = torch.randn((2,) + tuple(shape), generator=gen, device=_device(), dtype=torch.float64)
        return 0.4 - 0.2 * g + 0.05 * r[0], 0.6 + 0.2 * g + 0.05 * r[1]
    return w, densities


def prepare(case, seed):
    kind = case["kind"]
    if kind == "sweep":
        ctxs, views, streams = [], [], []
        for i, m in enumerate(_members(case)):
            ctx = _context(m)
            v, s = _views(ctx, _fields(m, seed * 64 + i), ALL_FIELDS)
            ctxs.append(ctx)
            views.append(v)
            streams.append(s)
        return {"kind": kind, "ctxs": ctxs, "group": pkg.Group(ctxs), "views": views,
                "streams": streams}
    if kind == "anderson":
        w, densities = _anderson_inputs(case, seed)
        ctx = pkg.Context(nx=case["nx"], ny=case["ny"], nz=case["nz"], hAB=case["chi"],
                          batch=case["batch"], ds0=0.5, precision=pkg.PREC_FP32,
                          mixing=pkg.MIX_ANDERSON, anderson_history=case["hist"], wopt=WOPT,
                          wcmp=WCMP, anderson_lambda=ANDERSON_LAMBDA, anderson_start=1e9)
        (wa, wb, pa, pb), s = _views(ctx, w, ALL_FIELDS)
        for k in range(case["hist"] + 1):
            a, b = densities()
            pa.copy_(a)
            pb.copy_(b)
            torch.cuda.synchronize()
            if k < case["hist"]:
                ctx.phi_w()
                ctx.synchronize()
        return {"kind": kind, "ctx": ctx, "views": [wa, wb]}
    ctx = _context(case)
    st = {"kind": kind, "ctx": ctx, "f32": case["prec"] == "fp32", "its": case.get("its", 1)}
    st["views"], st["stream"] = _views(ctx, _fields(case, seed),
                                       ALL_FIELDS if kind != "stress" else ALL_FIELDS[2:])
    if kind == "adjoint":
        r = torch.randn((2,) + ctx.shape, generator=_gen(seed + 1), device=_device(),
                        dtype=torch.float64)
        st["bars"] = (r[0].cpu().numpy(), r[1].cpu().numpy())
        st["qbar"] = np.full(case["batch"], 0.5)
    return st


# -- one pass -----------------------------------------------------------------

def _f32(views, stream):
    with torch.cuda.stream(stream):
        return [v.float() for v in views]


def run(st):
    kind = st["kind"]
    if kind == "scf":                # SCF iterations of a solve that goes on
        _, fe = st["ctx"].converge(1e-300, st["its"])
        if st["f32"]:
            return _f32(st["views"], st["stream"]) + [fe.astype(np.float32)]
        return st["views"] + [fe]
    if kind == "sweep":              # iterations of every instance
        st["group"].iterate(SWEEP_ITS)
        return [_f32(v, s) for v, s in zip(st["views"], st["streams"])]
    if kind == "stress":             # densities and box stress at the present fields
        st["ctx"].get_conc()
        return [st["ctx"].stress(), *st["views"]]
    if kind == "adjoint":            # d(function of the densities and Q)/d(wA, wB)
        a, b, _ = st["ctx"].adjoint(*st["bars"], st["qbar"], want_L=False)
        return [a.astype(np.float32), b.astype(np.float32)] if st["f32"] else [a, b]
    st["ctx"].phi_w()                # anderson: the field update alone
    return st["views"]


# -- what a pass cannot do without --------------------------------------------

def _steps(c):
    return int(c["f"] / c["ds"] + 1e-8), int((1 - c["f"]) / c["ds"] + 1e-8)


def _march_flops(c):
    """Two chains of Ns split steps: a real transform and its inverse (2.5 M
    log2 M each), the gain and the two Boltzmann factors."""
    M = c["nx"] * c["ny"] * c["nz"]
    return (c.get("its", 1) * 2.0 * sum(_steps(c)) * c["batch"] * M * (5.0 * math.log2(M) + 3.0))


def work(case):
    kind = case["kind"]
    if kind == "sweep":
        each = [work(dict(m, kind="scf", its=SWEEP_ITS)) for m in _members(case)]
        return {k: sum(w[k] for w in each) for k in ("bytes", "flops")}
    pts = case["nx"] * case["ny"] * case["nz"] * case["batch"]
    if kind == "anderson":           # w and phi in, the history's u and d pairs, the new slot, w out
        h = case["hist"]
        return {"bytes": pts * (32.0 + 32.0 * h + 32.0 + 16.0), "flops": pts * 8.0 * (h + 1)}
    if kind == "scf":                # wA, wB in; wA, wB, phiA, phiB out
        return {"bytes": 48.0 * pts, "flops": _march_flops(case)}
    if kind == "stress":             # the march, then every stored step's spectrum once more
        return {"bytes": 32.0 * pts, "flops": 1.5 * _march_flops(case)}
    # adjoint: the march, and the reverse sweeps of both chains
    return {"bytes": 48.0 * pts, "flops": 2.0 * _march_flops(case)}


# -- the same in 64 bits with plain torch -------------------------------------

def _k2(n, L):
    i = torch.arange(n, device=_device(), dtype=torch.float64)
    i = torch.where(i <= n // 2 - 1, i, i - n)
    return (2 * PI_REF * i / L) ** 2


class _Exact:
    """getConc and its surroundings by real FFTs in float64."""

    def __init__(self, c, box=None):
        self.c = c
        L = box if box is not None else [c["lx"], c["ly"], c["lz"]]
        kx = _k2(c["nx"], L[0])[: c["nx"] // 2 + 1]
        ky, kz = _k2(c["ny"], L[1]), _k2(c["nz"], L[2])
        self.G = torch.exp(-c["ds"] * (kx[None, None, :] + ky[None, :, None] + kz[:, None, None]))
        self.shape = (c["nz"], c["ny"], c["nx"])
        self.nA, self.nB = _steps(c)

    def filt(self, x):
        d = (-3, -2, -1)
        return torch.fft.irfftn(torch.fft.rfftn(x, dim=d) * self.G, s=self.shape, dim=d)

    def conc(self, wa, wb, keep=False):
        """phiA, phiB, Q of one instance (wa mean-free already)."""
        WA, WB = torch.exp(-wa * self.c["ds"] / 2), torch.exp(-wb * self.c["ds"] / 2)
        N = self.nA + self.nB
        qc = [None] * (N + 1)        # q+(s), from the far end
        qc[N] = torch.ones_like(wa)
        for s in range(N, 0, -1):
            W = WA if s <= self.nA else WB
            qc[s - 1] = W * self.filt(W * qc[s])
        q, qs = torch.ones_like(wa), []
        pa = 0.5 * q * qc[0]
        pb = torch.zeros_like(wa)
        for s in range(1, N + 1):
            if keep:
                qs.append(q)
            W = WA if s <= self.nA else WB
            q = W * self.filt(W * q)
            if s <= self.nA:
                pa = pa + (0.5 if s == self.nA else 1.0) * q * qc[s]
            if s >= self.nA:
                pb = pb + (0.5 if s in (self.nA, N) else 1.0) * q * qc[s]
            if not keep:
                qc[s - 1] = None
        Q = q.mean()
        out = pa * (self.c["ds"] / Q), pb * (self.c["ds"] / Q), Q
        return (out, qs, qc, (WA, WB)) if keep else out


def _phi_w(wa, wb, pa, pb, chi):
    eta, ps = (wa + wb - chi) / 2, 1.0 - pa - pb
    return chi * pb + eta - wa - WCMP * ps, chi * pa + eta - wb - WCMP * ps


def _exact_scf(c, seed):
    wa, wb = _fields(c, seed)
    ex, outs = _Exact(c), []
    for b in range(c["batch"]):
        a, d = wa[b], wb[b]
        for _ in range(c["its"]):
            a, d = a - a.mean(), d - d.mean()
            a = a - a.mean()
            pa, pb, Q = ex.conc(a, d)
            ra, rb = _phi_w(a, d, pa, pb, c["chi"])
            a, d = a + WOPT * ra, d + WOPT * rb
        fab, fw = (c["chi"] * pa * pb).mean(), -(a * pa + d * pb).mean()
        fe = torch.stack([fab + fw - Q.log(), fab, fw, -Q.log(), (1 - pa - pb).abs().max()])
        outs.append((a, d, pa, pb, fe))
    return [torch.stack(v) for v in zip(*outs)]


def _exact_stress(c, seed):
    wa, wb = _fields(c, seed)
    ex = _Exact(c)
    L, n = [c["lx"], c["ly"], c["lz"]], [c["nx"], c["ny"], c["nz"]]
    k2 = [_k2(n[a], L[a]) for a in range(3)]
    k2[0] = k2[0][: n[0] // 2 + 1]
    shape = [(1, 1, -1), (1, -1, 1), (-1, 1, 1)]
    M, d, outs = n[0] * n[1] * n[2], (-3, -2, -1), []
    # every mode but kx = 0 and kx = Nyquist stands for itself and its conjugate
    mult = torch.full((n[0] // 2 + 1,), 2.0, device=_device(), dtype=torch.float64)
    mult[0] = mult[-1] = 1.0
    for b in range(c["batch"]):
        (pa, pb, Q), qs, qc, W = ex.conc(wa[b] - wa[b].mean(), wb[b], keep=True)
        sig = torch.zeros(3, device=_device(), dtype=torch.float64)
        for s in range(1, ex.nA + ex.nB + 1):
            w = W[0] if s <= ex.nA else W[1]
            X = torch.fft.rfftn(w * qs[s - 1], dim=d)
            Y = torch.fft.rfftn(w * qc[s], dim=d)
            P = (X * Y.conj()).real * ex.G * mult / M
            for a in range(3):
                sig[a] += (P * (2 * c["ds"] * k2[a] / L[a]).reshape(shape[a])).sum()
        outs.append((-sig / (M * Q), pa, pb))
    return [torch.stack(v) for v in zip(*outs)]


def _exact_adjoint(c, seed):
    wa, wb = _fields(c, seed)
    r = torch.randn((2,) + tuple(wa.shape), generator=_gen(seed + 1), device=_device(),
                    dtype=torch.float64)
    ex, outs = _Exact(c), []
    for b in range(c["batch"]):
        a, d = wa[b].clone().requires_grad_(True), wb[b].clone().requires_grad_(True)
        (pa, pb, Q), *_ = ex.conc(a - a.mean(), d, keep=True)
        y = (r[0, b] * pa).sum() + (r[1, b] * pb).sum() + 0.5 * Q
        outs.append(torch.autograd.grad(y, (a, d)))
    return [torch.stack(v) for v in zip(*outs)]


def _exact_anderson(c, seed):
    (wa, wb), densities = _anderson_inputs(c, seed)
    w, us, ds = torch.stack([wa, wb], 1), [], []
    for _ in range(c["hist"] + 1):
        pa, pb = densities()
        d = torch.stack(_phi_w(w[:, 0], w[:, 1], pa, pb, c["chi"]), 1)
        d = d - d.mean(dim=(-3, -2, -1), keepdim=True)
        us.insert(0, w + ANDERSON_LAMBDA * d)
        ds.insert(0, d)
        if len(ds) == 1:
            w = w + WOPT * d
            continue
        new = []
        for b in range(c["batch"]):
            D = torch.stack([x[b].reshape(-1) for x in ds])
            G = D @ D.T
            U = G[0, 0] - G[0, 1:, None] - G[0, None, 1:] + G[1:, 1:]
            U = U + torch.eye(len(U), device=U.device, dtype=U.dtype) * 1e-12 * U.diagonal().max()
            x = torch.linalg.solve(U, G[0, 0] - G[0, 1:])
            a = torch.cat([1 - x.sum().reshape(1), x])
            new.append(sum(a[k] * us[k][b] for k in range(len(us))))
        w = torch.stack(new)
    return [w[:, 0].contiguous(), w[:, 1].contiguous()]


def exact(case, seed):
    kind = case["kind"]
    if kind == "sweep":
        return [_exact_scf(dict(m, its=SWEEP_ITS), seed * 64 + i)[:4]
                for i, m in enumerate(_members(case))]
    return {"scf": _exact_scf, "stress": _exact_stress, "adjoint": _exact_adjoint,
            "anderson": _exact_anderson}[kind](case, seed)
