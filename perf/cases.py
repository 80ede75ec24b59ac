"""The work that users of medusa_b200 have it do, as cases that can be timed and compared.

A pass is what a program does with the library between two looks at its state: the state
goes to the device, a number of RK2 steps is taken, the state comes back (the tabulated
EOS update is one call on device arrays).  Kinds of case:

  embed     mdg_advance_1d_noalloc: one 1-D problem on device arrays of the caller's, a
            handful of steps (a sub-cycle inside another code): latency and launches;
  tube      Solver, one 1-D Cartesian problem in plain FP64 (the Sod tube job);
  ensemble  run_host over uneven 1-D spherical Sod/Noh/Sedov problems, plain FP64 or mixed;
  shear     Solver, 2-D periodic Kelvin-Helmholtz box, plain FP64 or mixed;
  rt        Solver, 2-D Rayleigh-Taylor with fixed gravity (periodic/reflecting), odd sizes;
  blast     Solver, Sedov blast on the dendritic spherical grid, 3-D or 2-D (r, theta);
  eos       EosTable.given_rex_device: the tabulated EOS zone update.

Initial states are the problem setups' with a seeded perturbation of density and velocity,
in page-locked host memory; grids and solvers are kept, as a program keeps them.
"""
import ctypes
import dataclasses
import functools
import math

import numpy as np
import torch

import medusa_b200 as mb
from medusa_b200 import eos_table as ET
from medusa_b200 import problems as P
from medusa_b200.solver import desc_of, run_host

KINDS_1D = ("sod", "noh", "sedov")
GAMMAS = (4.0 / 3.0, 1.4, 5.0 / 3.0)
NOISE = 0.01          # relative density noise of the perturbed initial states


def listed():
    return [
        # a host code's sub-cycle: 20 steps of a small shell problem on its own device arrays
        dict(name="embed_200", kind="embed", n1=200, steps=20),
        # the Sod tube of the drop-in tests and the bench, a stretch of its 572 steps
        dict(name="tube_1024_fp64", kind="tube", n1=1024, steps=100),
        # a parameter study in plain FP64: uneven problems in one batch
        dict(name="ens_400_fp64", kind="ensemble", prec="fp64", count=400, nmin=128, nmax=8192, parts=1, steps=40),
        # a small study in mixed precision: few, small, odd-sized problems
        dict(name="ens_24_mixed", kind="ensemble", prec="mixed", count=24, nmin=101, nmax=1501, parts=1, steps=40),
        # the headline ensemble, in four solvers whose copies overlap each other's steps
        dict(name="ens_2048_mixed", kind="ensemble", prec="mixed", count=2048, nmin=128, nmax=8192, parts=4, steps=40),
        # 2-D shear layer, an ordinary box in plain FP64 and the full-size one in mixed precision
        dict(name="shear_512_fp64", kind="shear", prec="fp64", n1=512, n2=512, steps=40),
        dict(name="shear_2048_mixed", kind="shear", prec="mixed", n1=2048, n2=2048, steps=20),
        # 2-D with gravity and reflecting walls on sizes that no tile divides
        dict(name="rt_187x411_fp64", kind="rt", prec="fp64", n1=187, n2=411, steps=60),
        # axisymmetric blast on the (r, theta) grid, mixed precision
        dict(name="blast2d_400x256_mixed", kind="blast", prec="mixed", ndim=2, n1=400, n2=256, n3=1, radius="uniform",
             steps=60),
        # the solve server's 3-D request size in plain FP64, and the full-size 3-D grid (radius
        # log-spaced from 1e-3) in mixed precision
        dict(name="blast3d_128_fp64", kind="blast", prec="fp64", ndim=3, n1=128, n2=64, n3=128, radius="uniform",
             steps=20),
        dict(name="blast3d_384_mixed", kind="blast", prec="mixed", ndim=3, n1=384, n2=128, n3=256, radius="sinh",
             steps=10),
        # EOS update of a large 3-D domain's zones at the reference table's size
        dict(name="eos_4m", kind="eos", zones=4194304),
    ]


def _log_int(rng, a, b):
    return int(round(math.exp(rng.uniform(math.log(a), math.log(b)))))


def draw(rng):
    kind = rng.choice(("embed", "tube", "ensemble", "ensemble", "shear", "shear", "rt", "blast", "blast", "eos"))
    prec = rng.choice(("fp64", "mixed"))
    if kind == "embed":
        return dict(kind=kind, n1=_log_int(rng, 64, 4096), steps=rng.randint(5, 40))
    if kind == "tube":
        return dict(kind=kind, n1=_log_int(rng, 96, 8192), steps=rng.randint(20, 120))
    if kind == "ensemble":
        count = _log_int(rng, 12, 1024 if prec == "mixed" else 320)
        nmin = _log_int(rng, 64, 512)
        return dict(kind=kind, prec=prec, count=count, nmin=nmin, nmax=_log_int(rng, 2 * nmin, 8192),
                    parts=rng.choice((1, 2, 4)), steps=rng.randint(20, 40))
    if kind in ("shear", "rt"):
        n1 = _log_int(rng, 48, 1400)
        n2 = max(40, min(1800, int(round(n1 * math.exp(rng.uniform(-0.9, 0.9))))))
        return dict(kind=kind, prec=prec, n1=n1, n2=n2, steps=rng.randint(10, 30))
    if kind == "blast":
        if rng.random() < 0.4:
            return dict(kind=kind, prec=prec, ndim=2, n1=_log_int(rng, 64, 400), n2=2 ** rng.randint(5, 8), n3=1,
                        radius=rng.choice(("uniform", "sinh")), steps=rng.randint(10, 60))
        k = rng.randint(4, 6)
        return dict(kind=kind, prec=prec, ndim=3, n1=_log_int(rng, 48, 220), n2=2 ** k, n3=2 ** (k + 1),
                    radius=rng.choice(("uniform", "sinh")), steps=rng.randint(5, 20))
    return dict(kind=kind, zones=_log_int(rng, 1000, 4000000))


# ------------------------------------------------------------------------- setups
def _u(seed, k, shape):
    """Uniform doubles in [-1, 1) from the seed, on the GPU."""
    g = torch.Generator(device="cuda").manual_seed((int(seed) * 1000003 + k) & 0x7FFFFFFFFFFFFFFF)
    return 2.0 * torch.rand(shape, generator=g, device="cuda", dtype=torch.float64) - 1.0


def _pinned(t):
    return t.cpu().pin_memory()


@functools.lru_cache(maxsize=None)
def _blast_grid(ndim, n1, n2, n3, radius):
    """The blast problem (its grid and quiescent state) of a size: the same for every seed."""
    kw = dict(coords="sinh_rt", r_in=1.0e-3) if radius == "sinh" else {}
    pb = P.sedov_3d(n1, n2, n3, **kw) if ndim == 3 else P.sedov_2d_spherical(n1, n2, **kw)
    return pb, torch.from_numpy(pb.ic)


def _ensemble(case, seed):
    """(problems without states, parameters per problem) of a seeded ensemble: zone counts
    log-uniform in [nmin, nmax], kinds in turn, pressure and density ratios log-uniform."""
    zone_rng = np.random.RandomState(977 * case["count"] + case["nmin"])   # sizes belong to the case
    rng = np.random.RandomState(seed % (2 ** 31))
    base = {(k, g): P.spherical_1d(k, 8, g) for k in KINDS_1D for g in GAMMAS}
    pbs, par = [], []
    for m in range(case["count"]):
        n1 = int(round(math.exp(zone_rng.uniform(math.log(case["nmin"]), math.log(case["nmax"])))))
        kind = KINDS_1D[m % 3]
        gam = GAMMAS[zone_rng.randint(3)]
        rr, pr = math.exp(rng.uniform(math.log(2.0), math.log(100.0))), math.exp(rng.uniform(math.log(2.0), math.log(1.0e4)))
        pbs.append(dataclasses.replace(base[kind, gam], n=(n1, 1, 1), dx=(1.0 / n1, 2.0, 2.0 * math.pi)))
        par.append((kind, gam, rr, pr))
    return pbs, par


def _ensemble_state(pbs, par, seed):
    """The [zone][5] states of the problems one after the other (CUDA, FP64)."""
    n = torch.tensor([p.n[0] for p in pbs], device="cuda")
    own = torch.repeat_interleave(torch.arange(len(pbs), device="cuda"), n)
    first = torch.cumsum(n, 0) - n
    r = (torch.arange(own.numel(), device="cuda") - first[own] + 0.5).double() / n[own].double()
    col = lambda f: torch.tensor([f(*q) for q in par], device="cuda", dtype=torch.float64)[own]
    gm1 = col(lambda k, g, rr, pr: g - 1.0)
    r0 = col(lambda k, g, rr, pr: {"sod": 0.5, "sedov": 0.05, "noh": -1.0}[k])
    rin = col(lambda k, g, rr, pr: rr if k == "sod" else 1.0)
    pin = col(lambda k, g, rr, pr: {"sod": pr, "sedov": 1.0e-5 * pr, "noh": 1.0}[k])
    pout = col(lambda k, g, rr, pr: {"sod": 1.0, "sedov": 1.0e-5, "noh": 1.0e-6}[k])
    v = col(lambda k, g, rr, pr: -1.0 if k == "noh" else 0.0)
    ic = torch.zeros((own.numel(), 5), device="cuda", dtype=torch.float64)
    ic[:, 0] = torch.where(r < r0, rin, 1.0) * (1.0 + NOISE * _u(seed, 1, own.shape))
    ic[:, 1] = torch.where(r < r0, pin, pout) / gm1
    ic[:, 2] = v
    return ic


def _parts(pbs, k):
    """The problem list cut into k runs of about equal zone count."""
    total, run, cuts = sum(p.n[0] for p in pbs), 0, [0]
    for m, p in enumerate(pbs):
        if run * k >= total * len(cuts) and m > cuts[-1] and len(cuts) < k:
            cuts.append(m)
        run += p.n[0]
    cuts.append(len(pbs))
    return [(a, b) for a, b in zip(cuts[:-1], cuts[1:]) if b > a]


def _box(case):
    """The 2-D problem of a case, without its state."""
    n1, n2 = case["n1"], case["n2"]
    if case["kind"] == "shear":
        pb = P.kelvin_helmholtz(4, 4)
        return dataclasses.replace(pb, n=(n1, n2, 1), dx=(1.0 / n1, 1.0 / n2, 1.0))
    pb = P.rayleigh_taylor_2d(4, 4)
    return dataclasses.replace(pb, n=(n1, n2, 1), dx=(0.5 / n1, 1.0 / n2, 1.0))


def _single(case, seed):
    """(problem, state) of a one-problem Solver case (state: CUDA [zone][5])."""
    kind = case["kind"]
    if kind == "tube" or kind == "embed":
        n1 = case["n1"]
        if kind == "tube":
            pb = dataclasses.replace(P.sod(8), n=(n1, 1, 1), dx=(1.0 / n1, 1.0, 1.0))
        else:
            pb = dataclasses.replace(P.spherical_1d("sod", 8, 1.4), n=(n1, 1, 1), dx=(1.0 / n1, 2.0, 2.0 * math.pi))
        x = (torch.arange(n1, device="cuda", dtype=torch.float64) + 0.5) / n1
        ic = torch.zeros((n1, 5), device="cuda", dtype=torch.float64)
        ic[:, 0] = torch.where(x < 0.5, 1.0, 0.125) * (1.0 + NOISE * _u(seed, 1, x.shape))
        ic[:, 1] = torch.where(x < 0.5, 1.0, 0.1) / (pb.gam - 1.0)
        return pb, ic
    if kind == "blast":
        pb, ic = _blast_grid(case["ndim"], case["n1"], case["n2"], case["n3"], case["radius"])
        ic = ic.to("cuda")
        ic[:, 0] *= 1.0 + NOISE * _u(seed, 1, (ic.shape[0],))
        if case["radius"] == "uniform":
            ic[:, 2:] = 0.1 * NOISE * _u(seed, 2, (ic.shape[0], 3))
        return pb, ic
    pb = _box(case)
    n1, n2, _ = pb.n
    x = ((torch.arange(n1, device="cuda", dtype=torch.float64) + 0.5) * pb.dx[0])[:, None].expand(n1, n2)
    y = ((torch.arange(n2, device="cuda", dtype=torch.float64) + 0.5) * pb.dx[1])[None, :].expand(n1, n2)
    ic = torch.zeros((n1, n2, 5), device="cuda", dtype=torch.float64)
    if kind == "shear":
        inner = (y - 0.5).abs() < 0.25
        ic[..., 0] = torch.where(inner, 2.0, 1.0)
        ic[..., 1] = 2.5 / (pb.gam - 1.0)
        ic[..., 2] = torch.where(inner, 0.5, -0.5) + 1.0e-3 * _u(seed, 1, (n1, n2))
        ic[..., 3] = 0.01 * torch.sin(4.0 * math.pi * x) + 1.0e-3 * _u(seed, 2, (n1, n2))
    else:
        g, top = pb.grav[1], y >= 0.5
        base = 10.0 / 7.0 + 0.25
        ic[..., 0] = torch.where(top, 2.0, 1.0)
        ic[..., 1] = torch.where(top, base + 0.5 * g + 2.0 * g * (y - 0.5), base + g * y) / (pb.gam - 1.0)
        ic[..., 3] = 0.01 * _u(seed, 1, (n1, n2)) * torch.exp(-((y - 0.5) / 0.05) ** 2)
    return pb, ic.reshape(n1 * n2, 5)


@functools.lru_cache(maxsize=None)
def _eos_table():
    """The synthetic table at the reference's sizes (all records on the host, the energy record and
    the handle on the device): one table serves every call of a program."""
    tab = ET.synthetic_table()
    return tab, torch.from_numpy(tab[[0, 1, 2, 11]]).to("cuda"), ET.EosTable(tab)


def _eos_zones(case, seed):
    """Zones inside the table: log10 rho, Ye and log10 T uniform, the energy the table gives there,
    and as guess the temperature a time step earlier (a few per cent off)."""
    _, rec, _ = _eos_table()
    g, n = ET.REFERENCE_GRID, case["zones"]
    x = 0.5 + 0.498 * _u(seed, 1, (4, n))
    rl, ye, tl = (a + (b - a) * x[k] for k, (a, b) in enumerate(((g.r1, g.r2), (g.y1, g.y2), (g.t1, g.t2))))
    val = _eos_at(rec[:1], g, rl, ye, tl)[0]
    rho = 10.0 ** rl
    return rho, rho * val * ET.ERG_PER_UNIT, ye, 10.0 ** (tl + 0.03 * (x[3] - 0.5))


def _eos_corner(g, rl, ye):
    dr, dy = (g.r2 - g.r1) / (g.nr - 1), (g.y2 - g.y1) / (g.ny - 1)
    jr = ((rl - g.r1) / dr).long().clamp(0, g.nr - 2)
    jy = ((ye - g.y1) / dy).long().clamp(0, g.ny - 2)
    fr, fy = (rl - (g.r1 + jr.double() * dr)) / dr, (ye - (g.y1 + jy.double() * dy)) / dy
    return jr, jy, ((1 - fr) * (1 - fy), fy * (1 - fr), (1 - fy) * fr, fy * fr)


def _eos_row(rec, jr, jy, w, k):
    """The records at temperature row k, bilinear in (log rho, Ye)."""
    return sum(c * rec[:, jy + a, jr + b, k] for c, (a, b) in zip(w, ((0, 0), (1, 0), (0, 1), (1, 1))))


def _eos_at(rec, g, rl, ye, tl):
    jr, jy, w = _eos_corner(g, rl, ye)
    dt = (g.t2 - g.t1) / (g.nt - 1)
    jt = ((tl - g.t1) / dt).long().clamp(0, g.nt - 2)
    ft = (tl - (g.t1 + jt.double() * dt)) / dt
    return (1 - ft) * _eos_row(rec, jr, jy, w, jt) + ft * _eos_row(rec, jr, jy, w, jt + 1)


# ------------------------------------------------------------------------- a pass
def _prec(case):
    return mb.PREC_MIXED if case.get("prec") == "mixed" else mb.PREC_FP64


def prepare(case, seed):
    kind = case["kind"]
    if kind == "eos":
        rho, u, ye, temp = _eos_zones(case, seed)
        out = [torch.empty_like(rho) for _ in range(4)]
        return dict(kind=kind, table=_eos_table()[2], n=case["zones"], inp=(rho, u, ye), temp=temp, out=out)
    if kind == "ensemble":
        pbs, par = _ensemble(case, seed)
        ic = _ensemble_state(pbs, par, seed)
        solvers, ins, outs, at = [], [], [], 0
        for a, b in _parts(pbs, case["parts"]):
            nz = sum(p.n[0] for p in pbs[a:b])
            solvers.append(mb.Solver(pbs[a:b], precision=_prec(case), upload=False))
            ins.append(_pinned(ic[at:at + nz]))
            outs.append(torch.empty((nz, 5), dtype=torch.float64).pin_memory())
            at += nz
        return dict(kind=kind, solvers=solvers, ins=ins, outs=outs, steps=case["steps"])
    pb, ic = _single(case, seed)
    if kind == "embed":
        L = mb.library()
        L.mdg_advance_1d_noalloc.restype = ctypes.c_int
        L.mdg_advance_1d_noalloc.argtypes = [ctypes.c_void_p] * 3 + [ctypes.c_int] + [ctypes.c_void_p] * 3
        x = ic.t().contiguous()
        return dict(kind=kind, call=L.mdg_advance_1d_noalloc, desc=desc_of(pb), inp=x, out=torch.empty_like(x),
                    steps=case["steps"], t=ctypes.c_double(), dt=ctypes.c_double())
    return dict(kind=kind, solver=mb.Solver(pb, precision=_prec(case), upload=False), inp=_pinned(ic),
                out=torch.empty(ic.shape, dtype=torch.float64).pin_memory(), steps=case["steps"])


def _fields(states):
    """Density, internal energy and velocity of the [zone][5] states, as views."""
    return {"rho": [s[:, 0] for s in states], "u": [s[:, 1] for s in states], "v": [s[:, 2:] for s in states]}


def run(st):
    kind = st["kind"]
    if kind == "eos":
        st["table"].given_rex_device(st["n"], *(x.data_ptr() for x in st["inp"]), st["temp"].data_ptr(),
                                     *(x.data_ptr() for x in st["out"]), torch.cuda.current_stream().cuda_stream)
        return {k: x for k, x in zip(("temp", "press", "cs", "ent", "gam1"), [st["temp"]] + st["out"])}
    if kind == "ensemble":
        run_host(st["solvers"], [x.data_ptr() for x in st["ins"]], [x.data_ptr() for x in st["outs"]], st["steps"])
        return _fields(st["outs"])
    if kind == "embed":
        rc = st["call"](ctypes.byref(st["desc"]), st["inp"].data_ptr(), st["out"].data_ptr(), st["steps"],
                        torch.cuda.current_stream().cuda_stream, ctypes.byref(st["t"]), ctypes.byref(st["dt"]))
        if rc:
            raise RuntimeError("mdg_advance_1d_noalloc: status %d" % rc)
        s = st["out"]
        return {"rho": [s[0]], "u": [s[1]], "v": [s[2:].t()], "t": st["t"].value}
    s = st["solver"]
    s.upload_ptr(0, st["inp"].data_ptr())
    s.step(st["steps"])
    s.download_ptr(0, st["out"].data_ptr())
    s.synchronize()
    return dict(_fields([st["out"]]), t=s.time()[0])


def work(case):
    """A step is two RK stages; the first reads the state and writes one, the second reads the
    stage state and the base state and writes one (200 bytes per zone and step).  Operations per
    zone, direction and stage: about 420 for the six reconstructed variables, 150 for the
    Riemann problem, 80 for the update.  The EOS update streams 72 bytes a zone and reads 8
    table points of 32 bytes, with about 150 operations."""
    if case["kind"] == "eos":
        return {"bytes": (72.0 + 256.0) * case["zones"], "flops": 150.0 * case["zones"]}
    if case["kind"] == "ensemble":
        zones, nd = sum(p.n[0] for p in _ensemble(case, 0)[0]), 1
    elif case["kind"] in ("embed", "tube"):
        zones, nd = case["n1"], 1
    elif case["kind"] == "blast":
        pb, _ = _blast_grid(case["ndim"], case["n1"], case["n2"], case["n3"], case["radius"])
        zones, nd = pb.ncell, case["ndim"]
    else:
        zones, nd = case["n1"] * case["n2"], 2
    return {"bytes": 200.0 * zones * case["steps"], "flops": 2.0 * (570.0 * nd + 80.0) * zones * case["steps"]}


def tolerance(case):
    """About four times the difference from exact() seen over the ranges of draw() (blasts: between
    the two precisions; plain FP64 blasts like the other FP64 grids).  The FP64 1-D figures are those of
    reconstruction coefficients formed from absolute coordinates, (x / dx)^2 ulps."""
    kind, mixed = case["kind"], case.get("prec") == "mixed"
    rel, big = {
        "eos": (1e-14, 1e-13),
        "embed": (1e-6, 6e-5), "tube": (1e-6, 6e-5),
        "ensemble": (2e-6, 5e-4) if mixed else (1e-6, 6e-5),
        "shear": (2e-7, 2e-6) if mixed else (5e-11, 2e-9),
        "rt": (5e-5, 1e-3) if mixed else (3e-8, 4e-6),      # v: noise-driven, far below the sound speed
        "blast": (1e-4, 4e-2) if mixed else (1e-9, 1e-5),
    }[kind]
    return {"rel": rel, "max": big}


# ------------------------------------------------------------------------- the same in 64 bits
class _Fit:
    """Geometry of the parabolic reconstruction along the last axis: moments of the volume weight
    (x^2 on the radius, 1 on Cartesian axes) over a zone and its neighbours about the zone's own
    centre, lengths in units of the zone width."""

    def __init__(self, xc, spherical):
        # xc: zone centres in units of the zone width
        def moments(c):
            # zone [c - 1/2, c + 1/2]: integrals of w s^k, k = 0, 1, 2, with w = (xc + s)^2 or 1
            p = [((c + 0.5) ** (k + 1) - (c - 0.5) ** (k + 1)) / (k + 1) for k in range(5)]
            if not spherical:
                return [torch.full_like(xc, q) for q in p[:3]]
            return [xc * xc * p[k] + 2.0 * xc * p[k + 1] + p[k + 2] for k in range(3)]
        self.gm, self.bm, self.am = moments(-1.0)
        self.g0, self.b0, self.a0 = moments(0.0)
        self.gp, self.bp, self.ap = moments(1.0)
        # slopes of the averages: mean of s and s^2 in each zone relative to the centre zone's
        b0, a0 = self.b0 / self.g0, self.a0 / self.g0
        self.sm, self.qm = self.bm / self.gm - b0, self.am / self.gm - a0
        self.sp, self.qp = self.bp / self.gp - b0, self.ap / self.gp - a0
        self.det = self.qm * self.sp - self.qp * self.sm
        self.b, self.a = b0, a0


def _recon(f, am, a, ap):
    """Face values (left, right) of the zone averages a with neighbours am, ap."""
    dqm, dqp = am - a, ap - a
    A = (dqm * f.sp - dqp * f.sm) / f.det
    B = (f.qm * dqp - f.qp * dqm) / f.det
    at = lambda s: A * (s * s - f.a) + B * (s - f.b)     # parabola minus a
    l, r = at(-0.5), at(0.5)
    lo, hi = 0.75 * dqm, 0.75 * dqp
    l = torch.where(-l * (l - lo) < 0, lo, l)
    r = torch.where((hi - r) * r < 0, hi, r)
    # the parabola with zone average 0 through the limited face values
    B = r - l
    A = (0.5 * (l + r) + f.b * B) / (0.25 - f.a)
    s = -B / (2.0 * A)
    inside = (s > -0.5) & (s < 0.5)
    right = s > 0.0
    mr = 1.0 / (f.a - f.b + 0.25)       # mean of (s - 1/2)^2
    ml = 1.0 / (f.a + f.b + 0.25)
    nl = torch.where(inside & right, r - r * mr, l)
    nr = torch.where(inside & ~right, l - l * ml, r)
    flat = dqm * dqp >= 0
    return a + torch.where(flat, 0.0, nl), a + torch.where(flat, 0.0, nr)


def _waves(L, R, ul, ur, G):
    rl, pl, rr, pr = L[0], L[5], R[0], R[5]
    cl, cr = torch.sqrt(G * pl / rl), torch.sqrt(G * pr / rr)
    pmax, pmin = torch.maximum(pl, pr), torch.minimum(pl, pr)
    shock = (pmax - pmin) / pmin > 0.5
    pv = torch.clamp(0.5 * (pl + pr) - 0.125 * (ur - ul) * (rl + rr) * (cl + cr), min=0.0)
    plr = (pl / pr) ** ((G - 1) / (2 * G))
    s0 = (plr * ul / cl + ur / cr + 2 * (plr - 1) / (G - 1)) / (plr / cl + 1 / cr)
    ex = 2 * G / (G - 1)
    base = lambda x: torch.clamp(x, min=0.0)
    p2 = 0.5 * (pl * base(1 + (G - 1) / (2 * cl) * (ul - s0)) ** ex + pr * base(1 + (G - 1) / (2 * cr) * (s0 - ur)) ** ex)
    gl = torch.sqrt(2 / ((G + 1) * rl) / (pv + (G - 1) / (G + 1) * pl))
    gr = torch.sqrt(2 / ((G + 1) * rr) / (pv + (G - 1) / (G + 1) * pr))
    p3 = torch.clamp((gl * pl + gr * pr - (ur - ul)) / (gl + gr), min=0.0)
    keep = (pmax / pmin < 2) & (pv >= pmin) & (pv <= pmax)
    ps = torch.where(keep, pv, torch.where(pv < pmin, torch.clamp(p2, min=0.0), p3))
    ql = torch.sqrt(torch.where(ps <= pl, 1.0, 1 + (G + 1) / (2 * G) * (ps / pl - 1)))
    qr = torch.sqrt(torch.where(ps <= pr, 1.0, 1 + (G + 1) / (2 * G) * (ps / pr - 1)))
    sl, sr = ul - cl * ql, ur + cr * qr
    ss = (pr - pl + rl * ul * (sl - ul) - rr * ur * (sr - ur)) / (rl * (sl - ul) - rr * (sr - ur))
    return sl, sr, ss, ps, shock


def _cons(W, d):
    """(conserved, flux density along direction d) of face states W = rho, u, v0, v1, v2, p."""
    rho, u, v, p = W[0], W[1], W[2:5], W[5]
    e = 0.5 * rho * (v[0] * v[0] + v[1] * v[1] + v[2] * v[2]) + u
    U = torch.stack([rho, e, rho * v[0], rho * v[1], rho * v[2]])
    F = U * v[d]
    F[1] += p * v[d]
    F[2 + d] += p
    return U, F


def _hllc(L, R, d, G):
    """(flux density, signal speed, shock flag) of the faces between states L and R."""
    ul, ur = L[2 + d], R[2 + d]
    sl, sr, ss, ps, shock = _waves(L, R, ul, ur, G)
    sr = torch.where(ss > sr, 1.001 * ss, sr)
    sl = torch.where(ss < sl, 1.001 * ss, sl)
    left = ss > 0
    W = torch.where(left, L, R)
    sk, uk = torch.where(left, sl, sr), torch.where(left, ul, ur)
    U, F = _cons(W, d)
    S = U * ((sk - uk) / (sk - ss))
    S[2 + d] = S[0] * ss
    S[1] = (U[1] * (sk - uk) - W[5] * uk + ps * ss) / (sk - ss)
    F = torch.where(sl > 0, _cons(L, d)[1], torch.where(sr < 0, _cons(R, d)[1], F + sk * (S - U)))
    return F, torch.maximum(sl.abs(), sr.abs()), shock


def _hlle(L, R, d, G):
    ul, ur = L[2 + d], R[2 + d]
    sl, sr, _, _, _ = _waves(L, R, ul, ur, G)
    (UL, FL), (UR, FR) = _cons(L, d), _cons(R, d)
    cmax, cmin = torch.clamp(sr, min=0.0), torch.clamp(sl, max=0.0).abs()
    F = (cmin * FR + cmax * FL - cmax * cmin * (UR - UL)) / (cmax + cmin)
    return F, torch.maximum(cmax, cmin)


def _source_dt(w, U, S):
    """The limit that the sources S of conserved U set to dt (0.02 of a variable's own time)."""
    mom = (w[2:5] * S[2:5]).sum(0)
    tiny = 1.0e-16
    a = torch.minimum(0.02 * U[0] / (S[0].abs() + tiny), 0.02 * U[1] / (S[1].abs() + tiny))
    return torch.minimum(a, 2.0 * w[1] / ((S[1].abs() - mom.abs()).abs() + tiny))


def _prim(U):
    v = U[2:5] / U[0]
    return torch.cat([U[:1], (U[1] - 0.5 * U[0] * (v * v).sum(0))[None], v])


def _next_dt(pb, k, mind, dtold):
    dt = pb.cfl * torch.clamp(mind, max=min(pb.dtmax, pb.initial_dt) if k == 0 else pb.dtmax)
    return dt * pb.dt_init_safety if k == 0 else torch.minimum(dtold * pb.dt_grow_safety, dt)


def _exact_1d(pbs, ic, steps):
    """Problems on the uniform radius (or one Cartesian tube): all zones in one row, each problem
    with two ghost zones a side."""
    sph = pbs[0].geom == P.SPHERICAL
    dev = ic.device
    n = torch.tensor([p.n[0] for p in pbs], device=dev)
    np_ = len(pbs)
    own = torch.repeat_interleave(torch.arange(np_, device=dev), n + 4)
    start = torch.cumsum(n + 4, 0) - (n + 4)
    z = torch.arange(own.numel(), device=dev) - start[own] - 2
    inner = (z >= 0) & (z < n[own])
    lo, hi = z < 0, z >= n[own]
    mirror = torch.where(lo & sph, -1 - z, z.clamp(min=0))
    src = start[own] + 2 + torch.minimum(mirror, n[own] - 1)
    col = lambda f: torch.tensor([f(p) for p in pbs], device=dev, dtype=torch.float64)
    G, dx = col(lambda p: p.gam)[own], (1.0 / n.double())[own]
    floor = col(lambda p: float(p.enforce_floors))[own] > 0
    rfl, efl = col(lambda p: p.rho_floor)[own], col(lambda p: p.e_floor)[own]
    noh = (col(lambda p: float(p.prob_kind == P.PROB_NOH))[own] > 0) & hi
    xc = z.double() + 0.5
    fit = _Fit(xc, sph)
    xe = z.double()                                   # lower edge, in zone widths
    area = xe * xe * dx * dx if sph else torch.ones_like(xe)
    vol = fit.g0 * dx ** 3 if sph else dx
    rcen = (xc + fit.b) * dx
    c101 = (xc / fit.g0 / dx) if sph else torch.zeros_like(dx)     # int r dr / int r^2 dr
    w = torch.zeros((5, own.numel()), device=dev, dtype=torch.float64)
    w[:, inner] = ic.t()
    flip = torch.ones((5, own.numel()), device=dev, dtype=torch.float64)
    if sph:
        flip[2, lo] = -1.0
        flip[4, lo] = -1.0

    def fill(w, t):
        w = w[:, src] * flip
        if sph:
            g = (1.0 + t[own] / rcen) ** 2
            q = torch.stack([g, 1.0e-6 / (G - 1), -torch.ones_like(g), torch.zeros_like(g), torch.zeros_like(g)])
            w = torch.where(noh, q, w)
        return w

    def seg_min(x, ok):
        big = torch.full((np_,), 1.0e100, device=dev, dtype=torch.float64)
        return big.scatter_reduce(0, own[ok], x[ok], "amin")

    def cons(w):
        return torch.cat([w[:1], (w[1] + 0.5 * w[0] * (w[2:5] ** 2).sum(0))[None], w[0] * w[2:5]])

    cs0 = torch.sqrt(G * (G - 1) * w[1] / w[0])
    mind = seg_min(dx / (w[2].abs() + cs0), inner)
    t, dtold = torch.zeros(np_, device=dev, dtype=torch.float64), torch.full((np_,), 1.0e100, device=dev, dtype=torch.float64)
    face = (z >= 0) & (z <= n[own])
    for k in range(steps):
        dt = _next_dt(pbs[0], k, mind, dtold)
        dtold = dt
        mind = torch.full_like(dt, 1.0e100)
        ph = w
        for stage in range(2):
            p = fill(ph, t + dt if stage else t)
            q = torch.cat([p, ((G - 1) * p[1])[None]])
            l, r = _recon(fit, torch.roll(q, 1, 1), q, torch.roll(q, -1, 1))
            F, sig, _ = _hllc(torch.roll(r, 1, 1), l, 0, G)
            F = torch.where(area < 1.0e-16, 0.0, F * area)      # the face at the origin
            sig = torch.where(area < 1.0e-16, 1.0e-200, sig)
            mind = torch.minimum(mind, seg_min(dx / sig, face))
            S = torch.zeros_like(p)
            S[2] = 2.0 * q[5] * c101
            base = cons(w)
            mind = torch.minimum(mind, seg_min(_source_dt(w, base, S), inner))
            dU = dt[own] * ((torch.roll(F, -1, 1) - F) / vol - S)
            new = _prim(base - dU if stage == 0 else 0.5 * base + 0.5 * cons(p) - 0.5 * dU)
            new = torch.cat([torch.where(floor, torch.maximum(new[:1], rfl), new[:1]),
                             torch.where(floor, torch.maximum(new[1:2], efl), new[1:2]), new[2:]])
            ph = torch.where(inner, new, torch.ones_like(new))
            if stage:
                cs = torch.sqrt(G * q[5] / q[0])
                mind = torch.minimum(mind, seg_min(dx / (ph[2].abs() + cs), inner))
        w = ph
        t = t + dt
    return w[:, inner].t().contiguous(), t


def _exact_2d(pb, ic, steps):
    n1, n2, _ = pb.n
    dev, G = ic.device, torch.tensor(pb.gam, device=ic.device, dtype=torch.float64)
    dx = pb.dx[:2]
    w = ic.t().reshape(5, n1, n2).contiguous()
    fit = _Fit(torch.zeros((), device=dev, dtype=torch.float64), False)
    refl = pb.bc_lo[1] == P.REFLECT
    g = pb.grav[1]

    def pad(w, d):
        """Two ghost zones a side along direction d (axis 1 + d)."""
        ax = 1 + d
        n = w.shape[ax]
        lo, hi = w.narrow(ax, n - 2, 2), w.narrow(ax, 0, 2)
        if d == 1 and refl:
            lo, hi = w.narrow(ax, 0, 2).flip(ax).clone(), w.narrow(ax, n - 2, 2).flip(ax).clone()
            lo[3] *= -1.0
            hi[3] *= -1.0
        return torch.cat([lo, w, hi], ax)

    def cons(w):
        return torch.cat([w[:1], (w[1] + 0.5 * w[0] * (w[2:5] ** 2).sum(0))[None], w[0] * w[2:5]])

    def faces(p, d):
        """States either side of the n + 1 faces along direction d."""
        q = pad(p, d)
        q = torch.cat([q, ((G - 1) * q[1])[None]])
        ax, n = 1 + d, q.shape[1 + d]
        l, r = _recon(fit, q.narrow(ax, 0, n - 2), q.narrow(ax, 1, n - 2), q.narrow(ax, 2, n - 2))
        return r.narrow(ax, 0, n - 3), l.narrow(ax, 1, n - 3)

    cs = torch.sqrt(G * (G - 1) * w[1] / w[0])
    mind = (1.0 / ((w[2].abs() + cs) / dx[0] + (w[3].abs() + cs) / dx[1])).min()
    t, dtold = torch.zeros((), device=dev, dtype=torch.float64), torch.tensor(1.0e100, device=dev, dtype=torch.float64)
    for k in range(steps):
        dt = _next_dt(pb, k, mind, dtold)
        dtold = dt
        mind = torch.full_like(dt, 1.0e100)
        ph, marks = w, None
        for stage in range(2):
            p = ph
            F0, s0, sh = _hllc(*faces(p, 0), 0, G)
            # a direction-1 face beside a direction-0 shock, or on the boundary, takes HLLE: the faces
            # (i, j) and (i, j - 1) of this stage, in the second stage also faces i .. i + 2 of the first
            flag = sh[:n1].clone()
            if stage == 0:
                marks = torch.cat([sh, torch.zeros_like(sh[:2])])
            else:
                flag |= marks[:n1] | marks[1:n1 + 1] | marks[2:n1 + 2]
            e = torch.ones((n1, 1), dtype=torch.bool, device=dev)
            f = torch.cat([e, flag], 1) | torch.cat([flag, e], 1)
            L, R = faces(p, 1)
            Fc, sc, _ = _hllc(L, R, 1, G)
            Fe, se = _hlle(L, R, 1, G)
            F1, s1 = torch.where(f, Fe, Fc), torch.where(f, se, sc)
            mind = torch.minimum(mind, torch.minimum((dx[0] / s0).min(), (dx[1] / s1).min()))
            base = cons(w)
            S = torch.zeros_like(p)
            S[1], S[3] = p[0] * p[3] * g, p[0] * g
            mind = torch.minimum(mind, _source_dt(w, base, S).min())
            div = (F0[:, 1:] - F0[:, :-1]) / dx[0] + (F1[:, :, 1:] - F1[:, :, :-1]) / dx[1]
            dU = dt * (div - S)
            ph = _prim(base - dU if stage == 0 else 0.5 * base + 0.5 * cons(p) - 0.5 * dU)
            if stage:
                cs = torch.sqrt(G * (G - 1) * p[1] / p[0])
                mind = torch.minimum(mind, (1.0 / ((ph[2].abs() + cs) / dx[0] + (ph[3].abs() + cs) / dx[1])).min())
        w = ph
        t = t + dt
    return w.reshape(5, n1 * n2).t().contiguous(), t


def _exact_eos(case, seed):
    _, rec, _ = _eos_table()
    g = ET.REFERENCE_GRID
    rho, u, ye, _ = _eos_zones(case, seed)
    outs = []
    for a in range(0, case["zones"], 1 << 20):
        r, y = rho[a:a + (1 << 20)], ye[a:a + (1 << 20)]
        e = u[a:a + (1 << 20)] / r / ET.ERG_PER_UNIT
        jr, jy, w = _eos_corner(g, torch.log10(r), y)
        lo, hi = torch.zeros_like(jr), torch.full_like(jr, g.nt - 1)
        for _ in range(9):                           # the energy record grows with temperature
            mid = (lo + hi) // 2
            below = _eos_row(rec[:1], jr, jy, w, mid)[0] < e
            lo, hi = torch.where(below, mid, lo), torch.where(below, hi, mid)
        lo = lo.clamp(max=g.nt - 2)
        v0, v1 = _eos_row(rec, jr, jy, w, lo), _eos_row(rec, jr, jy, w, lo + 1)
        f = (e - v0[0]) / (v1[0] - v0[0])
        v = v0 + f * (v1 - v0)
        p = torch.exp(v[1]) * 1.60217733e33
        dt = (g.t2 - g.t1) / (g.nt - 1)
        outs.append([10.0 ** (g.t1 + (lo + f) * dt), p, torch.sqrt(v[3] * p / r), v[2], v[3]])
    return {k: torch.cat(x) for k, x in zip(("temp", "press", "cs", "ent", "gam1"), zip(*outs))}


def exact(case, seed):
    """The same with plain torch in 64 bits.  The dendritic grid's restriction and prolongation
    between refinement levels have no short form: None for the blasts."""
    kind = case["kind"]
    if kind == "blast":
        return None
    if kind == "eos":
        return _exact_eos(case, seed)
    if kind == "ensemble":
        pbs, par = _ensemble(case, seed)
        s, _ = _exact_1d(pbs, _ensemble_state(pbs, par, seed), case["steps"])
        cut = [sum(p.n[0] for p in pbs[a:b]) for a, b in _parts(pbs, case["parts"])]
        return _fields(list(torch.split(s, cut)))
    pb, ic = _single(case, seed)
    if kind in ("embed", "tube"):
        s, t = _exact_1d([pb], ic, case["steps"])
    else:
        s, t = _exact_2d(pb, ic, case["steps"])
    return dict(_fields([s]), t=float(t))
