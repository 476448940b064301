"""The work users have this library do, as measurable cases.

Each case is one pass through the public C interface (include/lmie_interface.h,
include/lmie_b200.h) the way a calling program uses it: the inputs, the output
arrays and (for re-weighting) the saved per-radius kernels are the caller's,
made once; a pass is the call.  The library takes host structures and returns
host arrays by its nature, so a pass includes the host's preparation and the
copies in both directions; the exception is `spheres`, whose radii and results
are device buffers.

Kinds of case:
  solve     one lmie_solution(): a size distribution at one wavelength
  bands     one lmie_solution_batch2() over the spectral bands of one aerosol
  batch     one lmie_solution_batch2() over independent uneven cases
  reweight  a retrieval loop: several save_control = 2 calls on the kernels of
            one save_control = 1 solve
  adjoint   one lmie_solution_adjoint(): loss and gradient over wavelengths
  spheres   one lmie_cross_sections_noalloc() on device buffers

`exact` restates the same quantities in plain torch FP64 from the textbook
formulas, with recurrences and contractions of its own.
"""
from __future__ import annotations

import ctypes as C
import dataclasses
import functools
import math
import os

import numpy as np
import torch

import lmie_b200
from lmie_b200 import abi, workloads

PD = C.POINTER(C.c_double)
THREADS = min(16, os.cpu_count() or 1)
PRECISION = {"fp64": abi.PRECISION_FP64, "tf32x3": abi.PRECISION_TF32X3, "int8": abi.PRECISION_INT8}
SCALARS = 13                # doubles of lmie_out_data after n_coef: 9 of the distribution, 4 cross sections
DERIVS = ("", "mr", "a1,a2", "mr,mi", "mr,mi,a1", "mr,mi,a1,a2")


def listed():
    return [
        # one sphere with its phase matrix: the smallest call, all latency
        dict(name="sphere", kind="solve", dist="mono", x_max=14.3, n_int=1, n_quad=1, derivs="", expansion="gc",
             n_angles=181, accuracy=1e-7),
        # the plain aerosol solve (200 radii, size parameters to 23) with two derivatives
        dict(name="aerosol", kind="solve", dist="log_normal", x_max=22.85, n_int=1, n_quad=200, derivs="mr,a1",
             expansion="gc", n_angles=181, accuracy=1e-7),
        # the linearised cloud droplet: 4 x 500 radii, size parameters to 436
        dict(name="cloud_droplet", kind="solve", dist="gamma", x_max=435.83, n_int=4, n_quad=500,
             derivs="mr,mi,a1,a2", expansion="gc", n_angles=181, accuracy=1e-7),
        # the large-particle configuration: size parameters to 5000, 16 x 500 radii, every coefficient kept
        # (the tail of its expansion is rounding noise, so a threshold there would not mean anything)
        dict(name="large_particles", kind="solve", dist="gamma", x_max=4999.7, n_int=16, n_quad=500,
             derivs="mr,mi,a1,a2", expansion="gc", n_angles=181, accuracy=0.0),
        # the bands of a radiative-transfer table: 30 wavelengths of one aerosol, Legendre coefficients,
        # an odd quadrature and a coarse angle grid
        dict(name="bands_legendre", kind="bands", n_bands=30, dist="log_normal", x_max=161.9, n_int=3, n_quad=41,
             derivs="mr,mi", expansion="lc", n_angles=91, accuracy=1e-7, precision="fp64"),
        # cross sections only over many uneven cases: no angles at all
        dict(name="batch_cross_sections", kind="batch", n_cases=777, derivs="", expansion="none", n_angles=0,
             accuracy=1e-7, precision="fp64"),
        # a look-up table of uneven cases with the Jacobian, in the reference's precision; an odd count
        dict(name="batch_fp64", kind="batch", n_cases=1531, derivs="mr,mi,a1,a2", expansion="gc", n_angles=181,
             accuracy=1e-7, precision="fp64"),
        # the benchmark's batch in its headline mode
        dict(name="batch_int8", kind="batch", n_cases=4096, derivs="mr,mi,a1,a2", expansion="gc", n_angles=181,
             accuracy=1e-7, precision="int8"),
        # the split-precision mode; its coefficients are off by some 1e-7, so its user truncates above that
        dict(name="batch_tf32x3", kind="batch", n_cases=512, derivs="mr,mi,a1,a2", expansion="gc", n_angles=181,
             accuracy=1e-5, precision="tf32x3"),
        # retrieval of the size distribution with the optical kernels kept
        dict(name="reweight", kind="reweight", dist="gamma", x_max=435.83, n_int=4, n_quad=500, n_angles=181, calls=4),
        # the gradient of a retrieval over 256 wavelengths x 64 bins x 32 radii
        dict(name="adjoint_retrieval", kind="adjoint", n_lambda=256, n_bins=64, n_quad=32, n_angles=181),
        # a host model that owns the GPU's memory asks for the cross sections of its own radii
        dict(name="spheres", kind="spheres", n_radii=1000, x_max=880.0),
    ]


def _log(rng, lo, hi):
    return math.exp(rng.uniform(math.log(lo), math.log(hi)))


def draw(rng):
    kind = rng.choice(("solve", "solve", "solve", "bands", "batch", "batch", "reweight", "adjoint", "spheres"))
    expansion = rng.choice(("gc", "gc", "gc", "lc", "none"))
    n_angles = 0 if expansion == "none" else rng.choice((19, 91, 181, 181, rng.randint(20, 361)))
    out = dict(expansion=expansion, n_angles=n_angles, derivs=rng.choice(DERIVS), accuracy=1e-7)
    if kind == "solve":
        dist = rng.choice(("mono", "log_normal", "gamma", "gamma"))
        mono = dist == "mono"
        if mono:
            out["derivs"] = rng.choice(("", "mr,mi"))
        return dict(kind=kind, dist=dist, x_max=round(_log(rng, 0.6, 500.0 if mono else 1100.0), 3),
                    n_int=1 if mono else rng.randint(1, 6), n_quad=1 if mono else int(_log(rng, 16, 500)), **out)
    if kind == "bands":
        return dict(kind=kind, n_bands=int(_log(rng, 3, 65)), dist=rng.choice(("log_normal", "gamma")),
                    x_max=round(_log(rng, 10.0, 400.0), 3), n_int=rng.randint(1, 4), n_quad=int(_log(rng, 16, 200)),
                    precision=rng.choice(("fp64", "fp64", "int8")), **out)
    if kind == "batch":
        p = rng.choice(("fp64", "fp64", "int8", "int8", "tf32x3"))
        if p == "tf32x3":
            out["accuracy"] = 1e-5
        return dict(kind=kind, n_cases=int(_log(rng, 40, 3000)), precision=p, **out)
    if kind == "reweight":
        return dict(kind=kind, dist="gamma", x_max=round(_log(rng, 20.0, 500.0), 3), n_int=rng.randint(1, 4),
                    n_quad=int(_log(rng, 32, 500)), n_angles=rng.choice((91, 181, 361)), calls=rng.randint(2, 6))
    if kind == "adjoint":
        return dict(kind=kind, n_lambda=int(_log(rng, 4, 257)), n_bins=int(_log(rng, 5, 65)),
                    n_quad=int(_log(rng, 4, 33)), n_angles=rng.choice((37, 91, 181)))
    return dict(kind=kind, n_radii=int(_log(rng, 1, 1025)), x_max=round(_log(rng, 1.0, 899.0), 3))


# ---------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------
def _distribution(dist, rng, r2):
    """a1, a2, r1, r2 of a distribution whose largest radius is r2."""
    v = rng.uniform(0.05, 0.25)
    r_eff = r2 / (1.0 + 10.0 * v)
    if dist == "mono":
        return r2, 0.0, r2, r2
    if dist == "gamma":
        return r_eff, v, 1e-3 * r_eff, r2
    return r_eff / (1.0 + v) ** 2.5, math.log(1.0 + v), 1e-3 * r_eff, r2


def _options(case):
    return dict(derivs=abi.deriv_unit(*[d for d in case["derivs"].split(",") if d]), n_angles=case["n_angles"],
                calc_gc=int(case["expansion"] == "gc"), calc_lc=int(case["expansion"] == "lc"),
                calc_pf=int(case["expansion"] != "none"), accuracy=case["accuracy"])


def _cases(case, seed):
    """The polydisperse problems of a case, as abi.Case."""
    rng = np.random.Generator(np.random.PCG64(seed))
    kind = case["kind"]
    if kind == "batch":
        # the workload's sizes, at other wavelengths (all lengths scaled alike) and refractive indices
        out = []
        for c in workloads.batched_uneven(case["n_cases"]):
            s = float(rng.uniform(0.8, 1.25))
            out.append(dataclasses.replace(c, lam=c.lam * s, a1=c.a1 * s, r1=c.r1 * s, r2=c.r2 * s,
                                           mr=float(rng.uniform(1.33, 1.6)),
                                           mi=math.exp(rng.uniform(math.log(1e-8), math.log(0.1))), **_options(case)))
        return out
    if kind == "bands":
        lam = np.exp(np.linspace(math.log(0.35), math.log(2.8), case["n_bands"])) * rng.uniform(0.97, 1.03)
        a1, a2, r1, r2 = _distribution(case["dist"], rng, case["x_max"] * lam[0] / (2.0 * math.pi))
        return [abi.Case(dist=case["dist"], lam=float(l), mr=float(rng.uniform(1.35, 1.6)),
                         mi=float(math.exp(rng.uniform(math.log(1e-6), math.log(0.05)))), a1=a1, a2=a2, r1=r1, r2=r2,
                         n_int2=case["n_int"], n_quad=case["n_quad"], **_options(case)) for l in lam]
    lam = rng.uniform(0.34, 1.1)
    a1, a2, r1, r2 = _distribution(case["dist"], rng, case["x_max"] * lam / (2.0 * math.pi))
    base = abi.Case(dist=case["dist"], lam=lam, mr=rng.uniform(1.31, 1.55),
                    mi=math.exp(rng.uniform(math.log(1e-7), math.log(1e-2))), a1=a1, a2=a2, r1=r1, r2=r2,
                    n_int2=case["n_int"], n_quad=case["n_quad"], n_angles=case["n_angles"])
    if kind == "solve":
        return [dataclasses.replace(base, **_options(case))]
    # reweight: the distributions the loop tries, for the kernels of `base`
    return [dataclasses.replace(base, derivs=abi.deriv_unit("a1", "a2"), a1=a1 * f, a2=a2 * g)
            for f, g in zip(rng.uniform(0.9, 1.0, case["calls"]), rng.uniform(0.9, 1.1, case["calls"]))]


class _Problems:
    """The library's input and output structures for a list of abi.Case, the
    outputs in flat arrays of the caller's: per kind one array over all cases,
    each case's block in the library's layout ([6][max_coef], [nd][6][max_coef],
    ...)."""

    def __init__(self, cases, **extra):
        lib = lmie_b200.library()
        n, nd = len(cases), cases[0].n_derivs
        self.lib, self.n, self.nd = lib, n, nd
        self.blocks = [abi.InputBlock(dataclasses.replace(c, **extra)) for c in cases]
        self.ins = (abi.lmie_in_data * n)(*[b.s for b in self.blocks])
        self.outs = (abi.lmie_out_data * n)()
        mc = np.array([_n1(c) * 2 for c in cases])
        na = np.array([c.n_angles for c in cases])
        self.keep, self.arrays = [], {}
        fields = np.frombuffer(self.outs, dtype=np.uint8).reshape(n, -1)
        self.arrays["n_coef"] = fields[:, :4].view(np.int32)[:, 0]
        scal = fields[:, 8:8 + 8 * SCALARS].view(np.float64)
        self.arrays["size"], self.arrays["cross"] = scal[:, :9], scal[:, 9:]
        if nd:
            lin = np.zeros((SCALARS, n, nd))
            self.arrays["size_l"], self.arrays["cross_l"] = lin[:9], lin[9:]
            for f, name in enumerate(abi._OUT_SCALARS):
                for i in range(n):
                    setattr(self.outs[i], name + "_l", C.cast(lin[f, i].ctypes.data, PD))
        c0 = cases[0]
        for name, on, cols in (("gc", c0.calc_gc, mc), ("lc", c0.calc_lc, mc), ("pf", c0.calc_pf, na)):
            if on:
                self._rows(name, 1, cols)
                if nd:
                    self._rows(name + "_l", nd, cols)
        if c0.calc_pf:
            th = np.zeros(int(na.sum()))
            self.arrays["theta"] = th
            for i, o in enumerate(np.cumsum(na) - na):
                self.outs[i].theta = C.cast(th.ctypes.data + 8 * int(o), PD)

    def _rows(self, name, lead, cols):
        data = np.zeros(int(cols.sum()) * lead * 6)
        first = np.cumsum(cols) - cols
        row = first[:, None] * (lead * 6) + np.arange(lead * 6)[None, :] * cols[:, None]
        rows = (data.ctypes.data + 8 * row).astype(np.uint64)                  # [n, lead * 6] row addresses
        self.keep.append(rows)
        self.arrays[name] = data
        planes = rows.ctypes.data + 8 * (np.arange(self.n)[:, None] * (lead * 6) + 6 * np.arange(lead)[None, :])
        planes = planes.astype(np.uint64)
        self.keep.append(planes)
        for i in range(self.n):
            if name.endswith("_l"):
                setattr(self.outs[i], name, C.cast(planes.ctypes.data + 8 * lead * i, abi.PPPD))
            else:
                setattr(self.outs[i], name, C.cast(int(planes[i, 0]), abi.PPD))


class _Kernels:
    """The save1 / save2 arrays of a save_control = 1 solve (the caller's to free)."""

    def __init__(self, case):
        lib = lmie_b200.library()
        p = _Problems([dataclasses.replace(case, save_control=1)])
        if lib.lmie_solution(C.byref(p.ins[0]), C.byref(p.outs[0]), 0, 0, THREADS, 0) != 0:
            raise RuntimeError("lmie_solution failed")
        self.save1, self.save2 = p.outs[0].save1, p.outs[0].save2
        self.free = C.CDLL(None).free
        self.free.argtypes, self.free.restype = [C.c_void_p], None

    def __del__(self):
        for s in (self.save1, self.save2):
            self.free(C.cast(s, C.c_void_p))


def _adjoint_problem(case, seed):
    return workloads.adjoint_retrieval(case["n_lambda"], case["n_bins"], case["n_quad"], case["n_angles"], seed=seed)


def _spheres_inputs(case, seed):
    """wavelength, m, radii: log-spaced sizes up to x_max in a shuffled order"""
    rng = np.random.Generator(np.random.PCG64(seed))
    lam = float(rng.uniform(0.34, 2.1))
    x = np.exp(rng.uniform(math.log(min(0.1, 0.1 * case["x_max"])), math.log(case["x_max"]), case["n_radii"]))
    return lam, float(rng.uniform(1.31, 1.6)), float(math.exp(rng.uniform(-16.0, -3.0))), x * lam / (2.0 * math.pi)


def prepare(case, seed):
    kind, lib = case["kind"], lmie_b200.library()
    if kind == "spheres":
        lam, mr, mi, r = _spheres_inputs(case, seed)
        radius = torch.from_numpy(r).cuda()
        out = torch.zeros(4, case["n_radii"], dtype=torch.float64, device="cuda")
        f = lib.lmie_cross_sections_noalloc
        f.restype = C.c_int
        f.argtypes = [C.c_int, C.c_void_p, C.c_double, C.c_double, C.c_double, C.c_void_p, C.c_void_p]
        stream = torch.cuda.current_stream().cuda_stream
        args = (case["n_radii"], radius.data_ptr(), lam, mr, mi, out.data_ptr(), stream)
        return dict(call=lambda: f(*args), out=out, keep=radius)
    if kind == "adjoint":
        p = _adjoint_problem(case, seed)
        f = lib.lmie_solution_adjoint
        f.restype = C.c_int
        f.argtypes = [C.c_int, PD, PD, PD, C.c_void_p, C.c_int, C.c_void_p, PD, PD, PD, PD, PD]
        ptr = lambda a: a.ctypes.data_as(PD)  # noqa: E731
        bins = lmie_b200.lmie_bins(p.n_bins, p.n_quad, ptr(p.edges), ptr(p.weight))
        w = (lmie_b200.lmie_loss_weights * p.n_lambda)()
        for k in range(p.n_lambda):
            w[k] = lmie_b200.lmie_loss_weights(*p.c[k], ptr(p.d11[k]), ptr(p.d12[k]))
        out = dict(loss=np.zeros(1), grad_mr=np.zeros(p.n_lambda), grad_mi=np.zeros(p.n_lambda),
                   grad_weight=np.zeros(p.n_bins), values=np.zeros((p.n_lambda, 3 + 2 * p.n_angles)))
        args = (p.n_lambda, ptr(p.lam), ptr(p.mr), ptr(p.mi), C.addressof(bins), p.n_angles, C.addressof(w),
                *[ptr(a) for a in out.values()])
        return dict(call=lambda: f(*args), out=out, keep=(p, bins, w))
    cases = _cases(case, seed)
    if kind == "reweight":
        p = _Problems(cases, save_control=2)
        kernels = _Kernels(cases[0])
        for o in p.outs:
            o.save1, o.save2 = kernels.save1, kernels.save2
        solve = lib.lmie_solution
        args = [(C.byref(p.ins[i]), C.byref(p.outs[i]), 0, 0, THREADS, 0) for i in range(p.n)]
        return dict(call=lambda: max(abs(solve(*a)) for a in args), out=p.arrays, keep=(p, kernels))
    p = _Problems(cases)
    if kind == "solve":
        args = (C.byref(p.ins[0]), C.byref(p.outs[0]), 0, 0, THREADS, 0)
        return dict(call=lambda: lib.lmie_solution(*args), out=p.arrays, keep=p)
    f = lib.lmie_solution_batch2
    f.restype = C.c_int
    f.argtypes = [C.c_int, C.POINTER(abi.lmie_in_data), C.POINTER(abi.lmie_out_data)] + [C.c_int] * 4
    args = (p.n, p.ins, p.outs, 0, 0, THREADS, PRECISION[case["precision"]])
    return dict(call=lambda: f(*args), out=p.arrays, keep=p)


def run(state):
    if state["call"]() != 0:
        raise RuntimeError("the library returned an error")
    return state["out"]


# ---------------------------------------------------------------------------
# work
# ---------------------------------------------------------------------------
def _order(x):
    """The truncation n1 of size parameter x."""
    x = np.asarray(x, dtype=np.float64)
    return (x + 4.05 * np.power(x, 1.0 / 3.0) + 8).astype(np.int64)


def _order2(n1, az):
    t = np.maximum(n1.astype(np.float64), az)
    return (t + 6.40 * np.power(t, 1.0 / 3.0) + 8).astype(np.int64)


def _n1(c):
    return int(_order(2.0 * math.pi * c.r2 / c.lam))


def _radii(c):
    """The quadrature of a case's distribution: radii and interval weights."""
    if c.dist == "mono":
        return np.array([c.a1]), np.array([1.0])
    t, w = _unit_gauss(c.n_quad)
    h = (c.r2 - c.r1) / c.n_int2
    lo = c.r1 + h * np.arange(c.n_int2)
    return ((lo + 0.5 * h)[:, None] + 0.5 * h * t).reshape(-1), np.tile(0.5 * h * w, c.n_int2)


def _recurrence_flops(x, az, ncol):
    n1 = _order(x)
    return float(np.sum(93.0 * n1 + 14.0 * _order2(n1, az) + ncol * (154.0 * n1 + 16.0 * _order2(n1, az))))


def work(case):
    """Bytes of the inputs and outputs; the recurrences, the sums over orders
    at every Gauss angle (8 flops per angle, order, radius and column) and the
    expansions."""
    kind = case["kind"]
    if kind == "spheres":
        x = 2.0 * math.pi * _spheres_inputs(case, 1)[3] / _spheres_inputs(case, 1)[0]
        return {"bytes": 40.0 * case["n_radii"], "flops": _recurrence_flops(x, 1.5 * x, 0)}
    if kind == "adjoint":
        p = _adjoint_problem(case, 1)
        r = np.repeat(p.edges[1:], p.n_quad)
        flops = 0.0
        for lam in p.lam:
            x = 2.0 * math.pi * r / lam
            # forward sweep, its reverse, and the angular sums in both directions
            flops += 2.0 * _recurrence_flops(x, 1.5 * x, 0) + 16.0 * p.n_angles * float(np.sum(_order(x)))
        return {"bytes": 8.0 * p.n_lambda * (8 + 4 * p.n_angles), "flops": flops}
    nbytes = flops = 0.0
    for c in _cases(case, 1):
        nd1 = sum(1 for d in c.derivs if "mr" in d or "mi" in d)
        ncol, mc = 1 + c.n_derivs, 2 * _n1(c)
        x = 2.0 * math.pi * _radii(c)[0] / c.lam
        on = c.calc_gc or c.calc_lc
        nbytes += 300.0 + 8.0 * ncol * (13 + (6 * mc if on else 0) + 6 * c.n_angles)
        if kind == "reweight":
            nbytes += 32.0 * len(x) * (mc + 1)
            flops += 8.0 * len(x) * mc * ncol
        else:
            flops += _recurrence_flops(x, c.mr * x, nd1)
            if on:
                flops += 8.0 * mc * float(np.sum(_order(x))) * (1 + nd1)
        if on:
            flops += 12.0 * mc * ncol * (mc + c.n_angles)
    return {"bytes": nbytes, "flops": flops}


# ---------------------------------------------------------------------------
# the same quantities in plain FP64
# ---------------------------------------------------------------------------
def _device():
    return torch.device("cuda" if torch.cuda.is_available() else "cpu")


def _t(a, dtype=torch.float64):
    return torch.as_tensor(np.ascontiguousarray(a), dtype=dtype, device=_device())


def _gauss_flat(counts):
    """Gauss-Legendre nodes (ascending) and weights of every count, one after
    another: Newton's iteration on P_n over all nodes at once."""
    counts = np.asarray(counts)
    n = np.repeat(counts, counts).astype(np.float64)
    i = np.concatenate([np.arange(c) for c in counts]).astype(np.float64)
    x0 = -(1.0 - (n - 1.0) / (8.0 * n ** 3)) * np.cos(math.pi * (4.0 * i + 3.0) / (4.0 * n + 2.0))
    x, nn = _t(x0), _t(n)

    def legendre(x):
        p0, p1 = torch.ones_like(x), x.clone()
        for k in range(1, int(counts.max())):
            p2 = p1 * x + (p1 * x - p0) * (k / (k + 1.0))
            more = nn > k
            p0, p1 = torch.where(more, p1, p0), torch.where(more, p2, p1)
        return p1, nn * (p0 - x * p1) / ((1.0 - x) * (1.0 + x))

    for _ in range(4):
        p, dp = legendre(x)
        x = x - torch.where(nn > 1, p / dp, x)
    _, dp = legendre(x)
    return x, 2.0 / ((1.0 - x) * (1.0 + x) * dp * dp)


@functools.lru_cache(maxsize=None)
def _unit_gauss(n):
    x, w = _gauss_flat([n])
    return x.cpu().numpy(), w.cpu().numpy()


def _mie(x, m, deriv):
    """a_n, b_n (n = 1 .. largest n1; zero past a radius' own n1) of the size
    parameters x and refractive indices m, and their derivatives w.r.t. m."""
    n1 = _order(x)
    n2 = _order2(n1, np.abs(m * x))
    N = int(n1.max())
    xt, mt = _t(x), _t(m, torch.complex128)
    k1, k2 = _t(n1), _t(n2)
    z = mt * xt
    D = torch.zeros_like(z)
    Dl = torch.zeros_like(z)
    Ds, Dls = [None] * (N + 1), [None] * (N + 1)
    for j in range(int(n2.max()) - 1, 0, -1):
        on = k2 > j
        c1 = (j + 1.0) / z
        c2 = D + c1
        if deriv:
            c5 = -c1 / z * xt
            Dl = torch.where(on, c5 + (Dl + c5) / (c2 * c2), Dl)
        D = torch.where(on, c1 - 1.0 / c2, D)
        if j <= N:
            Ds[j], Dls[j] = D, Dl
    rn, ratio = torch.zeros_like(xt), [None] * (N + 1)
    ratio[N] = rn
    for j in range(N - 1, 0, -1):
        rn = torch.where(k1 > j, 1.0 / ((2.0 * j + 1.0) / xt - rn), rn)
        ratio[j] = rn
    shape = (N, len(x))
    out = [torch.zeros(shape, dtype=torch.complex128, device=xt.device) for _ in range(4 if deriv else 2)]
    psi_p, chi_p = torch.sin(xt), torch.cos(xt)
    chi = chi_p / xt + psi_p
    for j in range(1, N + 1):
        on = k1 >= j
        psi = ratio[j] * psi_p
        zeta, zeta_p = torch.complex(psi, chi), torch.complex(psi_p, chi_p)
        D, Dl = Ds[j], Dls[j]
        ca, cb = D / mt + j / xt, D * mt + j / xt
        da, db = 1.0 / (ca * zeta - zeta_p), 1.0 / (cb * zeta - zeta_p)
        out[0][j - 1] = torch.where(on, (ca * psi - psi_p) * da, 0.0)
        out[1][j - 1] = torch.where(on, (cb * psi - psi_p) * db, 0.0)
        if deriv:      # psi_{n-1} chi_n - psi_n chi_{n-1} = 1
            out[2][j - 1] = torch.where(on, 1j * da * da * (Dl / mt - D / (mt * mt)), 0.0)
            out[3][j - 1] = torch.where(on, 1j * db * db * (D + mt * Dl), 0.0)
        psi_p, chi_p, chi = psi, chi, torch.where(on, (2.0 * j + 1.0) / xt * chi - chi_p, chi)
    return out


def _sums(ab):
    """Per radius: extinction, scattering, backscatter and asymmetry sums, and
    (Re, Im) = (d/dmr, d/dmi) of each as complex numbers when ab has derivatives."""
    a, b = ab[0], ab[1]
    N = a.shape[0]
    n = torch.arange(1, N + 1, dtype=torch.float64, device=a.device)[:, None]
    f1, f3, f4 = 2 * n + 1, n * (n + 2) / (n + 1), (2 * n + 1) / (n * (n + 1))
    sg = 1.0 - 2.0 * (n % 2)
    sb = (f1 * sg * (a - b)).sum(0)
    g = (f3[:-1] * (a[:-1] * a[1:].conj() + b[:-1] * b[1:].conj())).sum(0) + (f4[:-1] * a[:-1] * b[:-1].conj()).sum(0)
    val = [(f1 * (a + b)).sum(0).real, (f1 * (a.abs() ** 2 + b.abs() ** 2)).sum(0), sb.abs() ** 2, g.real]
    if len(ab) == 2:
        return val, None
    da, db = ab[2], ab[3]
    lin = [(f1 * (da + db)).sum(0), (2 * f1 * (a.conj() * da + b.conj() * db)).sum(0),
           2 * sb.conj() * (f1 * sg * (da - db)).sum(0),
           (f3[:-1] * (da[:-1] * a[1:].conj() + a[:-1].conj() * da[1:] + db[:-1] * b[1:].conj() +
                       b[:-1].conj() * db[1:])).sum(0) +
           (f4[:-1] * (da[:-1] * b[:-1].conj() + a[:-1].conj() * db[:-1])).sum(0)]
    return val, lin


def _pi_tau(mu, N):
    """pi_n + tau_n and pi_n - tau_n, [N][len(mu)], n = 1 .. N."""
    plus = torch.empty(N, len(mu), dtype=torch.float64, device=mu.device)
    minus = torch.empty_like(plus)
    p0, p1 = torch.zeros_like(mu), torch.ones_like(mu)
    for k in range(1, N + 1):
        t = mu * p1 - p0
        tau = k * t - p0
        plus[k - 1], minus[k - 1] = p1 + tau, p1 - tau
        p0, p1 = p1, mu * p1 + (k + 1.0) / k * t
    return plus, minus


def _phase(plus, minus, ab):
    """The four phase-matrix kernels of each radius at the angles of plus and
    minus ([orders][angles]), [4][angles][radii], and their derivatives."""
    N = plus.shape[0]
    n = torch.arange(1, N + 1, dtype=torch.float64, device=plus.device)[:, None]
    f4 = (2 * n + 1) / (n * (n + 1))
    q = [v[:N] for v in ab]

    def contract(basis, c):
        r = basis.T @ torch.view_as_real(f4 * c).reshape(N, -1)
        return torch.view_as_complex(r.reshape(basis.shape[1], -1, 2).contiguous())

    sp, sm = contract(plus, q[0] + q[1]), contract(minus, q[0] - q[1])
    A, Bm, Cc, Dd = sp.abs() ** 2, sm.abs() ** 2, (sp * sm.conj()).real, (sm * sp.conj()).imag
    val = [(A + Bm) / 4, (A - Bm) / 4, -Cc / 2, Dd / 2]
    if len(ab) == 2:
        return val, None
    dp, dm = contract(plus, q[2] + q[3]), contract(minus, q[2] - q[3])
    A, Bm = 2 * sp.conj() * dp, 2 * sm.conj() * dm
    Cc, Dd = sm.conj() * dp + sp.conj() * dm, 1j * (sm.conj() * dp - sp.conj() * dm)
    return val, [(A + Bm) / 4, (A - Bm) / 4, -Cc / 2, Dd / 2]


def _gsf(mu, nl):
    """The generalised spherical functions P00, P0+2, P2+2, P2-2, [4][nl][len(mu)]."""
    P = torch.zeros(4, nl, len(mu), dtype=torch.float64, device=mu.device)
    P[0, 0], P[0, 1], P[0, 2] = 1.0, mu, (3.0 * mu * mu - 1.0) / 2.0
    P[1, 2] = 0.25 * math.sqrt(6.0) * (mu * mu - 1.0)
    P[2, 2], P[3, 2] = 0.25 * (1.0 + mu) ** 2, 0.25 * (1.0 - mu) ** 2
    for j in range(2, nl - 1):
        t, q = (2.0 * j + 1.0) * mu, (j + 1.0) ** 2 - 4.0
        P[0, j + 1] = (t * P[0, j] - j * P[0, j - 1]) / (j + 1.0)
        P[1, j + 1] = (t * P[1, j] - math.sqrt(j * j - 4.0) * P[1, j - 1]) / math.sqrt(q)
        u, v, b = j * (j + 1.0) * t, 4.0 * (2.0 * j + 1.0), (j + 1.0) * (j * j - 4.0)
        P[2, j + 1] = ((u - v) * P[2, j] - b * P[2, j - 1]) / (j * q)
        P[3, j + 1] = ((u + v) * P[3, j] - b * P[3, j - 1]) / (j * q)
    return P


def _weights(c, r, qw):
    """n(r) qw of every output column ([1 + nd][radii]) and the distribution's scalars."""
    if c.dist == "mono":
        nr, unit = np.ones(1), {}
        norm = 1.0
    else:
        if c.dist == "gamma":
            e = (1.0 - 3.0 * c.a2) / c.a2
            nr = r ** e * np.exp(-r / (c.a1 * c.a2))
            unit = {"a1": r / (c.a1 ** 2 * c.a2), "a2": -np.log(r) / c.a2 ** 2 + r / (c.a1 * c.a2 ** 2)}
        else:
            d = np.log(r / c.a1)
            nr = np.exp(-d * d / (2.0 * c.a2)) / r
            unit = {"a1": d / (c.a2 * c.a1), "a2": d * d / (2.0 * c.a2 ** 2)}
        norm = float(np.sum(nr * qw))
        nr = nr / norm
    f = nr * qw
    w = [f]
    for d in c.derivs:
        (name,) = d
        g = unit.get(name, 0.0 * r)
        w.append(f * (g - np.sum(f * g)))
    s = [float(np.sum(f * r ** k)) for k in range(5)]
    reff = s[3] / s[2]
    size = [c.a1 if c.dist == "mono" else c.r1, c.a1 if c.dist == "mono" else c.r2, norm, reff,
            float(np.sum(f * (r - reff) ** 2 * r * r)) / (s[2] * reff ** 2), math.pi * s[2],
            4.0 / 3.0 * math.pi * s[3], s[1], s[4] / s[3]]
    return np.stack(w), size


def _solve_exact(c, r, w, ab, plus, minus, P, Pu, qw, out):
    """One case: ab [orders][its radii], the bases at its Gauss angles, the
    user-angle functions Pu; appends its outputs to the lists of `out`."""
    names = [next(iter(d)) for d in c.derivs]
    w = _t(w)
    val, lin = _sums(ab)

    def columns(v, g):
        """weighted radius sums of v ([..][radii]) for every column: [1 + nd][..]"""
        cols = [v @ w[0]]
        for k, name in enumerate(names):
            s = v @ w[1 + k]
            if name in ("mr", "mi"):
                s = s + (g.real if name == "mr" else g.imag) @ w[0]
            cols.append(s)
        return torch.stack(cols)

    e, s, b, g = (columns(v, lin[q] if lin else None) for q, v in enumerate(val))
    lam = c.lam * c.lam / (2.0 * math.pi)
    S = s[0]
    gn = 2.0 * g / S
    gn[1:] -= 2.0 * g[0] * s[1:] / S ** 2
    cross = torch.stack([e * lam, s * lam, b * lam / (8.0 * math.pi), gn]).cpu().numpy()
    out["cross"].append(cross[:, 0])
    out["cross_l"].append(cross[:, 1:])
    if not (c.calc_gc or c.calc_lc):
        out["n_coef"].append(0)
        return
    n_q, nl = plus.shape[1], 2 * plus.shape[0]
    F = torch.zeros(4, 1 + c.n_derivs, n_q, dtype=torch.float64, device=plus.device)
    step = max(1, int(24e6) // n_q)
    w_all = w
    for r0 in range(0, len(r), step):
        part = slice(r0, r0 + step)
        w = w_all[:, part]
        v, gl = _phase(plus, minus, [q[:, part] for q in ab])
        for el in range(4):
            F[el] += columns(v[el], gl[el] if gl else None)
    F = 2.0 * F / S
    F[:, 1:] -= F[:, :1] * (s[1:] / S)[None, :, None]
    l = torch.arange(nl, dtype=torch.float64, device=F.device)
    Fw = F * qw
    scale = (2.0 * l + 1.0) / 2.0
    if c.calc_gc:
        t = (Fw[0] + Fw[1]) @ P[2].T
        u = (Fw[0] - Fw[1]) @ P[3].T
        co = torch.stack([Fw[0] @ P[0].T, (t + u) / 2, (t - u) / 2, Fw[1] @ P[0].T, Fw[2] @ P[1].T, Fw[3] @ P[1].T])
    else:
        co = torch.stack([Fw[q] @ P[0].T for q in (0, 0, 1, 1, 2, 3)])
        co[5] = -co[5]
    co = (co * scale).transpose(0, 1).contiguous()           # [1 + nd][6][nl]
    co[1:, 0, 0] = 0.0
    small = (co[0, 0].abs() <= c.accuracy).nonzero()
    n = int(small[0]) + 1 if len(small) else nl
    out["n_coef"].append(n)
    pf = torch.empty(1 + c.n_derivs, 6, c.n_angles, dtype=torch.float64, device=F.device)
    k = co[:, :, :n]
    p = Pu[:, :n]
    if c.calc_gc:
        t, u = (k[:, 1] + k[:, 2]) @ p[2], (k[:, 1] - k[:, 2]) @ p[3]
        for el, v in enumerate((k[:, 0] @ p[0], (t + u) / 2, (t - u) / 2, k[:, 3] @ p[0], k[:, 4] @ p[1],
                                k[:, 5] @ p[1])):
            pf[:, el] = v
    else:
        for el in range(6):
            pf[:, el] = k[:, el] @ p[0] * (-1.0 if el == 5 else 1.0)
    kind = "gc" if c.calc_gc else "lc"
    for name, v in ((kind, co), ("pf", pf)):
        v = v.cpu().numpy()
        out[name].append(v[0].reshape(-1))
        out[name + "_l"].append(v[1:].reshape(-1))


def _solves_exact(cases):
    out = {k: [] for k in ("n_coef", "size", "cross", "cross_l", "gc", "gc_l", "lc", "lc_l", "pf", "pf_l")}
    done = {k: [None] * len(cases) for k in out}
    n1 = np.array([_n1(c) for c in cases])
    quad = [_radii(c) for c in cases]
    order = np.argsort(n1, kind="stable")
    on = cases[0].calc_gc or cases[0].calc_lc
    deriv = any(next(iter(d)) in ("mr", "mi") for d in cases[0].derivs)
    at = 0
    while at < len(order):
        # as many cases as share one pass of the recurrences within a few GB
        end = at + 1
        while end < len(order):
            idx = order[at:end + 1]
            if n1[idx[-1]] * sum(len(quad[i][0]) for i in idx) > 2e7 or n1[idx[-1]] * n1[idx].sum() > 1.6e7:
                break
            end += 1
        idx = order[at:end]
        x = np.concatenate([2.0 * math.pi * quad[i][0] / cases[i].lam for i in idx])
        m = np.concatenate([np.full(len(quad[i][0]), complex(cases[i].mr, -cases[i].mi)) for i in idx])
        ab = _mie(x, m, deriv)
        if on:
            mu, qw = _gauss_flat(2 * n1[idx])
            plus, minus = _pi_tau(mu, int(n1[idx].max()))
            P = _gsf(mu, 2 * int(n1[idx].max()))
            user = _t(np.cos(np.arange(cases[0].n_angles) * (math.pi / (cases[0].n_angles - 1))))
            Pu = _gsf(user, 2 * int(n1[idx].max()))
        r_at = q_at = 0
        for i in idx:
            c, (r, q), n = cases[i], quad[i], n1[i]
            w, size = _weights(c, r, q)
            for v in out.values():
                v.clear()
            rs, qs = slice(r_at, r_at + len(r)), slice(q_at, q_at + 2 * n)
            part = [v[:n, rs] for v in ab]
            if on:
                _solve_exact(c, r, w, part, plus[:n, qs], minus[:n, qs], P[:, :2 * n, qs], Pu, qw[qs], out)
                q_at += 2 * n
            else:
                _solve_exact(c, r, w, part, None, None, None, None, None, out)
            r_at += len(r)
            out["size"].append(size)
            for k, v in out.items():
                if v:
                    done[k][i] = v[0]
        at = end
    c0 = cases[0]
    res = {"n_coef": np.array(done["n_coef"], dtype=np.int32), "size": np.array(done["size"]),
           "cross": np.array(done["cross"])}
    names = (["gc"] if c0.calc_gc else []) + (["lc"] if c0.calc_lc else []) + (["pf"] if c0.calc_pf else [])
    for name in names:
        res[name] = np.concatenate(done[name])
        if c0.n_derivs:
            res[name + "_l"] = np.concatenate(done[name + "_l"])
    if c0.n_derivs:
        res["cross_l"] = np.stack(done["cross_l"], axis=1)
        res["size_l"] = None
    if c0.calc_pf:
        res["theta"] = np.concatenate([np.arange(c.n_angles) * (180.0 / (c.n_angles - 1)) for c in cases])
    return res


def _adjoint_exact(p):
    t, q = _unit_gauss(p.n_quad)
    lo, hi = p.edges[:-1, None], p.edges[1:, None]
    r = (0.5 * (lo + hi) + 0.5 * (hi - lo) * t).reshape(-1)
    q = (0.5 * (hi - lo) * q).reshape(-1)
    W = _t(np.repeat(p.weight, p.n_quad) * q)
    Nt = W.sum()
    mu = _t(np.cos(np.arange(p.n_angles) * (math.pi / (p.n_angles - 1))))
    loss, gm, values = 0.0, [], []
    gw = torch.zeros(len(r), dtype=torch.float64, device=W.device)
    step = max(1, int(2e7) // (int(_order(2.0 * math.pi * r.max() / p.lam.min())) * len(r)))
    for k0 in range(0, p.n_lambda, step):
        ks = range(k0, min(p.n_lambda, k0 + step))
        x = np.concatenate([2.0 * math.pi * r / p.lam[k] for k in ks])
        m = np.repeat(np.array([complex(p.mr[k], -p.mi[k]) for k in ks]), len(r))
        ab = _mie(x, m, True)
        val, lin = _sums(ab)
        plus, minus = _pi_tau(mu, ab[0].shape[0])
        for i, k in enumerate(ks):
            s = slice(i * len(r), (i + 1) * len(r))
            F, dF = _phase(plus, minus, [v[:, s] for v in ab])
            d = [_t(p.d11[k]), _t(p.d12[k])]
            e, sc, g = (val[j][s] for j in (0, 1, 3))
            de, ds, dg = (lin[j][s] for j in (0, 1, 3))
            phi = d[0] @ F[0] + d[1] @ F[2]
            dphi = d[0].to(dF[0].dtype) @ dF[0] + d[1].to(dF[0].dtype) @ dF[2]
            kap, (ce, cs, cg) = p.lam[k] ** 2 / (2.0 * math.pi), p.c[k]
            E, S, G, Phi = W @ e, W @ sc, W @ g, W @ phi
            loss += float(kap * (ce * E + cs * S) / Nt + 2 * (cg * G + Phi) / S)
            gw += kap * (ce * e + cs * sc) / Nt - kap * (ce * E + cs * S) / Nt ** 2
            gw += 2 * (cg * g + phi) / S - 2 * (cg * G + Phi) / S ** 2 * sc
            Wc = W.to(de.dtype)
            gm.append(complex(kap * (ce * (Wc @ de) + cs * (Wc @ ds)) / Nt + 2 * (cg * (Wc @ dg) + Wc @ dphi) / S -
                              2 * (cg * G + Phi) / S ** 2 * (Wc @ ds)))
            head = torch.stack([kap * E / Nt, kap * S / Nt, 2 * G / S])
            values.append(torch.cat([head, 2 * (F[0] @ W) / S, 2 * (F[2] @ W) / S]).cpu().numpy())
    gm = np.array(gm)
    gw = (gw.cpu().numpy() * q).reshape(p.n_bins, p.n_quad).sum(1)
    return dict(loss=np.array([loss]), grad_mr=gm.real.copy(), grad_mi=gm.imag.copy(), grad_weight=gw,
                values=np.stack(values))


def exact(case, seed):
    if case["kind"] == "spheres":
        lam, mr, mi, r = _spheres_inputs(case, seed)
        x = 2.0 * math.pi * r / lam
        e, s, b, g = _sums(_mie(x, np.full(len(x), complex(mr, -mi)), False))[0]
        k = lam * lam / (2.0 * math.pi)
        return torch.stack([e * k, s * k, b * k / (8.0 * math.pi), 2.0 * g / s])
    if case["kind"] == "adjoint":
        return _adjoint_exact(_adjoint_problem(case, seed))
    return _solves_exact(_cases(case, seed))
