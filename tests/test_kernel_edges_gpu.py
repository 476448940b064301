"""The kernels at the sizes where their tiles, groups and blocks end, and the
forms of a stage against each other.

Tolerances, fixed before the first run.  Against the oracle: the parity
tests' 1e-10 (rounding of n_max ~ 300 dependent steps, 1e-13, times a thousand
for nearly singular psi and for derivatives).  A case in a batch against the
same case alone, fixed-point sums against FP64 ones: an operand is rounded to
2^-49 of the largest one of its row or column, which summed over 130 orders is
2e-13 of the largest product; the phase matrix divides by at most a tenth of
it, and a linearised one may cancel two more digits: 1e-11 and 1e-9.
"""
import ctypes as C
import dataclasses

import numpy as np
import pytest

import adjoint_oracle
import libs
import lmie_b200
from lmie_b200 import abi, workloads
from lmie_b200.abi import deriv_unit
from test_parity_gpu import _reweight

pytestmark = pytest.mark.gpu

TOL = 1e-10


def n1(x):
    """The reference's truncation n1 of a size parameter above 8 (src/lmie_core.c:18-38)."""
    return int(x + 4.05 * x ** (1. / 3.) + 2.)


def x_of(orders):
    """A size parameter whose truncation is `orders`, away from multiples of pi."""
    x = 8.05
    while n1(x) < orders:
        x += 0.01
    x += 0.2
    while abs(np.sin(x)) < 0.3:
        x += 0.01
    assert n1(x) == orders
    return x


def gamma(x, lam=0.7, **kw):
    r2 = x * lam / (2. * np.pi)
    return abi.Case(dist="gamma", lam=lam, a1=0.35 * r2, a2=0.12, r1=1e-3 * r2, r2=r2, **kw)


def mono(x, lam=0.7, **kw):
    r = x * lam / (2. * np.pi)
    return abi.Case(dist="mono", lam=lam, a1=r, r1=r, r2=r, n_quad=1, **kw)


def assert_close(got, want, tol, label, tol_l=None):
    assert got.rc == 0 and want.rc == 0, label
    err = libs.compare(got, want)
    bad = {k: v for k, v in err.items() if k != "n_coef" and v > ((tol_l or tol) if k.endswith("_l") else tol)}
    assert not bad and err["n_coef"] == 0, (label, bad, err["n_coef"])


# one radius: the whole block forms its orders, 128 at a time, and the orders
# of the expansion in tiles of 32, those of the user angles in 64s
@pytest.mark.parametrize("orders, n_angles, derivs", [(31, 63, ("mr",)), (32, 64, ("mr", "mi")), (33, 65, ("lambda", "mi")),
                                                      (127, 1, ("mi",)), (129, 181, ("mr", "mi")),
                                                      (256, 129, ()), (257, 128, ("mr",))])
def test_one_radius(orders, n_angles, derivs):
    case = mono(x_of(orders), mr=1.37, mi=0.02, derivs=deriv_unit(*derivs), n_angles=max(n_angles, 2), calc_lc=1)
    assert_close(libs.run_product(case), libs.run_oracle(case), TOL, (orders, n_angles, derivs))


@pytest.mark.parametrize("x, mr, mi", [(0.05, 1.33, 0.), (3.3, 8., 0.5), (20.3, 4., 3.)])
def test_one_radius_far_from_usual(x, mr, mi):
    """Very small spheres and indices for which D starts long before psi."""
    case = mono(x, mr=mr, mi=mi, derivs=deriv_unit("mr", "mi"), calc_gc=0, calc_pf=0)
    assert_close(libs.run_product(case), libs.run_oracle(case), TOL, (x, mr, mi))


# several radii to a block, a warp per radius (a mean below 400 orders) or the
# block for each (above); with the m, the x and both columns
@pytest.mark.parametrize("orders, n_quad, derivs", [(34, 593, ("mr",)), (65, 700, ("lambda",)), (130, 640, ("a1", "r2")), (1900, 600, ("mi",))])
def test_many_radii(orders, n_quad, derivs):
    case = gamma(x_of(orders), mr=1.41, mi=0.03, n_int2=1, n_quad=n_quad, derivs=deriv_unit(*derivs), calc_gc=0, calc_pf=0)
    assert_close(libs.run_product(case), libs.run_oracle(case), TOL, (orders, n_quad, derivs))


# FP64 batches large enough for the fixed-point sums: radius groups of 12, 6, 6
# and 4 with remainders, chunks of 32 orders, weights and x column or not
@pytest.mark.parametrize("derivs", [(), ("a1",), ("mr",), ("mr", "mi", "a1", "a2"), ("r2", "a2"), ("lambda", "mr"),
                                    ("lambda",)])
def test_fixed_point_batch_against_single_solves(derivs):
    rng = np.random.Generator(np.random.PCG64(3))
    cases = []
    for k in range(132):
        orders = (31, 32, 33, 64, 65, 97)[k % 6]
        cases.append(gamma(x_of(orders), mr=float(rng.uniform(1.33, 1.5)), mi=float(rng.uniform(0.005, 0.05)), n_int2=1,
                           n_quad=(49, 53, 61, 100, 59, 57)[k % 6], derivs=deriv_unit(*derivs), accuracy=1e-6, n_angles=37))
    got = abi.solve_batch(libs.product(), cases, precision=abi.PRECISION_FP64)
    for k in range(12):
        assert_close(got[k], libs.run_product(cases[k]), 1e-11, (derivs, k), 1e-9)


@pytest.mark.parametrize("n_bins, n_quad, n_angles", [(1, 31, 3), (3, 11, 16), (2, 16, 17), (1, 7, 47), (5, 1, 96),
                                                      (2, 17, 145), (1, 5, 193), (1, 3, 255)])
def test_adjoint_tiles(n_bins, n_quad, n_angles):
    """Half-angles in tiles of 8, radii in pairs and blocks of 32; the bounds of the adjoint's own tests at x ~ 40.
    (A single bin's weight cancels: its gradient is zero but for rounding.)"""
    p = workloads.adjoint_retrieval(n_lambda=2, n_bins=n_bins, n_quad=n_quad, n_angles=n_angles, lam_range=(0.5, 1.1),
                                    r_range=(0.05, 3.0))
    got, want = lmie_b200.adjoint(p), adjoint_oracle.solve(p)

    def rel(name):
        a, b = np.asarray(got[name], float), np.asarray(want[name], float)
        return float(np.max(np.abs(a - b)) / np.max(np.abs(b)))
    for name in ("cext", "csca", "g", "p11", "p12", "loss"):
        assert rel(name) <= 1e-10, (name, rel(name))
    for name in ("grad_mr", "grad_mi") + (("grad_weight",) if n_bins > 1 else ()):
        assert rel(name) <= 1e-8, (name, rel(name))


# radii dealt out to 32 rows, angles in 16s, columns in fours
@pytest.mark.parametrize("n_quad, orders, derivs", [(1, 20, ()), (31, 31, ("a1",)), (33, 33, ("a1", "a2", "a1")),
                                                    (64, 50, ("a1", "a2", "a1", "a2", "a1"))])
def test_reweighting(n_quad, orders, derivs):
    base = gamma(x_of(orders), mr=1.4, mi=0.01, n_int2=1, n_quad=n_quad, save_control=1, derivs=deriv_unit(*derivs))
    kept = libs.run_product(base)
    assert kept.rc == 0
    new = dataclasses.replace(base, a2=0.2, save_control=2)
    got = _reweight(libs.product(), "lmie", new, kept.save1, kept.save2)
    want = _reweight(libs.oracle(), "oracle", new, kept.save1, kept.save2)
    assert_close(got, want, TOL, (n_quad, orders, derivs))


@pytest.mark.parametrize("n", [1, 3, 1024])
def test_cross_sections_without_allocation(n):
    """Orders around the block's 128 and the largest accepted size, against the oracle."""
    import torch
    lam, mr, mi = 0.7, 1.39, 0.015
    xs = np.array(([x_of(128), 898.6, x_of(127), x_of(129)] + list(np.geomspace(0.1, 899., 1024)))[:n])
    radii = xs * lam / (2. * np.pi)
    d_r = torch.tensor(radii, device="cuda")
    d_out = torch.zeros(4, n, dtype=torch.float64, device="cuda")
    torch.cuda.synchronize()
    f = libs.product().lmie_cross_sections_noalloc
    f.restype = C.c_int
    f.argtypes = [C.c_int, C.c_void_p, C.c_double, C.c_double, C.c_double, C.c_void_p, C.c_void_p]
    assert f(n, d_r.data_ptr(), lam, mr, mi, d_out.data_ptr(), None) == 0
    got = d_out.cpu().numpy()
    for i in range(min(n, 5)):
        r = float(radii[i])
        want = libs.run_oracle(abi.Case(dist="mono", lam=lam, mr=mr, mi=mi, a1=r, r1=r, r2=r, n_quad=1, calc_gc=0, calc_pf=0))
        for q, name in enumerate(("cext", "csca", "cbak", "g")):
            assert abs(got[q, i] - want.scalars[name]) <= TOL * abs(want.scalars[name]), (xs[i], name)
