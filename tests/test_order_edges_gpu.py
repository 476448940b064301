"""The kernels at the orders where their chunks, rounds and tiles end.

The order counts are the library's own (lmie_calc_max_coef() is twice the
truncation of the largest radius).  K1 forms the orders of a radius 32 or 128
at a time, D in one of two ways below and above 32; the expansions go in tiles
of 32 and 64 coefficients; the fixed-point sums in chunks of 32 orders.

Tolerances, fixed before the first run.  Against the oracle: the parity tests'
1e-10 for values (rounding of some 300 dependent steps, 1e-13, times a thousand
for nearly singular psi); a derivative of a moderately absorbing sphere (mi
0.01 and more) loses another two digits, 1e-8.  For radii of 2100 orders both
are ten times as large.  Fixed-point sums with seven digits against the FP64
kernel: an operand is rounded to 2^-55 of the largest of its row or column, so
what differs is the FP64 kernel's own rounding of up to 128 terms, 2^-53 each:
1.5e-14 of the largest value of an expansion or a phase matrix, 1e-13 with a
margin; a derivative may cancel two digits of it, 1e-11.
"""
import ctypes as C
import functools
import math

import numpy as np
import pytest

import libs
from lmie_b200 import abi
from lmie_b200.abi import deriv_unit
from test_fp64_sums_gpu import _mono, fp64_kernel

pytestmark = pytest.mark.gpu

TOL, TOL_L = 1e-10, 1e-8
LAM = 0.7


def n1(x):
    """The library's truncation of size parameter x."""
    r = x * LAM / (2. * math.pi)
    case = abi.Case(dist="mono", lam=LAM, a1=r, r1=r, r2=r, n_quad=1)
    return libs.product().lmie_calc_max_coef(LAM, abi.InputBlock(case).s.dist_type, r, 0., 0., r, r) // 2


@functools.lru_cache(None)
def x_of(orders):
    """A size parameter of that many orders, away from the ends of its range and from multiples of pi."""
    x = 1.
    while n1(x) < orders:
        x += 0.01
    x += 0.2
    while abs(math.sin(x)) < 0.3:
        x += 0.01
    assert n1(x) == orders
    return x


def mono(orders, **kw):
    r = x_of(orders) * LAM / (2. * math.pi)
    return abi.Case(dist="mono", lam=LAM, a1=r, r1=r, r2=r, n_quad=1, **kw)


def gamma(orders, n_quad, **kw):
    r2 = x_of(orders) * LAM / (2. * math.pi)
    return abi.Case(dist="gamma", lam=LAM, a1=0.35 * r2, a2=0.12, r1=1e-2 * r2, r2=r2, n_int2=1, n_quad=n_quad, **kw)


def assert_close(got, want, label, tol=TOL, tol_l=TOL_L):
    assert got.rc == 0 and want.rc == 0, label
    err = libs.compare(got, want)
    bad = {k: v for k, v in err.items() if k != "n_coef" and v > (tol_l if k.endswith("_l") else tol)}
    assert not bad and err["n_coef"] == 0, (label, bad, err["n_coef"])


def test_the_order_counts_are_the_reference_formula():
    for x in (1., 7.9, 8.1, 45., 333.3, 2000.):
        assert n1(x) == int(x + 4.05 * x ** (1. / 3.) + 8)


@pytest.mark.parametrize("orders, n_angles, derivs", [(31, 63, ("mr",)), (32, 64, ()), (33, 65, ()), (33, 64, ("mr", "mi")),
                                                      (64, 37, ()), (65, 181, ("mi",)), (127, 19, ()), (128, 181, ("mr", "mi")),
                                                      (129, 33, ("mi",)), (256, 129, ()), (257, 128, ("mr",))])
def test_one_radius(orders, n_angles, derivs):
    case = mono(orders, mr=1.37, mi=0.02, derivs=deriv_unit(*derivs), n_angles=n_angles, calc_lc=1)
    assert_close(libs.run_product(case), libs.run_oracle(case), (orders, n_angles, derivs))


# a warp per radius: rounds of 32 orders; with the m, the x and both columns, and values only
@pytest.mark.parametrize("orders", [32, 33, 64, 65, 96])
@pytest.mark.parametrize("derivs", [(), ("mr",), ("lambda",), ("r2", "mi")])
def test_many_radii(orders, derivs):
    case = gamma(orders, 640, mr=1.41, mi=0.03, derivs=deriv_unit(*derivs), calc_gc=0, calc_pf=0)
    assert_close(libs.run_product(case), libs.run_oracle(case), (orders, derivs))


# the thread-per-radius form: long radii, and several rounds of blocks of them
@pytest.mark.parametrize("orders, n_quad, derivs", [(2150, 2600, ("mr",)), (2150, 11000, ())])
def test_a_thread_per_radius(orders, n_quad, derivs):
    case = gamma(orders, n_quad, mr=1.41, mi=0.03, derivs=deriv_unit(*derivs), calc_gc=0, calc_pf=0)
    assert_close(libs.run_product(case), libs.run_oracle(case), (orders, n_quad, derivs), 10. * TOL, 10. * TOL_L)


# seven digits: groups of 12, 6, 6 and 4 radii with remainders, last chunks of one order, of 31 and full ones
@pytest.mark.parametrize("derivs", [(), ("a1",), ("mr",), ("mr", "mi", "a1", "a2"), ("r2", "a2"), ("lambda", "mr"), ("lambda",)])
def test_fixed_point_sums_against_the_fp64_kernel(derivs):
    rng = np.random.Generator(np.random.PCG64(5))
    cases = [gamma((31, 32, 33, 64, 65, 96, 97)[k % 7], (49, 53, 61, 100, 59, 57, 48)[k % 7],
                   mr=float(rng.uniform(1.33, 1.5)), mi=float(rng.uniform(0.005, 0.05)), derivs=deriv_unit(*derivs),
                   accuracy=1e-6, n_angles=37) for k in range(133)]
    lib = libs.product()
    got = abi.solve_batch(lib, cases, precision=abi.PRECISION_FP64)
    for k in range(14):
        assert_close(got[k], fp64_kernel(cases[k]), (derivs, k), 1e-13, 1e-11)


def test_seven_digits_are_seven():
    """The median error of single radii's expansions, against the FP64 kernel, of 80 cases of some 60 orders: 64
    roundings of 2^-53 of random sign are 9e-16 of 2l + 1, twice that is the bound; six digits are beyond it."""
    lib = libs.product()
    cases = [_mono(np.random.Generator(np.random.PCG64(17 + k)), 20., 70.) for k in range(80)]
    ref = [fp64_kernel(c) for c in cases]
    med = {}
    for precision in (abi.PRECISION_FP64, abi.PRECISION_INT8):
        err = []
        for g, w in zip(abi.solve_batch(lib, cases, precision=precision), ref):
            err.append(float(np.max(np.abs(g.gc[0] - w.gc[0]) / (2. * np.arange(w.gc.shape[1]) + 1.))))
        med[precision] = float(np.median(err))
    assert med[abi.PRECISION_FP64] <= 16 * 2.**-53 < med[abi.PRECISION_INT8], med


@pytest.mark.parametrize("orders", [31, 32, 33, 127, 128, 129])
def test_cross_sections_without_allocation(orders):
    import torch
    mr, mi = 1.39, 0.015
    radii = np.array([x_of(orders), 3.3, x_of(32)]) * LAM / (2. * math.pi)
    d_r = torch.tensor(radii, device="cuda")
    d_out = torch.zeros(4, 3, dtype=torch.float64, device="cuda")
    torch.cuda.synchronize()
    f = libs.product().lmie_cross_sections_noalloc
    f.restype = C.c_int
    f.argtypes = [C.c_int, C.c_void_p, C.c_double, C.c_double, C.c_double, C.c_void_p, C.c_void_p]
    assert f(3, d_r.data_ptr(), LAM, mr, mi, d_out.data_ptr(), None) == 0
    got = d_out.cpu().numpy()
    for i, r in enumerate(radii):
        want = libs.run_oracle(abi.Case(dist="mono", lam=LAM, mr=mr, mi=mi, a1=r, r1=r, r2=r, n_quad=1, calc_gc=0, calc_pf=0))
        for q, name in enumerate(("cext", "csca", "cbak", "g")):
            assert abs(got[q, i] - want.scalars[name]) <= TOL * abs(want.scalars[name]), (orders, i, name)
