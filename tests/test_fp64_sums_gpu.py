"""Which angular sums a solve in the reference's precision takes, and how far
the fixed-point ones are from the FP64 kernel's.

The FP64 kernel's results of any case come from lmieb_solution_partial() over
all radii and lmieb_solution_finish(), which never use the fixed-point sums.
"""
import ctypes as C
import math

import numpy as np
import pytest

import libs
from lmie_b200 import abi

pytestmark = pytest.mark.gpu


def fp64_kernel(case):
    lib = libs.product()
    return abi.solve_finish(lib, case, abi.solve_partial(lib, case, 0, 1))


def gamma(x, n_quad, lam=0.7, **kw):
    r2 = x * lam / (2. * math.pi)
    return abi.Case(dist="gamma", lam=lam, a1=0.35 * r2, a2=0.12, r1=0.2 * r2, r2=r2, n_int2=1, n_quad=n_quad, **kw)


@pytest.mark.parametrize("derivs", [(), ("mr",)])
def test_more_orders_than_the_fixed_point_sums_take(derivs):
    """A solve of more than 5120 orders is the FP64 kernel's, cut into work items as its own work asks: the same
    bits as the integrals taken away and brought back."""
    case = gamma(5180., 300, mr=1.4, mi=1e-3, derivs=abi.deriv_unit(*derivs), calc_pf=0)
    assert libs.product().lmie_calc_max_coef(case.lam, abi.InputBlock(case).s.dist_type, case.a1, case.a2, case.a3,
                                             case.r1, case.r2) > 2 * 5120
    got, want = libs.run_product(case), fp64_kernel(case)
    assert got.rc == 0 and want.rc == 0 and got.n_coef == want.n_coef
    for name in ("gc",) + (("gc_l",) if derivs else ()):
        assert np.array_equal(getattr(got, name), getattr(want, name)), name
    assert got.scalars == want.scalars


def _log(rng, lo, hi):
    return math.exp(rng.uniform(math.log(lo), math.log(hi)))


def _index(rng):
    return dict(mr=rng.uniform(1.2, 1.7), mi=_log(rng, 1e-9, 0.1))


def _mono(rng, lo, hi):
    r = _log(rng, lo, hi) * 0.7 / (2. * math.pi)
    return abi.Case(dist="mono", lam=0.7, a1=r, r1=r, r2=r, n_quad=1, accuracy=0., calc_pf=0, **_index(rng))


def _narrow(rng, lo, hi, n_lo, n_hi):
    """A log-normal whose radii, many as they are, do not average anything: over a range of 1e-7 .. 0.1 of their size."""
    w, r2 = _log(rng, 1e-7, 0.1), _log(rng, lo, hi) * 0.7 / (2. * math.pi)
    return abi.Case(dist="log_normal", lam=0.7, a1=(1. - w / 2.) * r2, a2=_log(rng, 1e-4, 0.1), r1=(1. - w) * r2, r2=r2,
                    n_int2=1, n_quad=int(_log(rng, n_lo, n_hi)), accuracy=0., calc_pf=0, **_index(rng))


FAMILIES = {
    "single radii": lambda rng: [_mono(rng, 8., 1100.) for _ in range(80)],
    "many radii in a narrow range": lambda rng: [_narrow(rng, 15., 120., 100, 700) for _ in range(80)],
    "large, few radii": lambda rng: [_narrow(rng, 1130., 4900., 1, 30) for _ in range(8)],
    "broad": lambda rng: [gamma(_log(rng, 8., 700.), int(_log(rng, 4, 300)), accuracy=0., calc_pf=0, **_index(rng))
                          for _ in range(40)],
}


@pytest.mark.parametrize("name", FAMILIES)
@pytest.mark.parametrize("precision", [abi.PRECISION_FP64, abi.PRECISION_INT8])
def test_expansion_error_within_the_band_in_use(name, precision):
    """The expansion coefficients near the truncation threshold (1e-9 .. 1e-5 of 2l + 1; nothing is truncated here)
    against the FP64 kernel's: within the library's own re-solve band, with a factor of 1.5 to spare."""
    band = libs.product().lmieb_truncation_band
    band.restype, band.argtypes = C.c_double, [C.c_int]
    cases = FAMILIES[name](np.random.Generator(np.random.PCG64(11)))
    got = abi.solve_batch(libs.product(), cases, n_threads=16, precision=precision)
    for i, (c, g) in enumerate(zip(cases, got)):
        want = fp64_kernel(c)
        assert g.rc == 0 and want.rc == 0 and g.n_coef == want.n_coef
        beta, scale = np.abs(want.gc[0]), 2. * np.arange(want.gc.shape[1]) + 1.
        near = (beta <= 1e-5 * scale) & (beta >= 1e-9 * scale)
        err = float(np.max((np.abs(g.gc[0] - want.gc[0]) / scale)[near])) if near.any() else 0.
        x = 2. * math.pi * c.r2 / c.lam
        assert err <= band(int(x + 4.05 * x ** (1. / 3.) + 8)) / 1.5, (i, c.n_quad, x, err)
