"""Which angular sums a solve in the reference's precision takes, and how far
the fixed-point ones are from the FP64 kernel's.

The FP64 kernel's results of any case come from lmieb_solution_partial() over
all radii and lmieb_solution_finish(), which never use the fixed-point sums.
"""
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
