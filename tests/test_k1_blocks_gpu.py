"""K1's blocks of a batch, cut by one thread or by the host's pool (csrc/driver.cu, k1_blocks), against single solves.

Bound, fixed before the first run: the same spheres' sums over at most 40
orders and 130 radii in another order, terms of one sign, 5200 roundings of
2^-53 each at most: 6e-13.
"""
import math

import pytest

import libs
from lmie_b200 import abi

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n_cases, n_quad", [(127, 129), (128, 128), (127, 130), (600, 40)])
def test_batches_around_the_serial_cut(n_cases, n_quad):
    cases = []
    for i in range(n_cases):
        r2 = (1. + 19. * i / n_cases) * 0.7 / (2. * math.pi)
        cases.append(abi.Case(dist="gamma", lam=0.7, mr=1.3 + 0.3 * i / n_cases, mi=1e-3, a1=0.35 * r2, a2=0.12, r1=0.2 * r2,
                              r2=r2, n_int2=1, n_quad=n_quad, calc_gc=0, calc_pf=0))
    got = abi.solve_batch(libs.product(), cases)
    for i in range(0, n_cases, 9):
        want = libs.run_product(cases[i])
        assert got[i].rc == 0 and want.rc == 0
        for k in ("cext", "csca"):
            assert abs(got[i].scalars[k] - want.scalars[k]) <= 6e-13 * want.scalars[k], (i, k)
