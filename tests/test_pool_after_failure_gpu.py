"""The pool of Gauss angles after a sub-batch that failed before it had them
computed: the next solve with as many angles computes them.  (The order is one
that no other test uses.)"""
import math
import os

import pytest

import libs
from lmie_b200 import abi

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("site, x", [("alloc", 1467.3), ("pinned", 1481.9), ("h2d", 1493.2)])
def test_angles_of_a_failed_solve_are_computed_by_the_next(site, x):
    r = x * 0.7 / (2. * math.pi)
    case = abi.Case(dist="mono", lam=0.7, mr=1.4, mi=0.01, a1=r, r1=r, r2=r, n_quad=1, accuracy=1e-6, n_angles=19)
    os.environ["LMIEB_FAULT"] = site
    try:
        assert libs.run_product(case).rc == -1
    finally:
        del os.environ["LMIEB_FAULT"]
    got, want = libs.run_product(case), libs.run_oracle(case)
    assert got.rc == 0 and got.n_coef == want.n_coef
    err = libs.compare(got, want)
    assert err["gc"] <= 1e-10 and err["pf"] <= 1e-9, err
