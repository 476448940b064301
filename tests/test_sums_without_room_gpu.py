"""Solves in the reference's precision on a device without room for the operands
of the fixed-point angular sums: they take the FP64 kernel's instead.

The shortage is made on the host: with LMIEB_FAULT=operands the arena with the
operands counts as one that could not be had."""
import os

import numpy as np
import pytest

import libs
from lmie_b200 import abi, workloads
from test_fp64_sums_gpu import fp64_kernel, gamma

pytestmark = pytest.mark.gpu


@pytest.fixture
def no_room():
    os.environ["LMIEB_FAULT"] = "operands"
    yield
    del os.environ["LMIEB_FAULT"]


@pytest.mark.parametrize("x, n_quad, derivs", [(150., 200, ("mr", "a1")), (420., 333, ("lambda",)), (12., 40, ())])
def test_a_solve_takes_the_fp64_kernel(no_room, x, n_quad, derivs):
    case = gamma(x, n_quad, mr=1.42, mi=2e-3, derivs=abi.deriv_unit(*derivs))
    got, want = libs.run_product(case), fp64_kernel(case)
    assert got.rc == 0 and want.rc == 0 and got.n_coef == want.n_coef
    assert got.scalars == want.scalars
    for name in ("gc", "pf") + (("gc_l", "pf_l") if derivs else ()):
        assert np.array_equal(getattr(got, name), getattr(want, name)), name


def test_a_batch_and_the_call_after_it(no_room):
    lib, cases = libs.product(), workloads.batched_uneven(40)
    got = abi.solve_batch(lib, cases, precision=abi.PRECISION_FP64)
    del os.environ["LMIEB_FAULT"]
    after = abi.solve_batch(lib, cases, precision=abi.PRECISION_FP64)
    os.environ["LMIEB_FAULT"] = ""
    for a, b in zip(got, after):
        assert a.rc == 0 and b.rc == 0 and a.n_coef == b.n_coef
        err = libs.compare(a, b)
        assert all(err[k] <= (1e-9 if k.endswith("_l") else 1e-11) for k in err), err
    assert any(not np.array_equal(a.gc, b.gc) for a, b in zip(got, after))
