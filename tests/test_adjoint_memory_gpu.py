"""lmie_solution_adjoint where the device has no room for the orders of all
wavelengths: the wavelengths go through in passes.  A wavelength's arithmetic
does not depend on its company, so every output keeps its bits.

The shortage is made on the host: with LMIEB_FAULT=adjoint the allocation of
the whole counts as failed, and the passes are as small as they can be."""
import os

import numpy as np
import pytest

import lmie_b200
from lmie_b200 import workloads

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n_lambda, n_bins, n_quad, n_angles", [(1, 4, 8, 19), (5, 6, 7, 37), (17, 9, 16, 91)])
def test_passes_keep_every_bit(n_lambda, n_bins, n_quad, n_angles, capfd):
    p = workloads.adjoint_retrieval(n_lambda=n_lambda, n_bins=n_bins, n_quad=n_quad, n_angles=n_angles,
                                    lam_range=(0.4, 1.2), r_range=(0.05, 9.0))
    want = lmie_b200.adjoint(p)
    os.environ["LMIEB_FAULT"] = "adjoint"
    try:
        capfd.readouterr()
        got = lmie_b200.adjoint(p)
        assert "injected failure at \"adjoint\"" in capfd.readouterr().err
    finally:
        del os.environ["LMIEB_FAULT"]
    again = lmie_b200.adjoint(p)
    for name in ("loss", "cext", "csca", "g", "p11", "p12", "grad_mr", "grad_mi", "grad_weight"):
        assert np.array_equal(np.asarray(got[name]), np.asarray(want[name])), name
        assert np.array_equal(np.asarray(again[name]), np.asarray(want[name])), name
