"""lmie_solution_adjoint at every number of half-angle tiles (8 half-angles
each), with the last tile full and with one half-angle in it, against its CPU
oracle.  Tolerances: those of the adjoint's tests at x ~ 40."""
import numpy as np
import pytest

import adjoint_oracle
import lmie_b200
from lmie_b200 import workloads

pytestmark = pytest.mark.gpu


# not among them: two angles, where p12 is zero, and 33 and 31 angles, whose signed loss cancels
NO_SCALE = {(1, False), (3, False), (2, True)}


@pytest.mark.parametrize("tiles, full", [(t, f) for t in range(1, 17) for f in (False, True) if (t, f) not in NO_SCALE])
def test_every_number_of_tiles(tiles, full):
    n_angles = 16 * tiles - 1 if full else max(16 * tiles - 15, 2)
    assert ((n_angles + 1) // 2 + 7) // 8 == tiles
    p = workloads.adjoint_retrieval(n_lambda=2, n_bins=3, n_quad=3, n_angles=n_angles, lam_range=(0.5, 1.1),
                                    r_range=(0.05, 3.0))
    got, want = lmie_b200.adjoint(p), adjoint_oracle.solve(p)
    for name, tol in (("cext", 1e-10), ("csca", 1e-10), ("g", 1e-10), ("p11", 1e-10), ("p12", 1e-10), ("loss", 1e-10),
                      ("grad_mr", 1e-8), ("grad_mi", 1e-8), ("grad_weight", 1e-8)):
        a, b = np.asarray(got[name], float), np.asarray(want[name], float)
        err = float(np.max(np.abs(a - b)) / np.max(np.abs(b)))
        assert err <= tol, (name, err)
