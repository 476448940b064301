"""Derivatives of single spheres' cross sections against extended precision,
where the way they are formed shows.

Bounds, fixed before the first run, on the median over the spheres:
- absorbing spheres (mi x from 10 to 100, x from 100 to 900) by mr and mi.  D
  is formed in about x steps with a rounding of 2^-53 each, of random sign at
  most x^(1/2) 2^-53 = 3e-15 and in the same direction x 2^-53 = 1e-13; its
  tangent likewise.  d Cext, a difference of the orders' oscillating terms, may
  have all of it twice, 2e-13; d Csca sums terms of one sign: 1e-14.  (With
  dD/dz as a difference of terms of order 1: 1e-12 and 3e-14.)
- small spheres (x from 0.02 to 0.5) by the wavelength.  g is a sum whose terms
  cancel to x^2 of their size, so eight roundings of 2^-52 make 8 2^-52 / x^2.
  (With psi' as a difference of two terms: 13 to 20.)
"""
import numpy as np
import pytest

import libs
import mie_extended
from lmie_b200 import abi
from lmie_b200.abi import deriv_unit

pytestmark = pytest.mark.gpu

LAM = 0.7
EPS = 2.**-52


def solve(x, mr, mi, derivs, extra=()):
    r = x * LAM / (2. * np.pi)
    cases = [abi.Case(dist="mono", lam=LAM, mr=mr, mi=mi, a1=v, r1=v, r2=v, n_quad=1, calc_gc=0, calc_pf=0,
                      derivs=deriv_unit(*derivs)) for v in r]
    got = abi.solve_batch(libs.product(), cases + list(extra))
    assert all(g.rc == 0 for g in got)
    # the size parameters the library formed
    return 2. * np.pi * r / LAM, got[:x.size]


def long_radii(n, derivs):
    """A case whose radii have K1 run a thread per radius."""
    r2 = 2200. * LAM / (2. * np.pi)
    return abi.Case(dist="gamma", lam=LAM, mr=1.4, mi=0.01, a1=0.3 * r2, a2=0.1, r1=0.5 * r2, r2=r2, n_int2=1, n_quad=n,
                    calc_gc=0, calc_pf=0, derivs=deriv_unit(*derivs))


@pytest.mark.parametrize("mr, mi", [(1.4, 0.11), (1.6, 0.1)])
@pytest.mark.parametrize("threads", [False, True])
def test_absorbing_spheres_by_the_refractive_index(mr, mi, threads):
    x, got = solve(np.geomspace(100., 900., 240), mr, mi, ("mr", "mi"), [long_radii(2600, ("mr", "mi"))] if threads else ())
    for k, m_l in enumerate((1., -1j)):
        want = mie_extended.cross_sections(x, mr, mi, 0., m_l)
        for name, bound in (("cext", 2e-13), ("csca", 1e-14)):
            w = want[name].d * (np.longdouble(LAM) * np.longdouble(LAM) / (2 * np.longdouble(np.pi)))
            err = np.abs(np.array([g.scalars_l[name][k] for g in got]).astype(np.longdouble) - w) / np.abs(w)
            assert np.median(err) <= bound, (name, k, float(np.median(err)))


@pytest.mark.parametrize("mr, mi", [(1.4, 0.01), (1.33, 1e-6)])
@pytest.mark.parametrize("threads", [False, True])
def test_small_spheres_by_the_wavelength(mr, mi, threads):
    x, got = solve(np.geomspace(0.02, 0.5, 300), mr, mi, ("lambda",), [long_radii(2600, ("lambda",))] if threads else ())
    want = mie_extended.cross_sections(x, mr, mi, -x.astype(np.longdouble) / np.longdouble(LAM), 0.)["g"].d
    err = np.abs(np.array([g.scalars_l["g"][0] for g in got]).astype(np.longdouble) - want) / np.abs(want)
    assert np.median(err * x * x) <= 8 * EPS, float(np.median(err * x * x)) / EPS
