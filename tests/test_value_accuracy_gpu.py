"""Cross sections of small absorbing spheres against extended precision.

Their extinction is the imaginary part of D_n, a small part of D_n itself, so
it shows how D is rounded.  Where only values are wanted the library forms D in
one of two ways (csrc/mie_radius.cuh); for few orders it has to be the chain of
D itself.

Bound, fixed before the first run: Cext of such a sphere is a product of about
a dozen quantities rounded to 2^-53, x cubed among them but with the library's
own x; half of that many half-ulp errors of random sign are under two ulps, so
the median over the spheres has to stay below 4 x 2^-52 = 9e-16 and the largest
below 32 x 2^-52 = 7e-15.  (D as a difference of a ratio and n/z: median 2e-15
to 3e-15, largest 1.2e-14.)
"""
import ctypes as C

import numpy as np
import pytest

import libs
from lmie_b200 import abi

pytestmark = pytest.mark.gpu

EPS = 2.**-52
LAM = 0.7


def cext_ld(x, mr, mi):
    """Cext of spheres of size parameters x (doubles), in 80-bit arithmetic with the library's truncations."""
    ld, cld = np.longdouble, np.clongdouble
    x = x.astype(ld)
    n1 = (x + 4.05 * np.cbrt(x) + 8).astype(int)
    m = cld(mr) - cld(1j) * ld(mi)
    z = m * x
    n2 = int(np.max(n1)) + 24
    D = np.zeros((n2 + 1, x.size), cld)
    for n in range(n2, 0, -1):
        D[n - 1] = n / z - 1 / (D[n] + n / z)
    r = np.zeros((int(np.max(n1)) + 1, x.size), ld)        # psi_n / psi_{n-1}, zero from n1 on
    for n in range(r.shape[0] - 2, 0, -1):
        r[n] = np.where(n < n1, 1 / ((2 * n + 1) / x - r[n + 1]), 0)
    psi, psi_p, chi, chi_p = None, np.sin(x), np.cos(x) / x + np.sin(x), np.cos(x)
    s = np.zeros_like(x)
    for n in range(1, r.shape[0]):
        psi = r[n] * psi_p
        zeta, zeta_p = psi + 1j * chi, psi_p + 1j * chi_p
        ca, cb = D[n] / m + n / x, m * D[n] + n / x
        a, b = (ca * psi - psi_p) / (ca * zeta - zeta_p), (cb * psi - psi_p) / (cb * zeta - zeta_p)
        s += np.where(n <= n1, (2 * n + 1) * (a + b).real, 0)
        psi_p, chi, chi_p = psi, (2 * n + 1) / x * chi - chi_p, chi
    return s * ld(LAM) * ld(LAM) / (2 * ld(np.pi))


def check(got, want):
    err = np.abs(got.astype(np.longdouble) - want) / want
    assert np.median(err) <= 4 * EPS and np.max(err) <= 32 * EPS, (float(np.median(err)), float(np.max(err)))


@pytest.mark.parametrize("mr, mi, lo, hi", [(1.4, 0.01, 1e-3, 0.1), (1.55, 0.1, 1e-3, 0.1), (1.33, 1e-3, 3e-3, 0.03)])
def test_cross_sections_of_small_absorbing_spheres(mr, mi, lo, hi):
    """lmie_cross_sections_noalloc, a block per radius."""
    import torch
    radii = np.geomspace(lo, hi, 1000) * LAM / (2. * np.pi)
    d_r = torch.tensor(radii, device="cuda")
    d_out = torch.zeros(4, radii.size, dtype=torch.float64, device="cuda")
    torch.cuda.synchronize()
    f = libs.product().lmie_cross_sections_noalloc
    f.restype = C.c_int
    f.argtypes = [C.c_int, C.c_void_p, C.c_double, C.c_double, C.c_double, C.c_void_p, C.c_void_p]
    assert f(radii.size, d_r.data_ptr(), LAM, mr, mi, d_out.data_ptr(), None) == 0
    check(d_out.cpu().numpy()[0], cext_ld(2. * np.pi * radii / LAM, mr, mi))


@pytest.mark.parametrize("with_large", [False, True])
def test_solves_of_small_absorbing_spheres(with_large):
    """The solve's values without derivatives; with larger spheres in the same call too."""
    radii = np.geomspace(1e-3, 0.1, 400) * LAM / (2. * np.pi)
    cases = [abi.Case(dist="mono", lam=LAM, mr=1.45, mi=0.02, a1=r, r1=r, r2=r, n_quad=1, calc_gc=0, calc_pf=0) for r in radii]
    if with_large:
        r2 = 40. * LAM / (2. * np.pi)
        cases += [abi.Case(dist="gamma", lam=LAM, mr=1.45, mi=0.02, a1=0.3 * r2, a2=0.1, r1=1e-3 * r2, r2=r2, n_int2=1,
                           n_quad=500, calc_gc=0, calc_pf=0)] * 4
    got = abi.solve_batch(libs.product(), cases)
    assert all(g.rc == 0 for g in got)
    check(np.array([g.scalars["cext"] for g in got[:radii.size]]), cext_ld(2. * np.pi * radii / LAM, 1.45, 0.02))
