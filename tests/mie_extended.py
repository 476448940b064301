"""Cross sections of single spheres and their derivatives in 80-bit arithmetic
(test infrastructure): the reference's recurrences (src/lmie_core.c:298-590)
with its truncations, values and one tangent carried together, vectorised over
spheres of one refractive index."""
import numpy as np

LD, CLD = np.longdouble, np.clongdouble


class Dual:
    """A value and its derivative."""

    def __init__(self, v, d):
        self.v, self.d = v, d

    def __add__(self, o):
        o = _dual(o)
        return Dual(self.v + o.v, self.d + o.d)

    def __sub__(self, o):
        o = _dual(o)
        return Dual(self.v - o.v, self.d - o.d)

    def __mul__(self, o):
        o = _dual(o)
        return Dual(self.v * o.v, self.d * o.v + self.v * o.d)

    def inv(self):
        i = 1 / self.v
        return Dual(i, -self.d * i * i)

    def __truediv__(self, o):
        return self * _dual(o).inv()

    def conj(self):
        return Dual(np.conj(self.v), np.conj(self.d))

    def real(self):
        return Dual(np.real(self.v), np.real(self.d))


def _dual(o):
    return o if isinstance(o, Dual) else Dual(o, 0 * o)


def cross_sections(x, mr, mi, x_l=0., m_l=0.):
    """Sums of Cext and Csca (times 2 pi / lambda^2) and g of the spheres, each
    with its derivative in the direction (x_l per sphere, m_l): {name: Dual}.
    x, mr, mi are doubles, x_l, m_l whatever the direction is."""
    x = np.asarray(x, dtype=np.float64)
    n1 = np.array([int(float(v) + 4.05 * float(v) ** (1. / 3.) + 8) for v in x])
    top = int(n1.max())
    az = np.hypot(float(mr), float(mi)) * x
    t = np.maximum(n1, az)
    n2 = np.array([int(float(v) + 6.40 * float(v) ** (1. / 3.) + 8) for v in t])
    X = Dual(x.astype(LD), np.broadcast_to(np.asarray(x_l, dtype=LD), x.shape))
    m = Dual(CLD(LD(mr)) - CLD(1j) * LD(mi), CLD(m_l))
    z = m * X
    D = [None] * (int(n2.max()) + 1)
    cur = Dual(np.zeros(x.shape, CLD), np.zeros(x.shape, CLD))
    for n in range(int(n2.max()), 0, -1):              # D_{n-1} from D_n, zero at n2
        on = n <= n2
        g = Dual(CLD(n), CLD(0)) / z
        nx = g - (cur + g).inv()
        cur = Dual(np.where(on, nx.v, 0), np.where(on, nx.d, 0))
        if n - 1 <= top:
            D[n - 1] = cur
    r = [None] * (top + 1)                             # psi_n / psi_{n-1}, zero at n1
    cur = Dual(np.zeros(x.shape, LD), np.zeros(x.shape, LD))
    for n in range(top, 0, -1):
        nx = (Dual(LD(2 * n + 1), LD(0)) / X - cur).inv()
        on = n < n1
        cur = Dual(np.where(on, nx.v, 0), np.where(on, nx.d, 0))
        r[n] = cur
    s, c = Dual(np.sin(X.v), np.cos(X.v) * X.d), Dual(np.cos(X.v), -np.sin(X.v) * X.d)
    psi_p, chi_p, chi = s, c, c / X + s
    zero = Dual(np.zeros(x.shape, LD), np.zeros(x.shape, LD))
    ext, sca, asy, ap, bp = zero, zero, zero, zero, zero
    for n in range(1, top + 1):
        psi = r[n] * psi_p
        zeta = Dual(psi.v + 1j * chi.v, psi.d + 1j * chi.d)
        zeta_p = Dual(psi_p.v + 1j * chi_p.v, psi_p.d + 1j * chi_p.d)
        t = Dual(LD(n), LD(0)) / X
        ca, cb = D[n] / m + t, m * D[n] + t
        a = (ca * psi - psi_p) / (ca * zeta - zeta_p)
        b = (cb * psi - psi_p) / (cb * zeta - zeta_p)
        on = n <= n1
        a, b = (Dual(np.where(on, q.v, 0), np.where(on, q.d, 0)) for q in (a, b))
        ext = ext + (a + b).real() * LD(2 * n + 1)
        sca = sca + (a * a.conj() + b * b.conj()).real() * LD(2 * n + 1)
        if n > 1:
            asy = asy + (ap * a.conj() + bp * b.conj()).real() * (LD(n - 1) * (n + 1) / n) \
                + (ap * bp.conj()).real() * (LD(2 * n - 1) / (LD(n) * (n - 1)))
        ap, bp, psi_p = a, b, psi
        chi_p, chi = chi, Dual(LD(2 * n + 1), LD(0)) / X * chi - chi_p
    return {"cext": ext, "csca": sca, "g": asy / sca * LD(2)}
