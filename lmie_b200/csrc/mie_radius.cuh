// mie_radius.cuh -- the Mie coefficients of one radius: the recurrences and the
// formulas of an order, shared by K1's two forms (k_mie.cu: a thread per radius,
// a block per radius) and the device cross sections (k_noalloc.cu).
//
// The recurrences are run in their three-term forms,
//     P_{n-1} = (2n + 1)/z P_n - P_{n+1}        downward from D_{n2} = 0 (D_n = P_{n-1}/P_n - n/z),
//     u_{n-1} = (2n + 1)/x u_n - u_{n+1}        downward from psi_{n1} = 0 (psi_n = sin x u_n/u_0),
//     chi_{n+1} = (2n + 1)/x chi_n - chi_{n-1}  upward,
// with the starting values of the reference's ratio recurrences
// (src/lmie_core.c:298-440), from which they differ by rounding only.  An order
// costs two dependent FMAs of latency; the ratio forms wait for a reciprocal
// (a division takes more than 100 cycles from operand to result), and the
// reciprocal of P_n, from which D_n and dD/dz follow, is off the chain.  P and u
// grow by many orders of magnitude, so both are brought back to order 1 at the
// ends of blocks of MIE_B orders, by a power of two (exact).
//
// Derivatives: dD/dz = -1 + n/z^2 + rho (tau - 1/z), rho = P_{n-1}/P_n, tau =
// P_{n+1}/P_n -- the Riccati equation without its difference of large terms, no
// recurrence of its own; chi' = chi_{n-1} - n/x chi_n; psi' from the tangent of
// u's recurrence, since u is not exactly psi (it starts from zero at n1) and the
// reference differentiates what it computes.
//
// Every FMA is written out, and K1's and the cross sections' files are compiled
// without FMA contraction, so a radius' coefficients are the same bits
// whichever of them forms them (derivatives near resonances carry a rounding
// of a recurrence to 1e-12 of a case's cross section).
#pragma once

#include "dev_common.cuh"

constexpr int MIE_B = 4;                              // orders per block of the recurrences (a power of two)

// A block per radius: with a thread per radius a solve of few radii lasts as
// long as its largest radius' recurrences and orders one after the other.
// Three warps' first lanes run the three chains of the radius at the same time
// into shared memory, and then all threads form the orders side by side.
constexpr int MIE_BLOCK_T = 128;
constexpr int MIE_BLOCK_SMEM = 220 * 1024;            // what a block may take

// bytes for radii of up to n1 orders: P, u, chi (and u's tangent), two exponents per MIE_B orders, the
// coefficients passed from one round of orders to the next, reduction space
__host__ __device__ constexpr int mie_block_rows(int n1) { return (n1 + 2 * MIE_B) & ~(MIE_B - 1); }
__host__ __device__ constexpr int mie_block_smem(int n1, bool hx) {
    return mie_block_rows(n1) * (16 + 8 + 8 + (hx ? 8 : 0)) + mie_block_rows(n1) / MIE_B * 8 +
           (MIE_BLOCK_T + 1) * (hx ? 96 : 64) + 20 * (MIE_BLOCK_T / 32) * 8;
}

#ifdef __CUDACC__
namespace {

// 2^e, zero below the double range
__device__ __forceinline__ double mb_pow2(int e) {
    return e < -1022 ? 0. : __hiloint2double((1023 + min(e, 1023)) << 20, 0);
}

// exponent of the larger of two magnitudes (0 for zeros)
__device__ __forceinline__ int mb_exp(double a, double b) {
    const int ea = (__double2hiint(a) >> 20) & 0x7ff, eb = (__double2hiint(b) >> 20) & 0x7ff;
    const int e = max(ea, eb);
    return e ? e - 1023 : 0;
}

// a s + c, a b + c
__device__ __forceinline__ cplx cfma(cplx a, double s, cplx c) { return mk(fma(a.re, s, c.re), fma(a.im, s, c.im)); }
__device__ __forceinline__ cplx cfma(cplx a, cplx b, cplx c) {
    return mk(fma(a.re, b.re, fma(-a.im, b.im, c.re)), fma(a.re, b.im, fma(a.im, b.re, c.im)));
}
// conj(a) b + c
__device__ __forceinline__ cplx cfmac(cplx a, cplx b, cplx c) {
    return mk(fma(a.re, b.re, fma(a.im, b.im, c.re)), fma(a.re, b.im, fma(-a.im, b.re, c.im)));
}
__device__ __forceinline__ cplx cmulc(cplx a, cplx b) {
    return mk(fma(a.re, b.re, a.im * b.im), fma(a.re, b.im, -(a.im * b.re)));
}
// Re(a conj(b)) + c
__device__ __forceinline__ double rfmac(cplx a, cplx b, double c) { return fma(a.re, b.re, fma(a.im, b.im, c)); }
__device__ __forceinline__ double rmulc(cplx a, cplx b) { return fma(a.re, b.re, a.im * b.im); }

// What every order of a radius needs.
template <bool HX>
struct MieRadius {
    double x, xinv;
    cplx m, minv, minv2, zinv, zinv2;
    double xl;                  // HX: the x column's direction (x_l, m_l)
    cplx ml;
    __device__ __forceinline__ void set(double x_, cplx m_, cplx minv_, double xl_, cplx ml_) {
        x = x_;
        xinv = 1. / x;
        m = m_;
        minv = minv_;
        minv2 = minv * minv;
        zinv = cinv(mk(m.re * x, m.im * x));
        zinv2 = zinv * zinv;
        xl = xl_;
        ml = ml_;
    }
};

// The chain of P: cur = P_n, hi = P_{n+1}.
struct MieP {
    cplx hi, cur;
    __device__ __forceinline__ cplx next(int n, cplx zinv) const {
        const double c = 2. * n + 1., cr = c * zinv.re, ci = c * zinv.im;
        return mk(fma(cr, cur.re, fma(-ci, cur.im, -hi.re)), fma(cr, cur.im, fma(ci, cur.re, -hi.im)));
    }
    __device__ __forceinline__ void step(cplx nx) {
        hi = cur;
        cur = nx;
    }
    // at the end of a block of orders; returns the exponent taken out
    __device__ __forceinline__ int rescale() {
        const int g = mb_exp(cur.re, cur.im);
        if (g <= 40 && g >= -40) return 0;
        const double sc = mb_pow2(-g);
        cur = cur * sc;
        hi = hi * sc;
        return g;
    }
};

// The chain of u (and its tangent w.r.t. x): cur = u_n, hi = u_{n+1}.
template <bool HX>
struct MieU {
    double hi, cur, xhi, xcur;
    __device__ __forceinline__ void start() {         // u_{n1} = 0, u_{n1 - 1} = 1
        hi = -1.;
        cur = xhi = xcur = 0.;
    }
    __device__ __forceinline__ void step(int n, double xinv) {
        const double c = (2. * n + 1.) * xinv;
        if (HX) {
            const double xn = fma(c, xcur, fma(-c * xinv, cur, -xhi));
            xhi = xcur;
            xcur = xn;
        }
        const double nx = fma(c, cur, -hi);
        hi = cur;
        cur = nx;
    }
    __device__ __forceinline__ int rescale() {
        const int g = mb_exp(cur, hi);
        if (g <= 40 && g >= -40) return 0;
        const double sc = mb_pow2(-g);
        cur *= sc;
        hi *= sc;
        if (HX) {
            xcur *= sc;
            xhi *= sc;
        }
        return g;
    }
};

// D_n and, with TAN, dD/dz from P_{n-1}, P_n, P_{n+1} (scaled alike)
template <bool TAN, bool HX>
__device__ __forceinline__ void mie_d(const MieRadius<HX> &c, int n, cplx lo, cplx cur, cplx hi, cplx &D, cplx &Dz) {
    const cplx inv = cinv(cur), rho = lo * inv, nz = (double) n * c.zinv;
    D = rho - nz;
    if (TAN) Dz = cfma(rho, cfma(hi, inv, -c.zinv), cfma(c.zinv2, (double) n, mk(-1., 0.)));
}

// The coefficients of order n and their tangents: a, b; am, bm w.r.t. m; ax, bx
// in the x column's direction.
struct MieAB {
    cplx a, b, am, bm, ax, bx;
};
template <bool HM, bool HX>
__device__ __forceinline__ MieAB mie_ab(const MieRadius<HX> &c, int n, cplx D, cplx Dz, double psi, double psi_p,
                                        double chi, double chi_p, double psix, double psix_p) {
    MieAB r;
    const cplx zeta = mk(psi, chi), zeta_p = mk(psi_p, chi_p);
    const double tt = n * c.xinv;
    const cplx ca = cfma(D, c.minv, mk(tt, 0.));
    const cplx na = cfma(ca, psi, mk(-psi_p, 0.));
    const cplx ida = cinv(cfma(ca, zeta, -zeta_p));
    r.a = na * ida;
    const cplx cb = cfma(c.m, D, mk(tt, 0.));
    const cplx nb = cfma(cb, psi, mk(-psi_p, 0.));
    const cplx idb = cinv(cfma(cb, zeta, -zeta_p));
    r.b = nb * idb;
    r.am = r.bm = r.ax = r.bx = mk(0., 0.);
    const cplx ida2 = ida * ida, idb2 = idb * idb;
    if (HM) {
        const cplx Dm = Dz * c.x;
        const cplx da = cfma(Dm, c.minv, -(D * c.minv2)) * ida2, db = cfma(c.m, Dm, D) * idb2;
        const double W = fma(psi_p, chi, -(psi * chi_p));
        r.am = mk(-W * da.im, W * da.re);             // i W da
        r.bm = mk(-W * db.im, W * db.re);
    }
    if (HX) {
        const cplx Dx = Dz * cfma(c.ml, c.x, c.m * c.xl);
        const double chix = c.xl * fma(-tt, chi, chi_p), chix_p = c.xl * fma(tt, chi_p, -chi);
        const cplx zetal = mk(psix, chix), zetal_p = mk(psix_p, chix_p), tl = mk(-tt * c.xinv * c.xl, 0.);
        const cplx c6 = cfma(Dx, c.minv, cfma(-(D * c.minv2), c.ml, tl));
        r.ax = cfma(cfma(c6, psi, cfma(ca, psix, mk(-psix_p, 0.))), ida,
                    -(na * (cfma(c6, zeta, cfma(ca, zetal, -zetal_p)) * ida2)));
        const cplx c4 = cfma(c.ml, D, cfma(c.m, Dx, tl));
        r.bx = cfma(cfma(c4, psi, cfma(cb, psix, mk(-psix_p, 0.))), idb,
                    -(nb * (cfma(c4, zeta, cfma(cb, zetal, -zetal_p)) * idb2)));
    }
    return r;
}

// Sums over the orders: se, ss, Re sb, Im sb, sg, then with HM their
// derivatives w.r.t. mr and mi, with HX those in the x column's direction.
template <bool HM, bool HX>
struct MieSums {
    static constexpr int N = 5 * (1 + 2 * HM + HX), M = HM ? 5 : 0, X = 5 * (1 + 2 * HM) - (HX ? 0 : 5);
    double v[N];
    __device__ __forceinline__ void zero() {
#pragma unroll
        for (int q = 0; q < N; ++q) v[q] = 0.;
    }
    // order n, p the coefficients of order n - 1 (zeros for n = 1)
    __device__ __forceinline__ void add(int n, const MieAB &q, const MieAB &p) {
        const double f1 = 2. * n + 1., sgn = (n & 1) ? -f1 : f1;
        // the asymmetry factors of order n - 1: (n^2 - 1) / n, (2n - 1) / (n (n - 1))
        const double f3 = (double) (n - 1) * (n + 1) / n, f4 = n >= 2 ? (2. * n - 1.) / ((double) n * (n - 1)) : 0.;
        v[0] = fma(f1, q.a.re + q.b.re, v[0]);
        v[1] = fma(f1, rfmac(q.a, q.a, rmulc(q.b, q.b)), v[1]);
        v[2] = fma(sgn, q.a.re - q.b.re, v[2]);
        v[3] = fma(sgn, q.a.im - q.b.im, v[3]);
        v[4] = fma(f3, rfmac(p.a, q.a, rmulc(p.b, q.b)), fma(f4, rmulc(p.a, p.b), v[4]));
        if (HM) {
            // complex derivatives: the real part is d/dmr, the imaginary part d/dmi
            const cplx s = q.am + q.bm, d = q.am - q.bm, w = cfmac(q.a, q.am, cmulc(q.b, q.bm));
            v[M + 0] = fma(f1, s.re, v[M + 0]);
            v[2 * M + 0] = fma(f1, s.im, v[2 * M + 0]);
            v[M + 1 * HM] = fma(2. * f1, w.re, v[M + 1 * HM]);
            v[2 * M + 1 * HM] = fma(2. * f1, w.im, v[2 * M + 1 * HM]);
            v[M + 2 * HM] = fma(sgn, d.re, v[M + 2 * HM]);
            v[M + 3 * HM] = fma(sgn, d.im, v[M + 3 * HM]);
            const cplx g3 = cfmac(q.a, p.am, cfmac(p.a, q.am, cfmac(q.b, p.bm, cmulc(p.b, q.bm))));
            const cplx g4 = cfmac(p.b, p.am, cmulc(p.a, p.bm));
            v[M + 4 * HM] = fma(f3, g3.re, fma(f4, g4.re, v[M + 4 * HM]));
            v[2 * M + 4 * HM] = fma(f3, g3.im, fma(f4, g4.im, v[2 * M + 4 * HM]));
        }
        if (HX) {
            v[X + 0] = fma(f1, q.ax.re + q.bx.re, v[X + 0]);
            v[X + 1 * HX] = fma(2. * f1, rfmac(q.a, q.ax, rmulc(q.b, q.bx)), v[X + 1 * HX]);
            v[X + 2 * HX] = fma(sgn, q.ax.re - q.bx.re, v[X + 2 * HX]);
            v[X + 3 * HX] = fma(sgn, q.ax.im - q.bx.im, v[X + 3 * HX]);
            const double g3 = rfmac(p.ax, q.a, rfmac(p.a, q.ax, rfmac(p.bx, q.b, rmulc(p.b, q.bx))));
            v[X + 4 * HX] = fma(f3, g3, fma(f4, rfmac(p.ax, p.b, rmulc(p.a, p.bx)), v[X + 4 * HX]));
        }
    }
    // sb is complex itself: its derivative w.r.t. mi is -i times the one w.r.t. mr
    __device__ __forceinline__ void close() {
        if (HM) {
            v[2 * M + 2 * HM] = v[M + 3 * HM];
            v[2 * M + 3 * HM] = -v[M + 2 * HM];
        }
    }
};

// The block's radius: n1 orders (the shared memory laid out for n1max), D_n
// from n2.  store(n, ab) is called once per order, by one thread each; all
// threads return with the sums.
template <bool HM, bool HX, class Store>
__device__ __forceinline__ void mie_block(unsigned char *smem, const MieRadius<HX> &c, int n1, int n2, int n1max,
                                          MieSums<HM, HX> &sums, Store &&store) {
    constexpr int T = MIE_BLOCK_T, NP = HX ? 12 : 8, NS = MieSums<HM, HX>::N;
    const int rows = mie_block_rows(n1max), tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    double2 *P = (double2 *) smem;                    // [n1 + 2]
    double *u = (double *) (P + rows), *chi = u + rows, *ux = chi + rows;
    double *pass = chi + rows + (HX ? rows : 0);      // [T + 1][NP] coefficients of the round (entry 0: the order before)
    double *red = pass + (T + 1) * NP;                // [20][T / 32]
    int *eP = (int *) (red + 20 * (T / 32)), *eU = eP + rows / MIE_B;
    __shared__ double sh_psi, sh_psix;                // psi_n = sh_psi u_n 2^(eU[n / MIE_B] - sh_eu)
    __shared__ int sh_eu;

    if (warp == 0) {
        if (lane == 0) {
            MieP p;
            p.hi = mk(1., 0.);                        // P_{n2} = 1, P_{n2 - 1} = n2 / z
            p.cur = (double) n2 * c.zinv;
            for (int n = n2 - 1, e = 0; n >= 0;) {
                const int b = n / MIE_B, n0 = b * MIE_B;
                if (n0 <= n1 + 1) eP[b] = e;
#pragma unroll 4
                for (; n >= n0; --n) {
                    if (n <= n1 + 1) P[n] = make_double2(p.cur.re, p.cur.im);
                    p.step(p.next(n, c.zinv));
                }
                e += p.rescale();
            }
        }
    } else if (warp == 1) {
        if (lane == 0) {
            MieU<HX> q;
            q.start();
            int e = 0;
            for (int n = n1; n >= 0;) {
                const int b = n / MIE_B, n0 = b * MIE_B;
                eU[b] = e;
#pragma unroll 4
                for (; n >= n0; --n) {
                    u[n] = q.cur;
                    if (HX) ux[n] = q.xcur;
                    q.step(n, c.xinv);
                }
                if (n >= 0) e += q.rescale();
            }
            sh_psi = sin(c.x) / u[0];
            if (HX) sh_psix = fma(-sh_psi, ux[0], cos(c.x)) / u[0];
            sh_eu = e;
        }
    } else if (warp == 2) {
        if (lane == 0) {
            double sinx, cosx;
            sincos(c.x, &sinx, &cosx);
            double lo = cosx, cur = fma(c.xinv, cosx, sinx);
            chi[0] = lo;
#pragma unroll 4
            for (int n = 1; n <= n1; ++n) {
                chi[n] = cur;
                const double nx = fma((2. * n + 1.) * c.xinv, cur, -lo);
                lo = cur;
                cur = nx;
            }
        }
    }
    if (tid < NP) pass[tid] = 0.;                     // order 0
    __syncthreads();

    const double spsi = sh_psi, spsix = HX ? sh_psix : 0.;
    const int eu0 = sh_eu;
    sums.zero();
    for (int j0 = 0; j0 < n1; j0 += T) {
        const int j = j0 + tid + 1;
        const bool on = j <= n1;
        MieAB q;
        q.a = q.b = q.am = q.bm = q.ax = q.bx = mk(0., 0.);
        if (on) {
            const double2 p1 = P[j], p0 = P[j - 1], p2 = P[j + 1];
            const int e1 = eP[j / MIE_B];
            cplx lo = mk(p0.x, p0.y), hi = mk(p2.x, p2.y), D, Dz;
            if (j % MIE_B == 0) lo = lo * mb_pow2(eP[j / MIE_B - 1] - e1);
            if (j % MIE_B == MIE_B - 1) hi = hi * mb_pow2(eP[j / MIE_B + 1] - e1);
            mie_d<HM || HX>(c, j, lo, mk(p1.x, p1.y), hi, D, Dz);
            const double s1 = mb_pow2(eU[j / MIE_B] - eu0), s0 = mb_pow2(eU[(j - 1) / MIE_B] - eu0);
            const double psi = spsi * u[j] * s1, psi_p = spsi * u[j - 1] * s0;
            double psix = 0., psix_p = 0.;
            if (HX) {
                psix = c.xl * (fma(spsix, u[j], spsi * ux[j]) * s1);
                psix_p = c.xl * (fma(spsix, u[j - 1], spsi * ux[j - 1]) * s0);
            }
            q = mie_ab<HM, HX>(c, j, D, Dz, psi, psi_p, chi[j], chi[j - 1], psix, psix_p);
            store(j, q);
        }
        double *ps = pass + (size_t) (tid + 1) * NP;
        ps[0] = q.a.re; ps[1] = q.a.im; ps[2] = q.b.re; ps[3] = q.b.im;
        if (HM) { ps[4] = q.am.re; ps[5] = q.am.im; ps[6] = q.bm.re; ps[7] = q.bm.im; }
        if (HX) { ps[NP - 4] = q.ax.re; ps[NP - 3] = q.ax.im; ps[NP - 2] = q.bx.re; ps[NP - 1] = q.bx.im; }
        __syncthreads();
        if (on) {
            const double *pv = pass + (size_t) tid * NP;
            MieAB p;
            p.a = mk(pv[0], pv[1]);
            p.b = mk(pv[2], pv[3]);
            p.am = p.bm = p.ax = p.bx = mk(0., 0.);
            if (HM) { p.am = mk(pv[4], pv[5]); p.bm = mk(pv[6], pv[7]); }
            if (HX) { p.ax = mk(pv[NP - 4], pv[NP - 3]); p.bx = mk(pv[NP - 2], pv[NP - 1]); }
            sums.add(j, q, p);
        }
        __syncthreads();
        // the round's last order for the next one
        if (tid < NP) pass[tid] = pass[(size_t) T * NP + tid];
        __syncthreads();
    }
#pragma unroll
    for (int q = 0; q < NS; ++q) {
        double v = sums.v[q];
#pragma unroll
        for (int o = 16; o; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
        if (lane == 0) red[q * (T / 32) + warp] = v;
    }
    __syncthreads();
#pragma unroll
    for (int q = 0; q < NS; ++q) {
        sums.v[q] = red[q * (T / 32)];
#pragma unroll
        for (int w = 1; w < T / 32; ++w) sums.v[q] += red[q * (T / 32) + w];
    }
    sums.close();
}

}  // namespace
#endif
