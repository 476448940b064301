// mie_radius.cuh -- the Mie coefficients of one radius: the recurrences and the
// formulas of an order, shared by K1's two forms (k_mie.cu: a thread per radius,
// a block per radius) and the device cross sections (k_noalloc.cu).
//
// The recurrences
//     D_n = (n + 1)/z - 1 / (D_{n+1} + (n + 1)/z)   downward from D_{n2} = 0,
//     u_{n-1} = (2n + 1)/x u_n - u_{n+1}            downward from psi_{n1} = 0 (psi_n = sin x u_n/u_0),
//     chi_{n+1} = (2n + 1)/x chi_n - chi_{n-1}      upward,
// have the starting values of the reference's (src/lmie_core.c:298-440), whose
// psi runs in ratios: an order of u costs one dependent FMA, a ratio waits for a
// reciprocal (60 cycles).  u grows by many orders of magnitude, so it is brought
// back to order 1 at the ends of blocks of MIE_B orders, by a power of two
// (exact).  Where only values are wanted, the block form runs D of radii with
// MIE_P_MIN orders and more in a three-term form too, P_{n-1} = (2n + 1)/z P_n -
// P_{n+1}, D_n = P_{n-1}/P_n - n/z: 18 cycles an order instead of 105 (107
// thousand radii 308 us instead of 495).  Its rounding is another one, which
// values show by 1e-11 at most; derivatives at the resonances of weakly absorbing
// spheres carry a rounding of D up to 1e-7 of their value, as far as the
// reference's own, so with derivatives D is rounded as it always was here.  Nor
// do small spheres take it: the difference of P_{n-1}/P_n and n/z takes bits from
// Im D, which is all of a small absorbing sphere's extinction (see MIE_P_MIN).
//
// Derivatives: dD/dz = n/z^2 - 1 + (n/z - D)(n/z + D), the Riccati equation with
// its difference of large terms in factors, no recurrence of its own, for
// radii through which light gets; of others D is near -i and the terms cancel, so
// where they are wanted by m theirs is the tangent of D's recurrence (see
// MIE_DZ_MIN).  chi' = chi_{n-1} - n/x chi_n.  psi' from the tangent of u's
// recurrence, since u is not exactly psi (it starts from zero at n1) and the
// reference differentiates what it computes; for radii of fewer than MIE_P_MIN
// orders, whose u grows by orders of magnitude between psi's few, from the tangent
// of the reference's ratios.
//
// Every FMA is written out, and K1's and the cross sections' files are compiled
// without FMA contraction, so with derivatives a radius' coefficients are the
// same bits whichever of them forms them (derivatives near resonances carry a
// rounding of a recurrence to 1e-12 of a case's cross section).  Without, the
// thread-per-radius form keeps the chain of D where a block runs P, and its
// values differ by that rounding.
#pragma once

#include "dev_common.cuh"

constexpr int MIE_B = 4;                              // orders per block of the recurrences (a power of two)

// A block's team for one radius or several: with a thread per radius a solve of
// few radii lasts as long as its largest radius' recurrences and orders one
// after the other, and one of many is held by the latency of an order (some 1800
// cycles with derivatives).  Here three warps run the three chains of the
// block's radii, a lane each, into shared memory, and then the orders are formed
// side by side: by all threads, radius after radius (TEAM 128), or by a
// warp per radius (TEAM 32).
constexpr int MIE_BLOCK_T = 128;
constexpr int MIE_BLOCK_MAX = 32;                     // radii of a block
constexpr int MIE_BLOCK_SMEM = 220 * 1024;            // what a block may take
// Orders from which a block runs D as ratios of P where only values are wanted.
// Largest relative errors against 113-bit arithmetic, 200 spheres of mi 1e-5 ..
// 0.1 each, chain of D / ratios of P: Cext at x 0.001 .. 0.1 (8 and 9 orders)
// 1.1e-15 / 1.2e-14, x 0.3 .. 1 2.4e-15 / 5.4e-15, x 1 .. 2 2.9e-15 / 3.7e-15; from
// x = 2 (15 orders) to 900 equal for Cext, Csca, Cbak, g and Cext - Csca.  A
// chain of D from below 32 orders takes at most 3 us.
//
// With the x column, psi and its tangent of smaller radii come from the ratios
// psi_n / psi_{n-1}, as the reference's: medians of d Cext/dx at x 1 .. 2 5.5e-16 (from u
// 7.7e-16), of dg/dx at 0.1 .. 0.3 2.3e-14 (1.0e-13); from x = 5 on u's are the better
// ones (x 100 .. 900 1.2e-12, ratios 1.9e-12).
constexpr int MIE_P_MIN = 32;
// mi x from which dD/dz for a derivative by m is the tangent of D's recurrence.
// Medians of d Cext/dmr of 400 spheres of x 100 .. 900 against 113-bit arithmetic,
// tangent / Riccati: mi x 0.3 .. 1 9.2e-14 / 9.4e-14, 1 .. 3 8.9e-14 / 1.0e-13,
// 3 .. 10 2.7e-13 / 4.1e-12, 30 .. 100 9.3e-15 / 7.2e-13; x 8 .. 96 alike.  By x the two
// are equal everywhere.  A block keeps the tangent as a correction of the Riccati
// equation's in 8 bytes an order: with 16, four blocks no longer fit an SM (4096
// uneven cases 4.66 ms, with 8 3.87, without the tangent 3.43).
constexpr double MIE_DZ_MIN = 1.;

// rows of shared memory of a radius of n1 orders; bytes of a block of that many rows: D, u, chi (hx: and u's
// tangent; dz: and D's, as a correction), two exponents per MIE_B orders, reduction space, what the team needs to know of each radius
__host__ __device__ constexpr int mie_block_rows(int n1) { return (n1 + 2 * MIE_B) & ~(MIE_B - 1); }
__host__ __device__ constexpr int mie_block_smem(int rows, bool hx, bool dz) {
    return rows * (16 + 8 + 8 + (hx ? 8 : 0) + (dz ? 8 : 0)) + rows / MIE_B * 8 + (4 * 12 + 20 * 4) * 8 + MIE_BLOCK_MAX * 72;
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

// whether a radius takes dD/dz from D's recurrence (where a derivative by m is wanted)
__host__ __device__ __forceinline__ bool mie_dz_chain(cplx m, double x) { return fabs(m.im) * x > MIE_DZ_MIN; }

// What every order of a radius needs.
template <bool HX>
struct MieRadius {
    double x, xinv;
    cplx m, minv, minv2, zinv, zinv2;
    double xl;                  // HX: the x column's direction (x_l, m_l)
    cplx ml;
    // the refractive index (and its part of the x column's direction)
    __device__ __forceinline__ void set_m(cplx m_, cplx minv_, cplx ml_) {
        m = m_;
        minv = minv_;
        minv2 = minv * minv;
        ml = ml_;
    }
    __device__ __forceinline__ void set_x(double x_, double xl_) {
        x = x_;
        xinv = 1. / x;
        zinv = cinv(mk(m.re * x, m.im * x));
        zinv2 = zinv * zinv;
        xl = xl_;
    }
};

// The chain of P, whose ratios are D (values only, MIE_P_MIN): P_{n-1} = (2n + 1)/z P_n - P_{n+1}, D_n = P_{n-1}/P_n - n/z;
// cur = P_n, hi = P_{n+1}.
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
    // at the end of a block of orders; returns the exponent taken out (of the
    // older value: it is there while the newer one is still being formed)
    __device__ __forceinline__ int rescale() {
        const int e = mb_exp(hi.re, hi.im), g = e <= 40 && e >= -40 ? 0 : e;
        const double sc = mb_pow2(-g);
        cur = cur * sc;
        hi = hi * sc;
        return g;
    }
};

// The chain of D_n (cur), from D_{n2} = 0, and its tangent dD/dz (dz).
struct MieD {
    cplx cur, dz;
    __device__ __forceinline__ void start() { cur = dz = mk(0., 0.); }
    // from D_{n + 1} to D_n; DZ: the tangent too
    template <bool DZ>
    __device__ __forceinline__ void step(int n, cplx zinv, cplx zinv2) {
        const double s = n + 1.;
        const cplx g = mk(__dmul_rn(s, zinv.re), __dmul_rn(s, zinv.im));
        const cplx e = mk(__dadd_rn(cur.re, g.re), __dadd_rn(cur.im, g.im));
        const double d = 1. / fma(e.re, e.re, e.im * e.im);
        const cplx i = mk(__dmul_rn(e.re, d), -__dmul_rn(e.im, d));   // 1 / e
        if (DZ) {
            const cplx h = -s * zinv2;                                // dg/dz
            dz = cfma(dz + h, i * i, h);
        }
        cur = mk(__dsub_rn(g.re, i.re), __dsub_rn(g.im, i.im));
    }
    __device__ __forceinline__ void step(int n, cplx zinv) { step<false>(n, zinv, zinv); }
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
        const int e = mb_exp(hi, hi), g = e <= 40 && e >= -40 ? 0 : e;
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

// One order of the ratio r_n = psi_n / psi_{n-1} and its tangent, from those of order n + 1 (zeros at n1).
__device__ __forceinline__ void mie_ratio(int n, double xinv, double &r, double &rx) {
    const double c = (2. * n + 1.) * xinv, q = 1. / (c - r);
    rx = fma(c, xinv, rx) * (q * q);
    r = q;
}

// dD/dz of D_n from the Riccati equation
template <bool HX>
__device__ __forceinline__ cplx mie_dz(const MieRadius<HX> &c, int n, cplx D) {
    const cplx nz = (double) n * c.zinv;
    return cfma(nz - D, nz + D, cfma(c.zinv2, (double) n, mk(-1., 0.)));
}

// The tangent dz of D's recurrence as what it corrects the Riccati equation's
// dD/dz by: that is a rounding of terms of order 1, and 24 bits of it are more
// than the sum can hold.
template <bool HX>
__device__ __forceinline__ float2 mie_dz_corr(const MieRadius<HX> &c, int n, cplx D, cplx dz) {
    const cplx e = dz - mie_dz(c, n, D);
    return make_float2((float) e.re, (float) e.im);
}
__device__ __forceinline__ cplx mie_dz_add(cplx ric, float2 e) { return mk(ric.re + (double) e.x, ric.im + (double) e.y); }

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
    // order n, p the coefficients of order n - 1 (zeros for n = 1); the asymmetry
    // factors of order n - 1: f3 = (n^2 - 1) / n, f4 = (2n - 1) / (n (n - 1)) (n = 1: any finite ones)
    __device__ __forceinline__ void add(int n, const MieAB &q, const MieAB &p, double f3, double f4) {
        const double f1 = 2. * n + 1., sgn = (n & 1) ? -f1 : f1;
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

// The block's radii, G of them, of one refractive index, in
// shared memory laid out for `rows`.  common(c) sets up what the radii share,
// radius(g, c, n1, n2) radius g; factors(n, f3, f4) gives MieSums::add's;
// begin(g) is called by a radius' team, then store(n, ab) once per order, by one
// thread each, and sum(sums) by all its threads.  dz: some of them take dD/dz from
// D's recurrence.
template <bool HM, bool HX, int TEAM, class Common, class Radius, class Factors, class Begin, class Store, class Sum>
__device__ __forceinline__ void mie_block(unsigned char *smem, int rows, bool dz, int G, Common &&common, Radius &&radius,
                                          Factors &&factors, Begin &&begin, Store &&store, Sum &&sum) {
    constexpr int T = MIE_BLOCK_T, W = T / 32, NP = HX ? 12 : 8, NS = MieSums<HM, HX>::N;
    static_assert(TEAM == T || TEAM == 32, "the block or a warp");
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    double2 *Ds = (double2 *) smem;
    float2 *Dzs = (float2 *) (Ds + rows);
    double *u = (double *) (dz ? Dzs + rows : Dzs), *chi = u + rows, *ux = chi + rows;
    double *pass = chi + rows + (HX ? rows : 0);      // [W][12] last coefficients of a warp
    double *red = pass + W * 12;                      // [20][W]
    // psi_n = spsi u_n 2^(eU[n / MIE_B] - eu)
    double *sh_psi = red + 20 * W, *sh_psix = sh_psi + MIE_BLOCK_MAX;
    double *sh_x = sh_psix + MIE_BLOCK_MAX, *sh_xinv = sh_x + MIE_BLOCK_MAX, *sh_zr = sh_xinv + MIE_BLOCK_MAX;
    double *sh_zi = sh_zr + MIE_BLOCK_MAX, *sh_xl = sh_zi + MIE_BLOCK_MAX;
    int *sh_eu = (int *) (sh_xl + MIE_BLOCK_MAX), *sh_row = sh_eu + MIE_BLOCK_MAX, *sh_n1 = sh_row + MIE_BLOCK_MAX;
    int *eU = sh_n1 + 2 * MIE_BLOCK_MAX, *eP = eU + rows / MIE_B;
    constexpr bool DER = HM || HX;
    auto chain_d = [](int n1) { return DER || n1 < MIE_P_MIN; };   // D itself in Ds, or P

    MieRadius<HX> c;
    common(c);
    if (warp < 3) {
        int n1 = 0, n2 = 0;
        if (lane < G) radius(lane, c, n1, n2);
        // first row: the rows of the radii before
        const int own = lane < G ? mie_block_rows(n1) : 0;
        int row = own;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int v = __shfl_up_sync(0xffffffffu, row, o);
            if (lane >= o) row += v;
        }
        row -= own;
        // The lanes' chains go block by block of MIE_B orders together, each at
        // its own order; a chain's first block is entered at its order.
        if (lane >= G) {
        } else if (warp == 0) {
            sh_row[lane] = row;
            sh_n1[lane] = n1;
            sh_x[lane] = c.x;
            sh_xinv[lane] = c.xinv;
            sh_zr[lane] = c.zinv.re;
            sh_zi[lane] = c.zinv.im;
            if (HX) sh_xl[lane] = c.xl;
            double2 *Dr = Ds + row;
            if (chain_d(n1)) {
                MieD p;
                p.start();
                if (DER && dz) {
                    float2 *Zr = Dzs + row;
                    for (int n = n2 - 1; n > n1; --n) p.step<true>(n, c.zinv, c.zinv2);
#pragma unroll 4
                    for (int n = n1; n >= 1; --n) {
                        p.step<true>(n, c.zinv, c.zinv2);
                        Dr[n] = make_double2(p.cur.re, p.cur.im);
                        Zr[n] = mie_dz_corr(c, n, p.cur, p.dz);
                    }
                } else {
                    for (int n = n2 - 1; n > n1; --n) p.step(n, c.zinv);
                    for (int n = n1; n >= 1; --n) {   // n2 > n1
                        p.step(n, c.zinv);
                        Dr[n] = make_double2(p.cur.re, p.cur.im);
                    }
                }
            } else {
                MieP p;
                p.hi = mk(1., 0.);                    // P_{n2} = 1, P_{n2 - 1} = n2 / z
                p.cur = (double) n2 * c.zinv;
                int *er = eP + row / MIE_B, b = (n2 - 1) / MIE_B, e = 0;
                for (int n = n2 - 1; n >= b * MIE_B; --n) p.step(p.next(n, c.zinv));   // n2 > n1 + 2 MIE_B
                e += p.rescale();
                for (--b; b * MIE_B > n1; --b) {
#pragma unroll
                    for (int i = MIE_B - 1; i >= 0; --i) p.step(p.next(b * MIE_B + i, c.zinv));
                    e += p.rescale();
                }
                for (; b >= 0; --b) {
                    er[b] = e;
#pragma unroll
                    for (int i = MIE_B - 1; i >= 0; --i) {
                        Dr[b * MIE_B + i] = make_double2(p.cur.re, p.cur.im);
                        p.step(p.next(b * MIE_B + i, c.zinv));
                    }
                    e += p.rescale();
                }
            }
        } else if (HX && warp == 1 && n1 < MIE_P_MIN) {
            // psi and psi' themselves in the place of u and its tangent
            double *ur = u + row, *uxr = ux + row, r = 0., rx = 0.;
            int *er = eU + row / MIE_B;
            ur[n1] = uxr[n1] = 0.;
            for (int n = n1 - 1; n >= 1; --n) {
                mie_ratio(n, c.xinv, r, rx);
                ur[n] = r;
                uxr[n] = rx;
            }
            double psi, px;
            sincos(c.x, &psi, &px);
            for (int n = 0; n <= n1; ++n) {
                if (n > 0) {
                    px = fma(uxr[n], psi, ur[n] * px);
                    psi = ur[n] * psi;
                }
                ur[n] = psi;
                uxr[n] = px;
                er[n / MIE_B] = 0;
            }
            sh_psi[lane] = 1.;
            sh_psix[lane] = 0.;
            sh_eu[lane] = 0;
        } else if (warp == 1) {
            MieU<HX> q;
            q.start();
            double *ur = u + row, *uxr = ux + row;
            int *er = eU + row / MIE_B, b = n1 / MIE_B, e = 0;
            er[b] = 0;
            for (int n = n1; n >= b * MIE_B; --n) {
                ur[n] = q.cur;
                if (HX) uxr[n] = q.xcur;
                if (n > 0) q.step(n, c.xinv);
            }
            for (--b; b >= 0; --b) {
                e += q.rescale();
                er[b] = e;
#pragma unroll
                for (int i = MIE_B - 1; i >= 0; --i) {
                    ur[b * MIE_B + i] = q.cur;
                    if (HX) uxr[b * MIE_B + i] = q.xcur;
                    if (b + i > 0) q.step(b * MIE_B + i, c.xinv);
                }
            }
            const double spsi = sin(c.x) / q.cur;
            sh_psi[lane] = spsi;
            if (HX) sh_psix[lane] = fma(-spsi, q.xcur, cos(c.x)) / q.cur;
            sh_eu[lane] = e;
        } else {
            double sinx, cosx;
            sincos(c.x, &sinx, &cosx);
            double lo = cosx, cur = fma(c.xinv, cosx, sinx);
            double *cr = chi + row;
            cr[0] = lo;
#pragma unroll 4
            for (int n = 1; n <= n1; ++n) {
                cr[n] = cur;
                const double nx = fma((2. * n + 1.) * c.xinv, cur, -lo);
                lo = cur;
                cur = nx;
            }
        }
    }
    __syncthreads();

    for (int g = TEAM == 32 ? warp : 0; g < G; g += TEAM == 32 ? W : 1) {
        begin(g);
        const int n1 = sh_n1[g];
        c.x = sh_x[g];
        c.xinv = sh_xinv[g];
        c.zinv = mk(sh_zr[g], sh_zi[g]);
        c.zinv2 = c.zinv * c.zinv;
        if (HX) c.xl = sh_xl[g];
        const double spsi = sh_psi[g], spsix = HX ? sh_psix[g] : 0.;
        const int eu0 = sh_eu[g], row = sh_row[g];
        const double2 *Dr = Ds + row;
        const float2 *Zr = Dzs + row;
        const bool zr = DER && dz && mie_dz_chain(c.m, c.x);
        const double *ur = u + row, *uxr = ux + row, *cr = chi + row;
        const int *eur = eU + row / MIE_B;
        MieSums<HM, HX> sums;
        sums.zero();
        // the coefficients of the order before: from the lane before, for lane 0 from lane 31 of the warp before
        // (order 0: zeros) or of the round before, kept in `last`
        double last[NP];
#pragma unroll
        for (int q = 0; q < NP; ++q) last[q] = 0.;
        for (int j0 = 0; j0 < n1; j0 += TEAM) {
            const int j = j0 + (TEAM == 32 ? lane : tid) + 1;
            const bool on = j <= n1;
            MieAB q;
            q.a = q.b = q.am = q.bm = q.ax = q.bx = mk(0., 0.);
            if (on) {
                const double2 dj = Dr[j];
                cplx D = mk(dj.x, dj.y), Dz = mk(0., 0.);
                if (DER) {
                    Dz = mie_dz(c, j, D);
                    if (zr) Dz = mie_dz_add(Dz, Zr[j]);
                }
                if (!chain_d(n1)) {
                    const double2 lo = Dr[j - 1];
                    const int *er = eP + row / MIE_B;
                    const double sc = j % MIE_B == 0 ? mb_pow2(er[j / MIE_B - 1] - er[j / MIE_B]) : 1.;
                    D = mk(lo.x * sc, lo.y * sc) * cinv(D) - (double) j * c.zinv;
                }
                const double s1 = mb_pow2(eur[j / MIE_B] - eu0), s0 = mb_pow2(eur[(j - 1) / MIE_B] - eu0);
                const double psi = spsi * ur[j] * s1, psi_p = spsi * ur[j - 1] * s0;
                double psix = 0., psix_p = 0.;
                if (HX) {
                    psix = c.xl * (fma(spsix, ur[j], spsi * uxr[j]) * s1);
                    psix_p = c.xl * (fma(spsix, ur[j - 1], spsi * uxr[j - 1]) * s0);
                }
                q = mie_ab<HM, HX>(c, j, D, Dz, psi, psi_p, cr[j], cr[j - 1], psix, psix_p);
                store(j, q);
            }
            double v[12] = {q.a.re, q.a.im, q.b.re, q.b.im};
            if (HM) { v[4] = q.am.re; v[5] = q.am.im; v[6] = q.bm.re; v[7] = q.bm.im; }
            if (HX) { v[NP - 4] = q.ax.re; v[NP - 3] = q.ax.im; v[NP - 2] = q.bx.re; v[NP - 1] = q.bx.im; }
            constexpr int NV = 4 * (1 + HM + HX);
            if (TEAM != 32) {
                if (lane == 31)
#pragma unroll
                    for (int k = 0; k < NP; ++k) pass[warp * 12 + k] = v[k];
                __syncthreads();
            }
            MieAB p;
            p.am = p.bm = p.ax = p.bx = mk(0., 0.);
            double w[12];
#pragma unroll
            for (int k = 0; k < NP; ++k) {
                if (k >= NV && !(HX && k >= NP - 4)) continue;
                w[k] = __shfl_sync(0xffffffffu, TEAM == 32 && lane == 31 ? last[k] : v[k], (lane + 31) & 31);
                if (TEAM == 32) {
                    last[k] = v[k];
                } else {
                    if (lane == 0) w[k] = warp == 0 ? last[k] : pass[(warp - 1) * 12 + k];
                    last[k] = pass[(W - 1) * 12 + k];
                }
            }
            p.a = mk(w[0], w[1]);
            p.b = mk(w[2], w[3]);
            if (HM) { p.am = mk(w[4], w[5]); p.bm = mk(w[6], w[7]); }
            if (HX) { p.ax = mk(w[NP - 4], w[NP - 3]); p.bx = mk(w[NP - 2], w[NP - 1]); }
            if (on) {
                double f3, f4;
                factors(j, f3, f4);
                sums.add(j, q, p, f3, f4);
            }
            if (TEAM != 32) __syncthreads();
        }
#pragma unroll
        for (int q = 0; q < NS; ++q) {
            double v = sums.v[q];
#pragma unroll
            for (int o = 16; o; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
            sums.v[q] = v;
            if (TEAM != 32 && lane == 0) red[q * W + warp] = v;
        }
        if (TEAM != 32) {
            __syncthreads();
#pragma unroll
            for (int q = 0; q < NS; ++q) {
                sums.v[q] = red[q * W];
#pragma unroll
                for (int w = 1; w < W; ++w) sums.v[q] += red[q * W + w];
            }
        }
        sums.close();
        sum(sums);
    }
}

}  // namespace
#endif
