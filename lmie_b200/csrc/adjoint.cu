// adjoint.cu -- lmie_solution_adjoint: reverse-mode gradient of an
// output-weighted scalar of many wavelengths sharing one binned size
// distribution (include/lmie_b200.h).  No counterpart in the reference; its
// forward model is the reference's Mie solution (src/lmie_core.c:263-790,
// src/lmie_schedule.c:1155-1199) for the per-radius SIZE_DIST_MONO solves
// combined with the bin weights.
//
// Per wavelength k (a "case") and quadrature radius r, with W_r = weight[b] q_r:
//   e_r = sum_n (2n+1) Re(a_n + b_n),  s_r = sum_n (2n+1)(|a_n|^2 + |b_n|^2),
//   g_r = sum_{n<n1} fv3_n Re(a_n a_{n+1}* + b_n b_{n+1}*) + fv4_n Re(a_n b_n*),
//   sp, sm at the user angles (sp = sum_n (pi_n + tau_n) fv4_n (a_n + b_n), sm
//   likewise with -), F11 = (|sp|^2 + |sm|^2)/4, F12 = -Re(sp sm*)/2,
//   phi_r = sum_i d11_i F11(theta_i) + d12_i F12(theta_i);
//   E = sum W e, S = sum W s, G = sum W g, Phi = sum W phi, N = sum W;
//   Cext = kappa E / N, Csca = kappa S / N (kappa = lambda^2 / 2 pi), g = 2 G / S,
//   P11 = 2 sum W F11 / S, P12 = 2 sum W F12 / S,
//   L_k = c_cext Cext + c_csca Csca + 2 (c_g G + Phi) / S.
// Reverse sweep: dL/dE, dL/dS, dL/dG, dL/dPhi, dL/dN per wavelength; per
// radius the adjoints of a_n, b_n (conj-gradient convention a_bar =
// dL/dRe a + i dL/dIm a) from the cross-section sums and, through the
// transposed angular contraction, from phi; then with the complex derivatives
// A_n = da_n/dm, B_n = db_n/dm,
//   dL/dmr = Re sum (conj(a_bar) A + conj(b_bar) B),  dL/dmi = Im sum (...)
// (m = mr - i mi).  The coefficients and A_n, B_n come from the recurrences
// and formulas of the solves (mie_radius.cuh); the reverse sweep reads them.
#include <algorithm>
#include <climits>
#include <cmath>
#include <cstdio>
#include <cstring>
#include <mutex>
#include <vector>

#include "dev_common.cuh"
#include "mie_radius.cuh"
#include "../../include/lmie_b200.h"

extern "C" int lmieb_calc_n1(double x);
extern "C" void lmieb_host_parallel(int n, int n_threads, void (*fn)(void *, int), void *arg);
extern "C" int lmieb_calc_n2(int n1, double zr, double zi);
extern "C" void lmieb_gauss_leg(int n, double x1, double x2, double *x, double *w);

namespace {

constexpr int ADJ_T = 128;         // threads of the angular and the summing kernels
constexpr int ADJ_GR = 32;         // radii per block of the angular kernel

struct Adj {
    int L, R;                      // wavelengths, radii
    int na, nhu;                   // user angles, half-angles (theta <= 90 deg)
    int G;                         // radius groups of the angular kernel
    const double *lam;             // [L]
    const cplx *m;                 // [L]
    const double *W, *q;           // [R]
    const double *rad;             // [R]
    const int *n1, *n2;            // [L*R]
    const int *ro;                 // [L*R] orders of the wavelength's radii before this one
    const long long *ko;           // [L] orders of the pass' wavelengths before this one
    const double *mu;              // [nhu] cosines of the half-angles
    int nt;                        // tiles of 8 half-angles (nhu rounded up, zeros there)
    int nrow;                      // orders in the tables
    double2 *tabf, *tabb;          // {X_n, Y_n}(mu_h) in the order of the angular kernel's fragments
    const double2 *dw;             // [L][8 nt][2] {d11, d12} / 2 at the half-angles and their mirrors (zeros: none)
    const double *cw;              // [L][3] c_cext, c_csca, c_g
    double4 *c4;                   // per order: fv4 (a + b), fv4 (a - b)
    double4 *d4;                   // per order: da/dm, db/dm
    double4 *b4;                   // per order: the adjoints of c4 per W dL/dPhi (before that, K1's checkpoints)
    double *esg;                   // [L*R][4] e, s, g, phi
    double *pfp;                   // [L][G][na][2] partial sums of W F11, W F12
    double *lw;                    // [L][8] dL/dE, dL/dS, dL/dG, dL/dPhi, dL/dN, loss, Cext, Csca
    double *vals;                  // [L][3 + 2 na]
    double *zr;                    // [L*R][3] dL/dmr, dL/dmi, dL/dW of the radius
    double *gout;                  // [2 L + n_bins] gradient outputs
    int n_bins;
    const int *bstart;             // [n_bins + 1] radii of each bin
};

__device__ __forceinline__ double fv3d(int j) { return (j + 2.) * j / (j + 1.); }
__device__ __forceinline__ double fv4d(int j) { return (2. * j + 1.) / (j * (j + 1.)); }

__device__ __forceinline__ long long order_offset(const Adj &P, int k, int r) {
    return P.ko[k] + P.ro[(size_t) k * P.R + r];
}

__device__ __forceinline__ void st4(double4 *p, double a, double b, double c, double d) {
    asm volatile("st.global.v4.f64 [%0], {%1, %2, %3, %4};" ::"l"(p), "d"(a), "d"(b), "d"(c), "d"(d) : "memory");
}
__device__ __forceinline__ double4 ld4(const double4 *p) {
    double4 v;
    asm volatile("ld.global.v4.f64 {%0, %1, %2, %3}, [%4];" : "=d"(v.x), "=d"(v.y), "=d"(v.z), "=d"(v.w) : "l"(p));
    return v;
}

// ---- forward: coefficients, their derivatives, cross-section sums (thread per (k, r)) ----
// K1's thread-per-radius form (k_mie.cu), with the checkpoints of a radius in
// the place of its adjoints: 5 doubles for every 4 orders where those take 16.
__global__ void __launch_bounds__(64) k_adj_coef(Adj P) {
    const int nrb = (P.R + 63) / 64, k = blockIdx.x % P.L;
    const int r = (nrb - 1 - (int) (blockIdx.x / P.L)) * 64 + threadIdx.x;   // large radii first
    if (r >= P.R) return;
    const size_t t = (size_t) k * P.R + r;
    const int n1 = P.n1[t], n2 = P.n2[t];
    const cplx m = P.m[k];
    MieRadius<false> c;
    c.set_m(m, cinv(m), mk(0., 0.));
    c.set_x(2. * LMIEB_PI * P.rad[r] / P.lam[k], 0.);
    const long long off = order_offset(P, k, r);
    double *const ck = (double *) (P.b4 + off);
    const int nb = n1 / MIE_B + 1;
    double u0;
    int eu = 0;
    {
        MieD p;
        p.start();                                   // D_{n2} = 0, n2 > n1 + MIE_B
        for (int n = n2 - 1; n >= nb * MIE_B; --n) p.step(n, c.zinv);
        MieU<false> q;
        q.start();
        for (int b = nb - 1; b >= 0; --b) {
            double *w = ck + 5 * b;
            w[0] = p.cur.re; w[1] = p.cur.im; w[2] = q.hi; w[3] = q.cur; w[4] = (double) eu;
#pragma unroll
            for (int i = MIE_B - 1; i >= 0; --i) {
                const int n = b * MIE_B + i;
                if (b > 0 || i > 0) p.step(n, c.zinv);
                if (n <= n1 && (b > 0 || i > 0)) q.step(n, c.xinv);
            }
            if (b > 0) eu += q.rescale();
        }
        u0 = q.cur;
    }
    double sinx, cosx;
    sincos(c.x, &sinx, &cosx);
    const double spsi = sinx / u0;
    double chi_p = cosx, chi = fma(c.xinv, cosx, sinx), psi_p = spsi * u0;
    MieSums<false, false> sums;
    sums.zero();
    MieAB prev;
    prev.a = prev.b = prev.am = prev.bm = prev.ax = prev.bx = mk(0., 0.);
    double f4p = 0.;                                  // fv4 of the order before
    for (int b = 0; b < nb; ++b) {
        const double *w = ck + 5 * b;
        cplx D[MIE_B], Dz[MIE_B];
        double ub[MIE_B];
        const double su = mb_pow2((int) w[4] - eu);
        MieD p;
        p.cur = mk(w[0], w[1]);
        MieU<false> u;
        u.hi = w[2];
        u.cur = w[3];
#pragma unroll
        for (int i = MIE_B - 1; i >= 0; --i) {
            const int n = b * MIE_B + i;
            ub[i] = u.cur;
            if (n > 0) {
                p.step(n, c.zinv);
                if (n <= n1) {
                    D[i] = p.cur;
                    Dz[i] = mie_dz(c, n, p.cur);
                    u.step(n, c.xinv);
                }
            }
        }
#pragma unroll
        for (int i = 0; i < MIE_B; ++i) {
            const int j = b * MIE_B + i;
            if (j < 1 || j > n1) continue;
            const double psi = spsi * ub[i] * su, f4 = fv4d(j), f3 = (double) (j - 1) * (j + 1) / j;
            const MieAB q = mie_ab<true, false>(c, j, D[i], Dz[i], psi, psi_p, chi, chi_p, 0., 0.);
            sums.add(j, q, prev, f3, f4p);
            st4(P.c4 + off + j - 1, f4 * (q.a.re + q.b.re), f4 * (q.a.im + q.b.im), f4 * (q.a.re - q.b.re),
                f4 * (q.a.im - q.b.im));
            st4(P.d4 + off + j - 1, q.am.re, q.am.im, q.bm.re, q.bm.im);
            const double chi_n = fma((2. * j + 1.) * c.xinv, chi, -chi_p);
            chi_p = chi;
            chi = chi_n;
            psi_p = psi;
            prev = q;
            f4p = f4;
        }
    }
    double *o = P.esg + t * 4;
    o[0] = sums.v[0];
    o[1] = sums.v[1];
    o[2] = sums.v[4];
}

__device__ __forceinline__ double block_sum128(double v, double *sh) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    __syncthreads();
    if ((threadIdx.x & 31) == 0) sh[threadIdx.x >> 5] = v;
    __syncthreads();
    double s = 0.;
#pragma unroll
    for (int w = 0; w < ADJ_T / 32; ++w) s += sh[w];
    return s;
}

// ---- pi_n, tau_n at the half-angles (thread per half-angle) ----
// The angular kernel sums over odd and even orders at once.  With sp(mu) =
// sum c_n (pi_n + tau_n), sm(mu) = sum d_n (pi_n - tau_n) and, at the mirror
// angle, pi_n -> s_n pi_n, tau_n -> -s_n tau_n (s_n = -(-1)^n),
//   X_n = pi_n (n odd), tau_n (n even),   Y_n the other one,
//   x = sum c_n X_n, y = sum c_n Y_n:            sp = x + y, sp(-mu) = x - y,
//   x = sum s_n d_n X_n, y = sum s_n d_n Y_n:    sm = x - y, sm(-mu) = x + y,
// half the products of four separate sums; likewise the transposed sums.
__global__ void k_adj_table(Adj P) {
    const int h = threadIdx.x;                          // 8 nt threads
    const double mu = h < P.nhu ? P.mu[h] : 0., on = h < P.nhu ? 1. : 0.;
    double p0 = 0., p1 = on;
    for (int n = 0; n < P.nrow; ++n) {                  // order n + 1
        const double o = n + 1., tau = fma(o * mu, p1, -(o + 1.) * p0);
        const double2 v = (n & 1) ? make_double2(tau, p1) : make_double2(p1, tau);
        const int t = h >> 3, c = h & 7;
        P.tabf[((size_t) (n >> 2) * P.nt + t) * 32 + c * 4 + (n & 3)] = v;
        P.tabb[(((size_t) (n >> 3) * P.nt + t) * 2 + (c & 1)) * 32 + (n & 7) * 4 + (c >> 1)] = v;
        const double r = 1. / o, p2 = fma(fma(2., o, 1.) * r * mu, p1, -(o + 1.) * r * p0);
        p0 = p1;
        p1 = p2;
    }
}

// c += a b: a one element of 8 x 4 (row lane / 4, column lane % 4), b one of
// 4 x 8 (row lane % 4, column lane / 4), c two of 8 x 8 (row lane / 4, columns
// 2 (lane % 4) and the next)
__device__ __forceinline__ void dmma(double (&c)[2], double a, double b) {
    asm("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0, %1}, {%2}, {%3}, {%0, %1};"
        : "+d"(c[0]), "+d"(c[1])
        : "d"(a), "d"(b));
}

// ---- both angular sweeps (block per (k, group of ADJ_GR radii)) ----
// Forward: sp, sm at the user angles, the phase matrix sums, phi_r; reverse:
// the adjoints of the coefficient columns from those of sp, sm.  These are
// linear in W dL/dPhi, which is known only when all radii have been summed: it
// is left out here and put in by k_adj_m, so that the sums over orders are
// formed once and stay in registers between the sweeps.
//
// A warp takes two radii at a time as the 8 rows of FP64 m8n8k4 products: row =
// (radius, {c.re, c.im, s d.re, s d.im}).  Forward, columns = 8 half-angles,
// K = orders; the sums of all half-angles are the accumulators (4 NT doubles).
// Reverse, columns = 8 orders, K = half-angles: an accumulator's two columns
// are half-angles 2 q and 2 q + 1 of its tile, which are taken as the K
// elements q of two products, so the accumulators are the operands as they are
// (tabb is laid out for that).  Bound by the FP64 pipe: 16 FMAs per order and
// half-angle.  256 wavelengths x 2048 radii x 181 angles (17.8 M orders):
// 3.0 ms (a thread per half-angle, radius by radius, with the forward sums
// formed again for the reverse sweep: 12.1 ms); the FMAs take 1.5 ms.
template <int NT>
__global__ void __launch_bounds__(ADJ_T, NT > 12 ? 2 : 3) k_adj_angles(Adj P) {
    constexpr int PF = NT > 6 && NT % 2 == 0 ? NT / 2 : NT;   // table entries loaded ahead
    extern __shared__ double psum[];                    // [4 warps][2 NT][32]: sums of F11, F12 over radii
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int q = lane & 3, row = lane >> 2, comp = row & 3, rr = row >> 2;
    const int k = blockIdx.x % P.L, grp = P.G - 1 - blockIdx.x / P.L;   // large radii first
    // Of the two values x + y, x - y of a half-angle, lane bit 2 tells which is
    // this lane's first: the first values of lanes 0-3 and 4-7 (components 0
    // and 1) are then those of an angle and of its mirror.  The sign of y does
    // this, together with sm's (table kernel).
    const bool b2 = lane & 4, b3 = lane & 8, flip = b2 != (comp >= 2);
    const double2 *dw = P.dw + (size_t) k * 16 * NT + 4 * q + b2;
    const int dwo = b2 ? -1 : 1;
    double *const ps = psum + warp * (2 * NT * 32) + lane;
#pragma unroll
    for (int i = 0; i < 2 * NT; ++i) ps[i * 32] = 0.;
    // This lane's radius of pair p and its coefficients are loaded a pair ahead,
    // further ones four steps ahead: the coefficients come from DRAM.
    const int r0 = grp * ADJ_GR + warp * (ADJ_GR / 4) + rr;
    const long long t0 = (long long) k * P.R;
    auto orders = [&](int p) { return p < ADJ_GR / 8 && r0 + 2 * p < P.R ? P.n1[t0 + r0 + 2 * p] : 0; };
    auto offset = [&](int p) { return order_offset(P, k, min(r0 + 2 * p, P.R - 1)); };
    auto column = [&](long long o) { return (const double *) (P.c4 + o) + comp; };
    int n1 = orders(0);
    long long off = offset(0);
    double a[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) a[i] = 4 * i + q < n1 ? column(off)[4 * (4 * i + q)] : 0.;
    for (int p = 0; p < ADJ_GR / 8; ++p) {
        const int r = r0 + 2 * p, n1_next = orders(p + 1);
        const bool on = r < P.R;
        const long long t = t0 + (on ? r : 0), off_next = offset(p + 1);
        const double W = on ? P.W[r] : 0.;
        const int nmax = max(n1, __shfl_xor_sync(0xffffffffu, n1, 16));
        if (nmax == 0) break;
        const double *src = column(off);
        double X[NT][2], Y[NT][2];
#pragma unroll
        for (int i = 0; i < NT; ++i) X[i][0] = X[i][1] = Y[i][0] = Y[i][1] = 0.;
        {
            // the next four orders' table entries are loaded as these are used
            const double2 *tb = P.tabf + lane;
            double2 b[PF];
#pragma unroll
            for (int i = 0; i < PF; ++i) b[i] = tb[i * 32];
            for (int n0 = 0; n0 < nmax; n0 += 4) {
                const int nn = n0 + q + 16;
                const double ax = comp >= 2 && (q & 1) ? -a[0] : a[0], ay = flip ? -ax : ax;
                a[0] = a[1];
                a[1] = a[2];
                a[2] = a[3];
                a[3] = nn < n1 ? src[4 * nn] : 0.;
#pragma unroll
                for (int i = 0; i < NT; ++i) {
                    dmma(X[i], ax, b[i % PF].x);
                    dmma(Y[i], ay, b[i % PF].y);
                    b[i % PF] = tb[(i + PF) * 32];
                }
                tb += NT * 32;
            }
        }
        // phase matrix elements and the adjoints of sp, sm: this lane has one
        // real component of (sp, sm) at an angle (v1) and at its mirror (v2), or
        // the other way round
        double phi = 0.;
#pragma unroll
        for (int i = 0; i < NT; ++i)
#pragma unroll
            for (int j = 0; j < 2; ++j) {
                const double v1 = X[i][j] + Y[i][j], v2 = X[i][j] - Y[i][j];
                // sm's component for sp's and the other way round
                const double p1 = __shfl_xor_sync(0xffffffffu, v1, 8), p2 = __shfl_xor_sync(0xffffffffu, v2, 8);
                const double2 w1 = dw[16 * i + 2 * j], w2 = dw[16 * i + 2 * j + dwo];
                const double s1 = w1.x * v1 - w1.y * p1, s2 = w2.x * v2 - w2.y * p2;
                phi += v1 * s1 + v2 * s2;
                X[i][j] = s1 + s2;
                Y[i][j] = s1 - s2;
                // sums over the four components, those of F12 twice the same two; of the two radii at the end
                double f = v1 * v1 + __shfl_xor_sync(0xffffffffu, v2 * v2, 4);
                const double g = v1 * p1 + __shfl_xor_sync(0xffffffffu, v2 * p2, 4);
                f += __shfl_xor_sync(0xffffffffu, f, 8);
                ps[(2 * i + j) * 32] += W * (b3 ? g : f);
            }
#pragma unroll
        for (int o = 1; o < 16; o <<= 1) phi += __shfl_xor_sync(0xffffffffu, phi, o);
        if (on && (lane & 15) == 0) P.esg[(size_t) t * 4 + 3] = .5 * phi;
#pragma unroll
        for (int i = 0; i < 4; ++i) a[i] = 4 * i + q < n1_next ? column(off_next)[4 * (4 * i + q)] : 0.;
        // the adjoints of the coefficient columns, 8 orders at a time (this lane: two of them)
        double *dst = (double *) (P.b4 + off) + comp;
        const double2 *tb = P.tabb + lane;
        double2 b[PF];
#pragma unroll
        for (int i = 0; i < PF; ++i) b[i] = tb[i * 32];
        for (int n0 = 0; n0 < nmax; n0 += 8) {
            double o[4][2] = {};                        // chains of products
#pragma unroll
            for (int i = 0; i < 2 * NT; ++i) {
                dmma(o[i & 1], X[i >> 1][i & 1], b[i % PF].x);
                dmma(o[2 + (i & 1)], Y[i >> 1][i & 1], b[i % PF].y);
                b[i % PF] = tb[(i + PF) * 32];
            }
            tb += 2 * NT * 32;
            const int n = n0 + 2 * q;
            const double y0 = o[2][0] + o[3][0], y1 = o[2][1] + o[3][1];
            const double v0 = (o[0][0] + o[1][0]) + (flip ? -y0 : y0), v1 = (o[0][1] + o[1][1]) + (flip ? -y1 : y1);
            if (n < n1) dst[4 * n] = v0;
            if (n + 1 < n1) dst[4 * n + 4] = comp >= 2 ? -v1 : v1;
        }
        n1 = n1_next;
        off = off_next;
    }
    __syncthreads();
    double *o = P.pfp + ((size_t) k * P.G + grp) * P.na * 2;
    for (int i = threadIdx.x; i < 4 * P.nhu; i += ADJ_T) {
        const int h = i >> 2, mir = i & 1, el = (i >> 1) & 1, hm = P.na - 1 - h;
        if (mir && hm == h) continue;
        const double *v = psum + ((h >> 3) * 2 + (h & 1)) * 32 + ((h & 7) >> 1) + 4 * mir + 8 * el;
        double sum = 0.;
        for (int w = 0; w < 4; ++w) sum += v[w * (2 * NT * 32)] + v[w * (2 * NT * 32) + 16];
        o[2 * (mir ? hm : h) + el] = el ? -.5 * sum : .25 * sum;
    }
}

// ---- per wavelength: loss, phase matrix, adjoints of the sums (block per k) ----
__global__ void __launch_bounds__(ADJ_T) k_adj_lambda(Adj P) {
    __shared__ double sh[ADJ_T / 32];
    const int k = blockIdx.x;
    double N = 0., E = 0., S = 0., Gs = 0., Ph = 0.;
    for (int r = threadIdx.x; r < P.R; r += ADJ_T) {
        const double W = P.W[r];
        const double *v = P.esg + ((size_t) k * P.R + r) * 4;
        N += W;
        E += W * v[0];
        S += W * v[1];
        Gs += W * v[2];
        Ph += W * v[3];
    }
    N = block_sum128(N, sh);
    E = block_sum128(E, sh);
    S = block_sum128(S, sh);
    Gs = block_sum128(Gs, sh);
    Ph = block_sum128(Ph, sh);
    const double lam = P.lam[k], kap = lam * lam / (2. * LMIEB_PI);
    const double *cw = P.cw + (size_t) k * 3;
    double *vals = P.vals + (size_t) k * (3 + 2 * P.na);
    for (int i = threadIdx.x; i < P.na; i += ADJ_T) {
        double a = 0., b = 0.;
        for (int g = 0; g < P.G; ++g) {
            const double *o = P.pfp + ((size_t) k * P.G + g) * P.na * 2;
            a += o[2 * i];
            b += o[2 * i + 1];
        }
        vals[3 + i] = 2. * a / S;
        vals[3 + P.na + i] = 2. * b / S;
    }
    if (threadIdx.x == 0) {
        double *o = P.lw + (size_t) k * 8;
        const double cext = kap * E / N, csca = kap * S / N, g = 2. * Gs / S;
        o[0] = cw[0] * kap / N;                                       // dL/dE
        o[1] = cw[1] * kap / N - 2. * (cw[2] * Gs + Ph) / (S * S);    // dL/dS
        o[2] = 2. * cw[2] / S;                                        // dL/dG
        o[3] = 2. / S;                                                // dL/dPhi
        o[4] = -(cw[0] * kap * E + cw[1] * kap * S) / (N * N);        // dL/dN
        o[5] = cw[0] * cext + cw[1] * csca + 2. * (cw[2] * Gs + Ph) / S;
        o[6] = cext;
        o[7] = csca;
        vals[0] = cext;
        vals[1] = csca;
        vals[2] = g;
    }
}

// ---- reverse: dL/dm of one radius (eight lanes per (k, r), orders dealt out) ----
// Bound by memory: 96 bytes per order, read once (the orders before from L1).
__global__ void __launch_bounds__(256) k_adj_m(Adj P) {
    const long long t = ((long long) blockIdx.x * blockDim.x + threadIdx.x) >> 3;
    const int lane = threadIdx.x & 7;
    const bool on = t < (long long) P.L * P.R;
    const int k = on ? (int) (t / P.R) : 0, r = on ? (int) (t % P.R) : 0;
    const int n1 = on ? P.n1[t] : 0;
    const double *lw = P.lw + (size_t) k * 8;
    const double W = P.W[r];
    const double aE = W * lw[0], aS = W * lw[1], aG = W * lw[2], aP = W * lw[3];
    const long long off = order_offset(P, k, r);
    cplx Z = mk(0., 0.);
    for (int j = lane + 1; j <= n1; j += 8) {
        const double4 c = ld4(P.c4 + off + j - 1), d = ld4(P.d4 + off + j - 1), v = ld4(P.b4 + off + j - 1);
        const double f1 = 2. * j + 1., f4 = fv4d(j), h = .5 / f4;
        const cplx a = mk(h * (c.x + c.z), h * (c.y + c.w)), b = mk(h * (c.x - c.z), h * (c.y - c.w));
        const cplx A = mk(d.x, d.y), Bd = mk(d.z, d.w);
        // adjoints of a_j, b_j except the a_{j+1}, b_{j+1} terms of g
        const double fp = aP * f4;
        cplx abar = mk(aE * f1, 0.) + a * (2. * aS * f1) + mk(v.x + v.z, v.y + v.w) * fp;
        cplx bbar = mk(aE * f1, 0.) + b * (2. * aS * f1) + mk(v.x - v.z, v.y - v.w) * fp;
        if (j < n1) {
            abar = abar + b * (aG * f4);
            bbar = bbar + a * (aG * f4);
        }
        if (j >= 2) {
            const double4 cp = ld4(P.c4 + off + j - 2), dp = ld4(P.d4 + off + j - 2);
            const double f3 = aG * fv3d(j - 1), hp = .5 / fv4d(j - 1) * f3;
            abar = abar + mk(hp * (cp.x + cp.z), hp * (cp.y + cp.w));
            bbar = bbar + mk(hp * (cp.x - cp.z), hp * (cp.y - cp.w));
            // the a_j, b_j term of the adjoints of a_{j-1}, b_{j-1}
            Z = Z + conjg(a) * mk(dp.x, dp.y) * f3 + conjg(b) * mk(dp.z, dp.w) * f3;
        }
        Z = Z + conjg(abar) * A + conjg(bbar) * Bd;
    }
#pragma unroll
    for (int o = 1; o < 8; o <<= 1) {
        Z.re += __shfl_xor_sync(0xffffffffu, Z.re, o);
        Z.im += __shfl_xor_sync(0xffffffffu, Z.im, o);
    }
    if (!on || lane) return;
    double *o = P.zr + (size_t) t * 3;
    o[0] = Z.re;   // dL/dmr of this radius
    o[1] = Z.im;   // dL/dmi
    const double *v = P.esg + (size_t) t * 4;
    o[2] = lw[0] * v[0] + lw[1] * v[1] + lw[2] * v[2] + lw[3] * v[3] + lw[4];   // dL/dW_r
}

// ---- gradients: dL/dmr, dL/dmi per wavelength, dL/dweight per bin ----
__global__ void __launch_bounds__(ADJ_T) k_adj_final(Adj P) {
    __shared__ double sh[ADJ_T / 32];
    if ((int) blockIdx.x < P.L) {
        const int k = blockIdx.x;
        double a = 0., b = 0.;
        for (int r = threadIdx.x; r < P.R; r += ADJ_T) {
            const double *o = P.zr + ((size_t) k * P.R + r) * 3;
            a += o[0];
            b += o[1];
        }
        a = block_sum128(a, sh);
        b = block_sum128(b, sh);
        if (threadIdx.x == 0) {
            P.gout[k] = a;
            P.gout[P.L + k] = b;
        }
    } else {
        const int bb = blockIdx.x - P.L;
        double s = 0.;
        const int r0 = P.bstart[bb], r1 = P.bstart[bb + 1];
        for (int i = threadIdx.x; i < P.L * (r1 - r0); i += ADJ_T) {
            const int k = i / (r1 - r0), r = r0 + i % (r1 - r0);
            s += P.q[r] * P.zr[((size_t) k * P.R + r) * 3 + 2];
        }
        s = block_sum128(s, sh);
        if (threadIdx.x == 0) P.gout[2 * P.L + bb] = s;
    }
}

// Tiles of 8 half-angles of the most angles that the entry point takes; there is
// a kernel for every number of them (the accumulators of all tiles stay in
// registers, and a tile too many costs as much as a used one).
constexpr int ADJ_MAX_TILES = (ADJ_T + 7) / 8;

template <int NT>
int launch_angles_nt(const Adj &P, cudaStream_t s) {
    constexpr int SMEM = 4 * 2 * NT * 32 * 8;
    static_assert(SMEM <= 48 * 1024, "no opt-in needed");
    k_adj_angles<NT><<<(unsigned) P.L * P.G, ADJ_T, SMEM, s>>>(P);
    LMIEB_CUDA_TRY(cudaGetLastError());
    return 0;
}

// the kernel of P.nt tiles
template <int NT = ADJ_MAX_TILES>
int launch_angles(const Adj &P, cudaStream_t s) {
    if (P.nt == NT) return launch_angles_nt<NT>(P, s);
    if constexpr (NT > 1) {
        return launch_angles<NT - 1>(P, s);
    } else {
        fprintf(stderr, "ERROR: lmie_solution_adjoint(): %d tiles of half-angles\n", P.nt);
        return -1;
    }
}

// device buffers of the last adjoint solve, kept for the next one
std::mutex g_amu;
char *g_dbuf = nullptr, *g_hbuf = nullptr;
size_t g_dcap = 0, g_hcap = 0;
bool g_dshort = false;             // the device had no room for all orders of that solve

// The columns of the orders (c4, d4, b4) are most of what a solve holds on the
// device, 96 bytes for every order of every radius and wavelength.  Where the
// device has no room for them all, the wavelengths go through in passes, as many
// at a time as fit ADJ_PASS_BYTES (still some 5 times the benchmark's 17.8 M
// orders, enough to fill the device) or the largest of them.
constexpr size_t ADJ_ORDER_BYTES = 3 * sizeof(double4), ADJ_PASS_BYTES = (size_t) 8 << 30;

size_t pad256(size_t b) { return (b + 255) & ~(size_t) 255; }

}  // namespace

extern "C" int lmieb_stream(void **stream);
extern "C" int lmieb_fault_injected(const char *site);

extern "C" int lmie_solution_adjoint(int n_lambda, const double *lambda, const double *mr, const double *mi,
                                     const lmie_bins *bins, int n_angles, const lmie_loss_weights *weights,
                                     double *loss, double *grad_mr, double *grad_mi, double *grad_weight,
                                     double *values) {
    if (n_lambda < 1 || !lambda || !mr || !mi || !bins || !weights || !loss || n_angles < 2 ||
        n_angles > 2 * ADJ_T - 1 || !bins->edges || !bins->weight || bins->n_bins < 1 || bins->n_quad < 1) {
        fprintf(stderr, "ERROR: lmie_solution_adjoint(): invalid arguments (n_angles must be 2..%d)\n",
                2 * ADJ_T - 1);
        return -1;
    }
    for (int b = 0; b < bins->n_bins; ++b)
        if (!(bins->edges[b] > 0.) || !(bins->edges[b + 1] > bins->edges[b]) || !(bins->weight[b] > 0.)) {
            fprintf(stderr, "ERROR: lmie_solution_adjoint(): bin %d: edges must ascend from > 0, weights > 0\n", b);
            return -1;
        }
    for (int k = 0; k < n_lambda; ++k)
        if (!(lambda[k] > 0.) || !(mr[k] > 0.) || !(mi[k] >= 0.)) {
            fprintf(stderr, "ERROR: lmie_solution_adjoint(): wavelength %d: lambda and mr must be > 0, mi >= 0\n", k);
            return -1;
        }
    void *sp = nullptr;
    if (lmieb_stream(&sp)) return -1;
    cudaStream_t s = (cudaStream_t) sp;
    std::lock_guard<std::mutex> lock(g_amu);

    const int L = n_lambda, nb = bins->n_bins, nq = bins->n_quad, R = nb * nq, na = n_angles;
    const int nhu = (na + 1) / 2, G = (R + ADJ_GR - 1) / ADJ_GR;
    // ---- inputs, in one pinned block; outputs in another part of it ----
    size_t in_bytes = 0;
    auto take = [&](size_t bytes) { const size_t at = in_bytes; in_bytes += pad256(bytes); return at; };
    const int nt = (nhu + 7) / 8;                       // tiles of 8 half-angles
    const size_t LR = (size_t) L * R;
    const size_t i_lam = take((size_t) L * 8), i_m = take((size_t) L * 16), i_W = take((size_t) R * 8);
    const size_t i_q = take((size_t) R * 8), i_rad = take((size_t) R * 8), i_bs = take((size_t) (nb + 1) * 4);
    const size_t i_n1 = take(LR * 4), i_n2 = take(LR * 4), i_ro = take(LR * 4), i_ko = take((size_t) L * 8);
    const size_t i_mu = take((size_t) nhu * 8), i_dw = take((size_t) L * 8 * nt * 32), i_cw = take((size_t) L * 3 * 8);
    const size_t out_vals = (size_t) L * (3 + 2 * na) * 8, out_lw = (size_t) L * 8 * 8;
    const size_t out_g = (size_t) (2 * L + nb) * 8;
    const size_t out_bytes = pad256(out_vals) + pad256(out_lw) + pad256(out_g);
    if (in_bytes + out_bytes > g_hcap) {
        if (g_hbuf) cudaFreeHost(g_hbuf);
        g_hbuf = nullptr;
        g_hcap = 0;
        LMIEB_CUDA_TRY(cudaMallocHost((void **) &g_hbuf, in_bytes + out_bytes));
        g_hcap = in_bytes + out_bytes;
    }
    char *const hb = g_hbuf;
    double *rad = (double *) (hb + i_rad), *q = (double *) (hb + i_q), *W = (double *) (hb + i_W);
    int *bstart = (int *) (hb + i_bs);
    for (int b = 0; b < nb; ++b) {
        bstart[b] = b * nq;
        lmieb_gauss_leg(nq, bins->edges[b], bins->edges[b + 1], rad + (size_t) b * nq, q + (size_t) b * nq);
        for (int i = 0; i < nq; ++i) W[b * nq + i] = bins->weight[b] * q[b * nq + i];
    }
    bstart[nb] = R;
    // the half-angles theta_h = h 180 / (na - 1), h < nhu
    double *mu = (double *) (hb + i_mu);
    for (int h = 0; h < nhu; ++h) mu[h] = cos(h * LMIEB_PI / (na - 1));
    // truncations and weights, one wavelength per task on the host's threads
    std::vector<long long> orders(L);
    std::vector<int> top(L);
    struct XJob {
        const double *rad, *lambda, *mr, *mi;
        const lmie_loss_weights *weights;
        double *lam;
        cplx *m;
        double *dw, *cw;
        int *n1, *n2, *ro;
        long long *orders;
        int *top;
        int R, na, nhu, nt;
    } xj{rad, lambda, mr, mi, weights, (double *) (hb + i_lam), (cplx *) (hb + i_m), (double *) (hb + i_dw),
         (double *) (hb + i_cw), (int *) (hb + i_n1), (int *) (hb + i_n2), (int *) (hb + i_ro), orders.data(), top.data(),
         R, na, nhu, nt};
    lmieb_host_parallel(L, 64, [](void *arg, int k) {
        const XJob &j = *(const XJob *) arg;
        const size_t t0 = (size_t) k * j.R;
        long long sum = 0;
        int top = 1;
        for (int r = 0; r < j.R; ++r) {
            const double x = 2. * LMIEB_PI * j.rad[r] / j.lambda[k];
            const int n1 = lmieb_calc_n1(x);
            j.n1[t0 + r] = n1;
            j.n2[t0 + r] = lmieb_calc_n2(n1, j.mr[k] * x, -j.mi[k] * x);
            j.ro[t0 + r] = (int) sum;
            sum += n1;
            top = std::max(top, n1);
        }
        j.orders[k] = sum;
        j.top[k] = top;
        j.lam[k] = j.lambda[k];
        j.m[k] = mk(j.mr[k], -j.mi[k]);
        const lmie_loss_weights &w = j.weights[k];
        j.cw[(size_t) k * 3] = w.c_cext;
        j.cw[(size_t) k * 3 + 1] = w.c_csca;
        j.cw[(size_t) k * 3 + 2] = w.c_g;
        double *dw = j.dw + (size_t) k * 8 * j.nt * 4;
        memset(dw, 0, (size_t) 8 * j.nt * 32);
        for (int i = 0; i < j.na; ++i) {
            double *o = dw + (i < j.nhu ? 4 * i : 4 * (j.na - 1 - i) + 2);
            o[0] = w.d_p11 ? .5 * w.d_p11[i] : 0.;
            o[1] = w.d_p12 ? .5 * w.d_p12[i] : 0.;
        }
    }, &xj);
    long long tot = 0, most = 0;                          // orders of all wavelengths, of the longest
    int n1max = 1, k_top = 0;
    for (int k = 0; k < L; ++k) {
        tot += orders[k];
        most = std::max(most, orders[k]);
        if (top[k] > n1max) {
            n1max = top[k];
            k_top = k;
        }
        if (orders[k] > INT_MAX) {
            fprintf(stderr, "ERROR: lmie_solution_adjoint(): %lld orders of wavelength %d\n", orders[k], k);
            return -1;
        }
    }
    // the longest radii this solve accepts
    if ((size_t) 2 * n1max * sizeof(cplx) + (size_t) 4 * nhu * sizeof(cplx) > 200 * 1024) {
        fprintf(stderr, "ERROR: lmie_solution_adjoint(): size parameters up to %.0f exceed this build's limit\n",
                2. * LMIEB_PI * *std::max_element(rad, rad + R) / lambda[k_top]);
        return -1;
    }
    const int nrow = ((n1max + 7) & ~7) + 8;              // the kernel loads 8 orders ahead

    const size_t b_tab = pad256((size_t) nrow * nt * 8 * 16);
    const size_t b_esg = pad256(LR * 4 * 8), b_pfp = pad256((size_t) L * G * na * 2 * 8), b_zr = pad256(LR * 3 * 8);
    const size_t fixed = in_bytes + out_bytes + 2 * b_tab + b_esg + b_pfp + b_zr + 3 * 256;
    auto room = [&](long long n) { return fixed + (size_t) n * ADJ_ORDER_BYTES; };
    long long cap = tot;                                  // orders of a pass
    const long long pass_most = std::min(tot, std::max(most, (long long) (ADJ_PASS_BYTES / ADJ_ORDER_BYTES)));
    const bool fail = lmieb_fault_injected("adjoint");
    if (fail || (room(tot) > g_dcap && !(g_dshort && room(pass_most) <= g_dcap))) {
        if (g_dbuf) cudaFree(g_dbuf);
        g_dbuf = nullptr;
        g_dcap = 0;
        cudaError_t e = fail ? cudaErrorMemoryAllocation : cudaMalloc((void **) &g_dbuf, room(tot));
        g_dshort = e == cudaErrorMemoryAllocation;
        if (g_dshort) {
            cudaGetLastError();
            // what is there, but for a tenth
            size_t fr = 0, all = 0;
            LMIEB_CUDA_TRY(cudaMemGetInfo(&fr, &all));
            const size_t use = fail ? 0 : fr / 10 * 9;
            cap = use > fixed ? (long long) ((use - fixed) / ADJ_ORDER_BYTES) : 0;
            cap = std::max(most, std::min(cap, pass_most));
            e = cudaMalloc((void **) &g_dbuf, room(cap));
            if (e == cudaErrorMemoryAllocation && cap > most) {
                cudaGetLastError();
                cap = most;
                e = cudaMalloc((void **) &g_dbuf, room(cap));
            }
        }
        LMIEB_CUDA_TRY(e);
        g_dcap = room(cap);
    } else if (room(tot) > g_dcap) {
        cap = (long long) ((g_dcap - fixed) / ADJ_ORDER_BYTES);
    }
    const size_t b_c = pad256((size_t) cap * sizeof(double4));
    long long *ko = (long long *) (hb + i_ko);
    std::vector<int> pass{0};                             // first wavelengths of the passes
    for (long long k = 0, n = 0; k < L; ++k) {
        if (n + orders[k] > cap) {
            pass.push_back((int) k);
            n = 0;
        }
        ko[k] = n;
        n += orders[k];
    }
    pass.push_back(L);
    char *d = g_dbuf;
    auto dp = [&](size_t at) { return (void *) (d + at); };
    Adj P;
    memset(&P, 0, sizeof(P));
    P.L = L; P.R = R; P.na = na; P.nhu = nhu; P.G = G; P.n_bins = nb;
    P.lam = (const double *) dp(i_lam); P.m = (const cplx *) dp(i_m);
    P.W = (const double *) dp(i_W); P.q = (const double *) dp(i_q); P.rad = (const double *) dp(i_rad);
    P.bstart = (const int *) dp(i_bs);
    P.n1 = (const int *) dp(i_n1); P.n2 = (const int *) dp(i_n2);
    P.ro = (const int *) dp(i_ro); P.ko = (const long long *) dp(i_ko);
    P.mu = (const double *) dp(i_mu); P.nt = nt; P.nrow = nrow;
    P.dw = (const double2 *) dp(i_dw); P.cw = (const double *) dp(i_cw);
    char *o = d + in_bytes;
    P.vals = (double *) o; o += pad256(out_vals);
    P.lw = (double *) o; o += pad256(out_lw);
    P.gout = (double *) o; o += pad256(out_g);
    P.c4 = (double4 *) o; o += b_c;
    P.d4 = (double4 *) o; o += b_c;
    P.b4 = (double4 *) o; o += b_c;
    P.esg = (double *) o; o += b_esg;
    P.pfp = (double *) o; o += b_pfp;
    P.zr = (double *) o; o += b_zr;
    P.tabf = (double2 *) o; o += b_tab;
    P.tabb = (double2 *) o; o += b_tab;

    // ---- run ----
    LMIEB_CUDA_TRY(cudaMemcpyAsync(d, g_hbuf, in_bytes, cudaMemcpyHostToDevice, s));
    for (size_t i = 0; i + 1 < pass.size(); ++i) {
        // the pass' wavelengths: their part of everything but the orders' columns and the tables
        const int k0 = pass[i], n = pass[i + 1] - k0;
        const size_t r0 = (size_t) k0 * R;
        Adj Q = P;
        Q.L = n;
        Q.lam += k0; Q.m += k0; Q.ko += k0;
        Q.n1 += r0; Q.n2 += r0; Q.ro += r0;
        Q.dw += (size_t) k0 * 16 * nt; Q.cw += (size_t) k0 * 3;
        Q.esg += r0 * 4; Q.zr += r0 * 3; Q.pfp += (size_t) k0 * G * na * 2;
        Q.lw += (size_t) k0 * 8; Q.vals += (size_t) k0 * (3 + 2 * na);
        k_adj_coef<<<(unsigned) n * ((R + 63) / 64), 64, 0, s>>>(Q);
        LMIEB_CUDA_TRY(cudaGetLastError());
        if (i == 0) {
            k_adj_table<<<1, 8 * nt, 0, s>>>(Q);
            LMIEB_CUDA_TRY(cudaGetLastError());
        }
        if (launch_angles(Q, s)) return -1;
        k_adj_lambda<<<n, ADJ_T, 0, s>>>(Q);
        LMIEB_CUDA_TRY(cudaGetLastError());
        k_adj_m<<<ceil_div(8 * (size_t) n * R, 256), 256, 0, s>>>(Q);
        LMIEB_CUDA_TRY(cudaGetLastError());
    }
    k_adj_final<<<L + nb, ADJ_T, 0, s>>>(P);
    LMIEB_CUDA_TRY(cudaGetLastError());
    char *ho = g_hbuf + in_bytes;
    LMIEB_CUDA_TRY(cudaMemcpyAsync(ho, d + in_bytes, out_bytes, cudaMemcpyDeviceToHost, s));
    LMIEB_CUDA_TRY(cudaStreamSynchronize(s));
    const double *hv = (const double *) ho;
    const double *hl = (const double *) (ho + pad256(out_vals));
    const double *hg = (const double *) (ho + pad256(out_vals) + pad256(out_lw));
    double sum = 0.;
    for (int k = 0; k < L; ++k) sum += hl[(size_t) k * 8 + 5];
    *loss = sum;
    if (grad_mr) memcpy(grad_mr, hg, (size_t) L * 8);
    if (grad_mi) memcpy(grad_mi, hg + L, (size_t) L * 8);
    if (grad_weight) memcpy(grad_weight, hg + 2 * L, (size_t) nb * 8);
    if (values) memcpy(values, hv, out_vals);
    return 0;
}
