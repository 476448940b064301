// k_mie.cu -- K1 in a tangent basis: the Mie recurrences, coefficients and
// per-radius sums of every radius with their derivatives in at most two
// directions, whatever the number of index1 derivatives.
//
// Every index1 derivative p of a sphere's coefficients is
//     da/dp = m_p da/dm + x_p da/dx,
// m_p the (complex) derivative of the refractive index, the same for all radii
// of a case, x_p that of the size parameter; a and b are analytic in m, so one
// complex column da/dm serves the derivatives w.r.t. mr and mi (dm/dmi = -i)
// and any combination of them.  K1 and the angular stages carry the columns
//   m   da/dm, when some derivative moves the refractive index;
//   x   da/dx, when some derivative moves the size parameters; with a single
//       index1 derivative that moves both, its own direction instead of both;
// and the derivatives are put together from their sums (k_reduce_scalars, the
// angular kernels).  A column costs as much as one derivative did, so the
// usual pair (mr, mi) costs half, and da/dm needs no derivatives of psi and
// chi:
//     da/dm = i W c' / den^2,  c' = d(D/m)/dm,  den = (D/m + n/x) zeta_n - zeta_{n-1},
//     W = psi_{n-1} chi_n - psi_n chi_{n-1}
// (the quotient rule's difference of two products is this), and likewise for b
// with c' = d(m D)/dm.  W is formed from the psi and chi at hand: it is 1, but
// for the last orders, where psi still feels its start from zero at n1, not to
// 1e-7, and the derivative of these a and b is wanted.  The recurrences and the
// formulas of an order are in mie_radius.cuh.
//
// Reference: src/lmie_core.c:298-370 (psi ratio, psi, chi), 386-440 (D), 455-510
// (a, b and tangents), 515-590 (cross-section and asymmetry sums per radius).
#include <cstdio>

#include "kernels.h"
#include "mie_radius.cuh"
#include "oz_layout.cuh"
#include "tc_layout.cuh"

namespace {

// m[c] = max(m[c], biased exponent of component c + ek) over the normal
// values among (Re cs, Im cs, Re cd, Im cd)
__device__ __forceinline__ void track(int (&m)[4], cplx cs, cplx cd, int ek) {
    const double v[4] = {cs.re, cs.im, cd.re, cd.im};
#pragma unroll
    for (int c = 0; c < 4; ++c) {
        const int ex = (__double2hiint(v[c]) >> 20) & 0x7FF;
        m[c] = max(m[c], ex ? ex + ek : 0);
    }
}

// Split-precision operand of K1's radius.  The 8 floats of order j and column
// slot cc of CC -- e = 0..7: S hi re, S hi im, S lo re, S lo im, D' hi re, D' hi
// im, D' lo re, D' lo im, with D' = s_j (a - b) fv4 -- are staged in the
// thread's slot u = (j - 1) % 4 of shared memory, tcbuf[((u * CC + cc) * 8 + e) *
// T + thread] (a warp's accesses hit consecutive banks); every 4 orders (and
// after the last) they go out as 16-byte pieces of the K-major core-matrix
// layout of tc_layout.cuh instead of 4-byte stores per order.
__device__ __forceinline__ void tc_stage(float *tcbuf, int CC, int j, int cc, cplx cs, cplx cd) {
    const int T = blockDim.x, u = (j - 1) & 3;
    const double sg = (j & 1) ? 1. : -1.;             // s_j of D'
    float *p = tcbuf + (size_t) ((u * CC + cc) * 8) * T + threadIdx.x;
    float h, l;
    tc_split(cs.re, h, l); p[0] = h; p[2 * T] = l;
    tc_split(cs.im, h, l); p[1 * T] = h; p[3 * T] = l;
    tc_split(sg * cd.re, h, l); p[4 * T] = h; p[6 * T] = l;
    tc_split(sg * cd.im, h, l); p[5 * T] = h; p[7 * T] = l;
}

// Writes the group of 4 orders that holds order j (orders after j in it are
// zero) of the CC columns; with gnk the radius' last one, and zeros after it
// up to the end of its group's gnk chunks (the operand buffer is not cleared
// between solves).
__device__ __forceinline__ void tc_flush(const float *tcbuf, float *__restrict__ rbase, int CC, int j, int pos,
                                         int gnk) {
    const int T = blockDim.x, last = (j - 1) & 3, k0 = (j - 1) - last;
    constexpr int P = TC_BPART / 4;
    const float4 z = make_float4(0.f, 0.f, 0.f, 0.f);
    for (int cc = 0; cc < CC; ++cc) {
        const int n = (pos * CC + cc) * 2;
        {
            const int kc = k0 / TC_KC, kk = k0 - kc * TC_KC;
            float *base = rbase + (size_t) kc * (TC_BSTAGE / 4);
            const int i0 = tc_idx(n, kk, TC_NP), d0 = tc_idx(TC_NHALF + n, kk, TC_NP);
            float v[8][4];
#pragma unroll
            for (int e = 0; e < 8; ++e)
#pragma unroll
                for (int u = 0; u < 4; ++u)
                    v[e][u] = u <= last ? tcbuf[(size_t) ((u * CC + cc) * 8 + e) * T + threadIdx.x] : 0.f;
            *(float4 *) (base + i0) = make_float4(v[0][0], v[0][1], v[0][2], v[0][3]);
            *(float4 *) (base + i0 + 4) = make_float4(v[1][0], v[1][1], v[1][2], v[1][3]);
            *(float4 *) (base + P + i0) = make_float4(v[2][0], v[2][1], v[2][2], v[2][3]);
            *(float4 *) (base + P + i0 + 4) = make_float4(v[3][0], v[3][1], v[3][2], v[3][3]);
            *(float4 *) (base + d0) = make_float4(v[4][0], v[4][1], v[4][2], v[4][3]);
            *(float4 *) (base + d0 + 4) = make_float4(v[5][0], v[5][1], v[5][2], v[5][3]);
            *(float4 *) (base + P + d0) = make_float4(v[6][0], v[6][1], v[6][2], v[6][3]);
            *(float4 *) (base + P + d0 + 4) = make_float4(v[7][0], v[7][1], v[7][2], v[7][3]);
        }
        for (int k = k0 + 4; k < gnk * TC_KC; k += 4) {
            const int kc = k / TC_KC, kk = k - kc * TC_KC;
            float *base = rbase + (size_t) kc * (TC_BSTAGE / 4);
            const int i0 = tc_idx(n, kk, TC_NP), d0 = tc_idx(TC_NHALF + n, kk, TC_NP);
            *(float4 *) (base + i0) = z;
            *(float4 *) (base + i0 + 4) = z;
            *(float4 *) (base + P + i0) = z;
            *(float4 *) (base + P + i0 + 4) = z;
            *(float4 *) (base + d0) = z;
            *(float4 *) (base + d0 + 4) = z;
            *(float4 *) (base + P + d0) = z;
            *(float4 *) (base + P + d0 + 4) = z;
        }
    }
}

// Where an order's coefficients go: the columns fv4 (a +- b) of coef, with the
// largest exponents of each (the column exponents of the fixed-point B operand)
// in mxe when `re` is set.
template <bool HM, bool HX>
__device__ __forceinline__ void put_columns(const MieAB &q, double f4, int j, double4 *cf, size_t tot, size_t at,
                                            bool re, int (&mxe)[1 + HM + HX][4]) {
    const int ek = oz_ek(j);
    auto put = [&](int col, cplx va, cplx vb) {
        const cplx cs = (va + vb) * f4, cd = (va - vb) * f4;
        cf[(size_t) col * tot + at + j - 1] = make_double4(cs.re, cs.im, cd.re, cd.im);
        if (re) track(mxe[col], cs, cd, ek);
    };
    put(0, q.a, q.b);
    if (HM) put(1 * HM, q.am, q.bm);
    if (HX) put((1 + HM) * HX, q.ax, q.bx);
}

// The columns of a split-precision case's order j in its operand (see tc_stage):
// put(col, a + b, a - b), times fv4, of the value and the index1 derivatives.
template <bool HM, bool HX, class Put>
__device__ __forceinline__ void tc_columns(const DevBatch &B, const DevCase &C, int r, const MieAB &q, double f4,
                                           Put &&put) {
    put(0, (q.a + q.b) * f4, (q.a - q.b) * f4);
    for (int k = 0; k < B.nd1; ++k) {
        cplx va = mk(0., 0.), vb = va;
        if (HM) {
            const cplx ml = B.m_l[C.ml_off + B.idx1[k]];
            va = ml * q.am;
            vb = ml * q.bm;
        }
        if (HX) {
            const double xc = B.x_own ? 1. : B.xl[(size_t) k * B.R + r];
            va = cfma(q.ax, xc, va);
            vb = cfma(q.bx, xc, vb);
        }
        put(1 + k, (va + vb) * f4, (va - vb) * f4);
    }
}

// order j of column cc of the radius at position pos of its group, CC columns
// in all (four lanes of consecutive orders write 16 bytes of each value)
__device__ __forceinline__ void tc_put(float *__restrict__ rbase, int CC, int pos, int j, int cc, cplx cs, cplx cd) {
    constexpr int P = TC_BPART / 4;
    const int kc = (j - 1) / TC_KC, kk = (j - 1) - kc * TC_KC, n = (pos * CC + cc) * 2;
    float *base = rbase + (size_t) kc * (TC_BSTAGE / 4);
    const int i0 = tc_idx(n, kk, TC_NP), d0 = tc_idx(TC_NHALF + n, kk, TC_NP);
    const double sg = (j & 1) ? 1. : -1.;             // s_j of D'
    float h, l;
    tc_split(cs.re, h, l); base[i0] = h; base[P + i0] = l;
    tc_split(cs.im, h, l); base[i0 + 4] = h; base[P + i0 + 4] = l;
    tc_split(sg * cd.re, h, l); base[d0] = h; base[P + d0] = l;
    tc_split(sg * cd.im, h, l); base[d0 + 4] = h; base[P + d0 + 4] = l;
}

// the radius of rank t in the launch order: cases in the order k1ord, each from
// its largest radius down
__device__ __forceinline__ int radius_of(const DevBatch &B, long long t) {
    const int kc = find_case(B.k1pre, B.ncase, t);
    const DevCase &C = B.cs[B.k1ord[kc]];
    return C.r0 + C.nr - 1 - (int) (t - B.k1pre[kc]);
}

// the x column's direction: x alone, or the single derivative's own
template <bool HX>
__device__ __forceinline__ MieRadius<HX> radius_setup(const DevBatch &B, const DevCase &C, int r) {
    MieRadius<HX> c;
    c.set_m(C.m, C.minv, HX && B.x_own ? B.m_l[C.ml_off + B.idx1[0]] : mk(0., 0.));
    c.set_x(B.x[r], HX && B.x_own ? B.xl[r] : 1.);
    return c;
}

// ---------------------------------------------------------------------------
// One thread per radius.  The downward recurrences keep only their values at
// the top of every block of MIE_B orders (checkpoints in ck); the ascending
// pass replays each block from its checkpoint (the same operations, so the same
// values), forms D_n and the orders' coefficients and tangents, writes the
// coefficient columns and sums the per-radius cross sections in order.  HM, HX:
// with the m, the x column; TC: the split-precision cases' derivatives go to the
// tensor-core operand instead; DZ: some radii's dD/dz is the tangent of D's
// recurrence; RATIO: psi of fewer than MIE_P_MIN orders.  (3000 radii up to x =
// 5000, values and a derivative by lambda 5.0 ms, by mr with DZ 5.3; with both
// decided order by order in one body 5.8 and 5.3.)  Bound by FP64 latency (a
// thread's chain) where few radii are long, by the FP64 pipe where many fill the SMs.
// Per-radius sums rs[(col 5 + q) R + r], q: se, ss, Re sb, Im sb, sg, of the
// columns 0 value, B.rs_m d/dmr, B.rs_m + 1 d/dmi (both from the m column),
// B.rs_x the x column.
// ---------------------------------------------------------------------------
template <bool HM, bool HX, bool TC, bool DZ, bool RATIO>
__device__ __forceinline__ void mie_thread(const DevBatch &B, const DevCase &C, int r, int n1, int n2,
                                           double *__restrict__ ck, double *__restrict__ coef,
                                           float *__restrict__ bop, double *__restrict__ rs) {
    constexpr int CW = k1_ck_width(HX, DZ);          // D (2), u (2), exponent, u's tangent (2), D's (2)
    const int R = B.R;
    const MieRadius<HX> c = radius_setup<HX>(B, C, r);
    const bool zr = DZ && mie_dz_chain(C.m, c.x);    // D's tangent
    const int nb = n1 / MIE_B + 1;
    double *ckr = ck + (size_t) B.ckoff[r] * CW;     // nb blocks of CW doubles
    const double *fv4 = B.fv + 3 * (B.n1max + 2), *fv3 = fv4 - (B.n1max + 2);

    auto d_step = [&](MieD &p, int n) {
        if (DZ && zr) p.step<true>(n, c.zinv, c.zinv2);
        else p.step(n, c.zinv);
    };
    // (the ratio of order n - 1; that of order 0 is not used)
    auto u_step = [&](MieU<HX> &q, int n) {
        if (RATIO) {                                  // q.cur, q.xcur: psi's ratio and its tangent
            mie_ratio(n - 1, c.xinv, q.cur, q.xcur);
        } else {
            q.step(n, c.xinv);
        }
    };
    // ---- downward: D from n2, u from n1 (n2 > n1 + MIE_B), block by block ----
    double u0, ux0 = 0.;
    int eu = 0;
    {
        MieD p;
        p.start();                                   // D_{n2} = 0, n2 > n1 + MIE_B
        for (int n = n2 - 1; n >= nb * MIE_B; --n) d_step(p, n);
        MieU<HX> q;
        q.start();
        for (int b = nb - 1; b >= 0; --b) {
            double *w = ckr + (size_t) b * CW;
            w[0] = p.cur.re; w[1] = p.cur.im; w[2] = q.hi; w[3] = q.cur; w[4] = (double) eu;
            if (HX) { w[5] = q.xhi; w[HX ? 6 : 0] = q.xcur; }
            if (DZ) { w[CW - 2] = p.dz.re; w[CW - 1] = p.dz.im; }
#pragma unroll
            for (int i = MIE_B - 1; i >= 0; --i) {
                const int k = b * MIE_B + i;
                if (b > 0 || i > 0) d_step(p, k);
                if (k <= n1 && (b > 0 || i > 0)) u_step(q, k);
            }
            if (b > 0 && !RATIO) eu += q.rescale();
        }
        u0 = q.cur;
        if (HX) ux0 = q.xcur;
    }

    // ---- ascending pass ----
    double sinx, cosx;
    sincos(c.x, &sinx, &cosx);
    const double spsi = sinx / u0, spsix = HX ? fma(-spsi, ux0, cosx) / u0 : 0.;
    double chi_p = cosx, chi_c = fma(c.xinv, cosx, sinx);       // chi_0, chi_1
    double psi_p = spsi * u0, px = HX ? fma(spsix, u0, spsi * ux0) : 0.;   // px: d psi / dx
    if (RATIO) {
        psi_p = sinx;
        px = cosx;
    }
    double psix_p = c.xl * px;
    MieSums<HM, HX> sums;
    sums.zero();
    MieAB prev;
    prev.a = prev.b = prev.am = prev.bm = prev.ax = prev.bx = mk(0., 0.);
    const size_t tot = (size_t) B.tot, off = (size_t) B.off[r];
    // split precision: the radii of tensor-core cases write the B operand
    const int tcode = TC ? B.tc_pos[r] : -1;
    const bool to_tc = TC && tcode >= 0;
    const int tpos = tcode & 255, tgnk = tcode >> 8;   // position in the group, the group's chunks
    float *const tcb = to_tc ? bop + B.tc_roff[r] : nullptr;
    const int n_tc = 1 + B.nd1;
    extern __shared__ float tcbuf[];                  // [4][1 + nd1][8][blockDim.x] with TC
    int *const re = B.oz_radexp;
    int mxe[1 + HM + HX][4];
#pragma unroll
    for (int q = 0; q < 4 * (1 + HM + HX); ++q) mxe[q / 4][q % 4] = 0;

    for (int b = 0; b < nb; ++b) {
        const double *w = ckr + (size_t) b * CW;
        cplx D[MIE_B], Dz[MIE_B];
        double ub[MIE_B], uxb[HX ? MIE_B : 1];
        const double su = mb_pow2((int) w[4] - eu);
        {
            MieD p;
            p.cur = mk(w[0], w[1]);
            p.dz = DZ ? mk(w[CW - 2], w[CW - 1]) : mk(0., 0.);
            MieU<HX> q;
            q.hi = w[2];
            q.cur = w[3];
            if (HX) { q.xhi = w[5]; q.xcur = w[HX ? 6 : 0]; }
#pragma unroll
            for (int i = MIE_B - 1; i >= 0; --i) {
                const int k = b * MIE_B + i;
                ub[i] = q.cur;
                if (HX) uxb[HX ? i : 0] = q.xcur;
                if (k > 0) {
                    d_step(p, k);
                    if (k <= n1) {
                        D[i] = p.cur;
                        if (HM || HX) {
                            Dz[i] = mie_dz(c, k, p.cur);
                            if (DZ && zr) Dz[i] = mie_dz_add(Dz[i], mie_dz_corr(c, k, p.cur, p.dz));
                        }
                        u_step(q, k);
                    }
                }
            }
        }
#pragma unroll
        for (int i = 0; i < MIE_B; ++i) {
            const int j = b * MIE_B + i;
            if (j < 1 || j > n1) continue;
            const double psi = RATIO ? ub[i] * psi_p : spsi * ub[i] * su;
            if (HX) px = RATIO ? fma(uxb[HX ? i : 0], psi_p, ub[i] * px) : fma(spsix, ub[i], spsi * uxb[HX ? i : 0]) * su;
            const double psix = c.xl * px;
            const MieAB q = mie_ab<HM, HX>(c, j, D[i], Dz[i], psi, psi_p, chi_c, chi_p, psix, psix_p);
            sums.add(j, q, prev, fv3[j - 1], fv4[j - 1]);
            const double f4 = fv4[j];
            if (to_tc) {
                tc_columns<HM, HX>(B, C, r, q, f4, [&](int cc, cplx cs, cplx cd) { tc_stage(tcbuf, n_tc, j, cc, cs, cd); });
                if (((j - 1) & 3) == 3 || j == n1) tc_flush(tcbuf, tcb, n_tc, j, tpos, j == n1 ? tgnk : 0);
            } else {
                put_columns<HM, HX>(q, f4, j, (double4 *) coef, tot, off, re != nullptr, mxe);
            }
            const double chi_n = fma((2. * j + 1.) * c.xinv, chi_c, -chi_p);
            chi_p = chi_c;
            chi_c = chi_n;
            psi_p = psi;
            psix_p = psix;
            prev = q;
        }
    }
    sums.close();
#pragma unroll
    for (int q = 0; q < MieSums<HM, HX>::N; ++q) rs[(size_t) q * R + r] = sums.v[q];
    if (re) {
#pragma unroll
        for (int k = 0; k < 1 + HM + HX; ++k)
            *(int4 *) (re + ((size_t) k * R + r) * 4) = make_int4(mxe[k][0], mxe[k][1], mxe[k][2], mxe[k][3]);
    }
}

template <bool HM, bool HX, bool TC, bool DZ>
__global__ void __launch_bounds__(64) k_mie(DevBatch B, double *__restrict__ ck, double *__restrict__ coef,
                                            float *__restrict__ bop, double *__restrict__ rs) {
    const long long t = (long long) blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= B.R) return;
    const int r = radius_of(B, t), n1 = B.n1r[r], n2 = B.n2r[r];
    const DevCase &C = B.cs[B.rcase[r]];
    if (HX && n1 < MIE_P_MIN) mie_thread<HM, HX, TC, DZ, HX>(B, C, r, n1, n2, ck, coef, bop, rs);
    else mie_thread<HM, HX, TC, DZ, false>(B, C, r, n1, n2, ck, coef, bop, rs);
}

// ---------------------------------------------------------------------------
// K1 by blocks: block i's B.k1_blk[i].y radii are of case .z, from radius .x
// down.  Bound by instruction issue (half of it taken, a third of the FP64
// pipe's) where the blocks are many, by the chains' latency where they are few.
// 107 thousand radii, 777 cases, values only: 303 us (a thread per radius: 789);
// 109 thousand, 766 cases, with the m column: 766 us (915), 4096 cases 3.43 ms,
// 3.87 with D's tangent for the sixth of the orders that takes it; the cloud
// droplet's 2000 radii up to x = 436: 69 us (a thread per radius 380).
// ---------------------------------------------------------------------------
template <bool HM, bool HX, bool TC, int TEAM>
__global__ void __launch_bounds__(MIE_BLOCK_T, HX ? 2 : 4) k_mie_block(DevBatch B, double *__restrict__ coef,
                                                                       float *__restrict__ bop,
                                                                       double *__restrict__ rs) {
    extern __shared__ __align__(16) unsigned char smem[];
    constexpr int NC = 1 + HM + HX;
    const int4 blk = B.k1_blk[blockIdx.x];
    const DevCase &C = B.cs[blk.z];
    const int R = B.R;
    const double *fv4 = B.fv + 3 * (B.n1max + 2), *fv3 = fv4 - (B.n1max + 2);
    const size_t tot = (size_t) B.tot;
    const bool re = B.oz_radexp != nullptr;
    int mxe[NC][4];
#pragma unroll
    for (int q = 0; q < 4 * NC; ++q) mxe[q / 4][q % 4] = 0;
    int r = 0, tcode = -1;                            // the team's radius, its operand position, its first order
    size_t off = 0;
    float *tcb = nullptr;
    constexpr int TS = TEAM == 32 ? 32 : MIE_BLOCK_T;
    const int tl = threadIdx.x % TS;
    mie_block<HM, HX, TEAM>(
        smem, (HM || HX) && blk.w ? B.k1_rows_dz : B.k1_rows, (HM || HX) && blk.w, blk.y,
        [&](MieRadius<HX> &c) {
            c.set_m(C.m, C.minv, HX && B.x_own ? B.m_l[C.ml_off + B.idx1[0]] : mk(0., 0.));
        },
        [&](int g, MieRadius<HX> &c, int &n1, int &n2) {
            const int q = blk.x - g;
            c.set_x(B.x[q], HX && B.x_own ? B.xl[q] : 1.);
            n1 = B.n1r[q];
            n2 = B.n2r[q];
        },
        [&](int n, double &f3, double &f4) {
            f3 = fv3[n - 1];
            f4 = fv4[n - 1];
        },
        [&](int g) {
            r = blk.x - g;
            off = (size_t) B.off[r];
            if (TC) {
                tcode = B.tc_pos[r];
                tcb = bop + B.tc_roff[r];
            }
        },
        [&](int j, const MieAB &q) {
            if (TC && tcode >= 0)
                tc_columns<HM, HX>(B, C, r, q, fv4[j], [&](int cc, cplx cs, cplx cd) {
                    tc_put(tcb, 1 + B.nd1, tcode & 255, j, cc, cs, cd);
                });
            else put_columns<HM, HX>(q, fv4[j], j, (double4 *) coef, tot, off, re, mxe);
        },
        [&](const MieSums<HM, HX> &sums) {
            if ((TEAM == 32 ? threadIdx.x & 31 : threadIdx.x) == 0)
#pragma unroll
                for (int q = 0; q < MieSums<HM, HX>::N; ++q) rs[(size_t) q * R + r] = sums.v[q];
            if (TC && tcode >= 0)
                // zeros up to the end of the group's chunks (the operand buffer is not cleared between solves)
                for (int j = B.n1r[r] + 1 + tl; j <= (tcode >> 8) * TC_KC; j += TS)
                    for (int cc = 0; cc <= B.nd1; ++cc)
                        tc_put(tcb, 1 + B.nd1, tcode & 255, j, cc, mk(0., 0.), mk(0., 0.));
            if (re) {
                // the largest exponents of the team
                __shared__ int mx[MIE_BLOCK_T / 32][4 * NC];
#pragma unroll
                for (int q = 0; q < 4 * NC; ++q) {
                    const int v = __reduce_max_sync(0xffffffffu, mxe[q / 4][q % 4]);
                    mxe[q / 4][q % 4] = 0;
                    if ((threadIdx.x & 31) == 0) mx[threadIdx.x >> 5][q] = v;
                }
                if (TEAM == 32) __syncwarp();
                else __syncthreads();
                const int l = TEAM == 32 ? threadIdx.x & 31 : threadIdx.x;
                if (l < 4 * NC) {
                    int v = 0;
                    if (TEAM == 32) v = mx[threadIdx.x >> 5][l];
                    else
                        for (int w = 0; w < MIE_BLOCK_T / 32; ++w) v = max(v, mx[w][l]);
                    B.oz_radexp[((size_t) (l / 4) * R + r) * 4 + l % 4] = v;
                }
                if (TEAM == 32) __syncwarp();
            }
        });
}

template <bool HM, bool HX, bool TC, int TEAM>
int launch_block(cudaStream_t s, const DevBatch &B, double *coef, float *bop, double *rs) {
    static bool attr = false;
    if (!attr) {
        LMIEB_CUDA_TRY(cudaFuncSetAttribute(k_mie_block<HM, HX, TC, TEAM>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                            MIE_BLOCK_SMEM));
        attr = true;
    }
    k_mie_block<HM, HX, TC, TEAM><<<B.k1_nblk, MIE_BLOCK_T, B.k1_smem, s>>>(B, coef, bop, rs);
    LMIEB_CUDA_TRY(cudaGetLastError());
    return 0;
}

template <bool HM, bool HX, bool DZ>
int launch_threads(cudaStream_t s, const DevBatch &B, double *ck, double *coef, float *bop, double *rs) {
    if (bop)
        k_mie<HM, HX, true, DZ>
            <<<ceil_div(B.R, 64), 64, 4 * 8 * (1 + B.nd1) * 64 * sizeof(float), s>>>(B, ck, coef, bop, rs);
    else
        k_mie<HM, HX, false, DZ><<<ceil_div(B.R, 64), 64, 0, s>>>(B, ck, coef, nullptr, rs);
    LMIEB_CUDA_TRY(cudaGetLastError());
    return 0;
}

template <bool HM, bool HX>
int launch(cudaStream_t s, const DevBatch &B, double *ck, double *coef, float *bop, double *rs) {
    // the orders of a radius by the whole block where it has one, or where they
    // are many: means of 700 and 250 orders took 520 and 125 us that way, 667 and
    // 112 us with a warp per radius
    if (B.k1_nblk && (B.k1_nblk == B.R || B.tot >= 400LL * B.R))
        return bop ? launch_block<HM, HX, true, MIE_BLOCK_T>(s, B, coef, bop, rs)
                   : launch_block<HM, HX, false, MIE_BLOCK_T>(s, B, coef, bop, rs);
    if (B.k1_nblk)
        return bop ? launch_block<HM, HX, true, 32>(s, B, coef, bop, rs)
                   : launch_block<HM, HX, false, 32>(s, B, coef, bop, rs);
    if (HM || HX)
        if (B.k1_dz) return launch_threads<HM, HX, HM || HX>(s, B, ck, coef, bop, rs);
    return launch_threads<HM, HX, false>(s, B, ck, coef, bop, rs);
}

}  // namespace

int launch_coef(cudaStream_t s, const DevBatch &B, double *ck, double *coef, float *bop, double *rs) {
    const bool hm = B.t_m > 0, hx = B.t_x > 0;
    if (hm) return hx ? launch<true, true>(s, B, ck, coef, bop, rs) : launch<true, false>(s, B, ck, coef, bop, rs);
    return hx ? launch<false, true>(s, B, ck, coef, bop, rs) : launch<false, false>(s, B, ck, coef, bop, rs);
}
