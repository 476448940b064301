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
// for the last orders, where the psi ratio still feels its start from zero at
// n1, not to 1e-7, and the derivative of these a and b is wanted.
//
// Reference: src/lmie_core.c:298-370 (psi ratio, psi, chi), 386-440 (D), 455-510
// (a, b and tangents), 515-590 (cross-section and asymmetry sums per radius).
#include <cstdio>

#include "kernels.h"
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

// conj(a) b
__device__ __forceinline__ cplx cmul(cplx a, cplx b) {
    return mk(a.re * b.re + a.im * b.im, a.re * b.im - a.im * b.re);
}

// ---------------------------------------------------------------------------
// One thread per radius.  The downward recurrences -- D_n(mx) from n2 and the
// psi ratio from n1, with their tangents -- keep only their values at the top
// of every block of K1_B orders (checkpoints in ck); the ascending pass replays
// each block from its checkpoint into local arrays (the same operations, so
// the same values), runs psi and chi upward, forms a_n, b_n and their tangents,
// writes the coefficient columns fv4 (a +- b) and sums the per-radius cross
// sections in order.  HM, HX: with the m, the x column; TC: the split-precision
// cases' derivatives go to the tensor-core operand instead.  Per-radius sums
// rs[(col 5 + q) R + r], q: se, ss, Re sb, Im sb, sg, of the columns 0 value,
// B.rs_m d/dmr, B.rs_m + 1 d/dmi (both from the m column), B.rs_x the x column.
// ---------------------------------------------------------------------------
template <bool HM, bool HX, bool TC>
__global__ void __launch_bounds__(64) k_mie(DevBatch B, double *__restrict__ ck, double *__restrict__ coef,
                                            float *__restrict__ bop, double *__restrict__ rs) {
    constexpr int CW = k1_ck_width(HM, HX);       // D (2), D_m (2), ratio (1), D_x (2), ratio_x (1)
    constexpr int QX = HM ? 5 : 3;
    // thread t takes the radius of rank t in the launch order: cases in the
    // order k1ord, each from its largest radius down
    const long long t = (long long) blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= B.R) return;
    const int kc = find_case(B.k1pre, B.ncase, t);
    const int r = [&] {
        const DevCase &Ck = B.cs[B.k1ord[kc]];
        return Ck.r0 + Ck.nr - 1 - (int) (t - B.k1pre[kc]);
    }();
    const int R = B.R;
    const DevCase &C = B.cs[B.rcase[r]];
    const int n1 = B.n1r[r], n2 = B.n2r[r];
    const double x = B.x[r];
    const double xinv = 1. / x;
    const cplx m = C.m, minv = C.minv;
    const cplx z = mk(m.re * x, m.im * x);
    const cplx zinv = cinv(z);
    const int nb = (n1 + K1_B - 1) / K1_B;
    double *ckr = ck + (size_t) B.ckoff[r] * CW;     // nb blocks of CW doubles
    const double *fv1 = B.fv, *fv3 = B.fv + 2 * (B.n1max + 2), *fv4 = B.fv + 3 * (B.n1max + 2);
    // the x column's direction: x alone, or the single derivative's own
    double xl = 1.;
    cplx ml = mk(0., 0.), zl = mk(0., 0.);
    if (HX) {
        if (B.x_own) {
            xl = B.xl[r];
            ml = B.m_l[C.ml_off + B.idx1[0]];
        }
        zl = ml * x + m * xl;
    }

    struct Chain {
        cplx D, Dm, Dx;
        double rn, rx;
    };
    auto d_step = [&](Chain &c, int j) {
        const cplx c1 = (j + 1.) * zinv;
        const cplx ic2 = cinv(c.D + c1);
        c.D = c1 - ic2;
        if (HM || HX) {
            const cplx c3 = -c1 * zinv;
            const cplx ic4 = ic2 * ic2;
            if (HM) {
                const cplx c5 = c3 * x;              // z_m = x
                c.Dm = c5 + (c.Dm + c5) * ic4;
            }
            if (HX) {
                const cplx c5 = c3 * zl;
                c.Dx = c5 + (c.Dx + c5) * ic4;
            }
        }
    };
    auto r_step = [&](Chain &c, int j) {
        const double a1 = (2. * j + 1.) * xinv;
        const double rnew = 1. / (a1 - c.rn);
        if (HX) {
            const double a2 = -a1 * xinv, a3 = rnew * rnew;
            c.rx = -(a2 * xl - c.rx) * a3;
        }
        c.rn = rnew;
    };
    auto put_d = [&](const Chain &c, double *q) {
        q[0] = c.D.re;
        q[1] = c.D.im;
        if (HM) {
            q[3] = c.Dm.re;
            q[4] = c.Dm.im;
        }
        if (HX) {
            q[QX] = c.Dx.re;
            q[QX + 1] = c.Dx.im;
        }
    };
    auto put_r = [&](const Chain &c, double *q) {
        q[2] = c.rn;
        if (HX) q[QX + 2] = c.rx;
    };
    // ---- downward sweeps: checkpoints only; the two chains (D_n from n2, the
    // psi ratio from n1 < n2) advance in one loop below n1 ----
    {
        Chain c;
        c.D = c.Dm = c.Dx = mk(0., 0.);
        c.rn = c.rx = 0.;
        for (int b = 0; b < nb; ++b) {
            double *q = ckr + (size_t) b * CW;
            if (b * K1_B + K1_B >= n2) put_d(c, q);
            if (b * K1_B + K1_B >= n1) put_r(c, q);
        }
        auto d_down = [&](int j) {
            d_step(c, j);
            if (j % K1_B == 0 && j / K1_B - 1 < nb) put_d(c, ckr + (size_t) (j / K1_B - 1) * CW);
        };
        for (int j = n2 - 1; j >= n1; --j) d_down(j);
        for (int j = n1 - 1; j >= 1; --j) {
            d_down(j);
            r_step(c, j);
            if (j % K1_B == 0 && j / K1_B - 1 < nb) put_r(c, ckr + (size_t) (j / K1_B - 1) * CW);
        }
    }

    // ---- ascending pass ----
    double sinx, cosx;
    sincos(x, &sinx, &cosx);
    double psi_p = sinx, chi_p = cosx, chi_c = xinv * cosx + sinx;     // psi_0, chi_0, chi_1
    double psix_p = 0., chix_p = 0., chix_c = 0.;
    if (HX) {
        psix_p = xl * cosx;
        chix_p = xl * -sinx;
        chix_c = (-xinv * xinv) * xl * cosx + xinv * chix_p + xl * cosx;
    }
    double acc[5] = {0., 0., 0., 0., 0.};
    double accr[5] = {0., 0., 0., 0., 0.}, acci[5] = {0., 0., 0., 0., 0.};   // d/dmr, d/dmi
    double accx[5] = {0., 0., 0., 0., 0.};
    cplx ap = mk(0., 0.), bp = mk(0., 0.), amp = ap, bmp = ap, axp = ap, bxp = ap;
    const cplx minv2 = minv * minv;
    const size_t tot = (size_t) B.tot, off = (size_t) B.off[r];
    double4 *cf = (double4 *) coef;
    // split precision: the radii of tensor-core cases write the B operand
    const int tcode = TC ? B.tc_pos[r] : -1;
    const bool to_tc = TC && tcode >= 0;
    const int tpos = tcode & 255, tgnk = tcode >> 8;   // position in the group, the group's chunks
    float *const tcb = to_tc ? bop + B.tc_roff[r] : nullptr;
    const int n_tc = 1 + B.nd1;
    extern __shared__ float tcbuf[];                  // [4][1 + nd1][8][blockDim.x] with TC
    // the largest (biased exponent + e_k) of each column and component, the
    // column exponents of the fixed-point B operand
    int *const re = B.oz_radexp;
    int mxe[1 + HM + HX][4];
#pragma unroll
    for (int q = 0; q < 4 * (1 + HM + HX); ++q) mxe[q / 4][q % 4] = 0;

    cplx Dloc[K1_B], Dmloc[HM ? K1_B : 1], Dxloc[HX ? K1_B : 1];
    double rloc[K1_B], rxloc[HX ? K1_B : 1];
    for (int b = 0; b < nb; ++b) {
        const int lo = b * K1_B + 1, hi = min(b * K1_B + K1_B, n1);
        const double *q = ckr + (size_t) b * CW;
        // replay D from the block's top (top <= n2) and the psi ratio from hi
        // (top >= hi) down to lo: one loop below hi, as in the downward sweeps
        {
            const int top = min(b * K1_B + K1_B, n2);
            Chain c;
            c.D = mk(q[0], q[1]);
            c.rn = q[2];
            c.Dm = HM ? mk(q[3], q[4]) : mk(0., 0.);
            c.Dx = HX ? mk(q[QX], q[QX + 1]) : mk(0., 0.);
            c.rx = HX ? q[QX + 2] : 0.;
            auto keep_d = [&](int j) {
                Dloc[j - lo] = c.D;
                if (HM) Dmloc[j - lo] = c.Dm;
                if (HX) Dxloc[j - lo] = c.Dx;
            };
            auto keep_r = [&](int j) {
                rloc[j - lo] = c.rn;
                if (HX) rxloc[j - lo] = c.rx;
            };
            if (top <= hi) keep_d(top);
            keep_r(hi);
            for (int j = top - 1; j >= hi; --j) {
                d_step(c, j);
                if (j <= hi) keep_d(j);
            }
            for (int j = hi - 1; j >= lo; --j) {
                d_step(c, j);
                keep_d(j);
                r_step(c, j);
                keep_r(j);
            }
        }
        for (int j = lo; j <= hi; ++j) {
            const double rj = rloc[j - lo];
            const double psi = rj * psi_p;
            const cplx D = Dloc[j - lo];
            const cplx zeta = mk(psi, chi_c), zeta_p = mk(psi_p, chi_p);
            const double tt = j * xinv;
            const cplx ca = D * minv + tt;
            const cplx na = ca * psi - psi_p;
            const cplx ida = cinv(ca * zeta - zeta_p);
            const cplx a = na * ida;
            const cplx cb = m * D + tt;
            const cplx nbq = cb * psi - psi_p;
            const cplx idb = cinv(cb * zeta - zeta_p);
            const cplx bb = nbq * idb;
            const cplx ida2 = ida * ida, idb2 = idb * idb;
            cplx am = ap, bm = ap, ax = ap, bx = ap;
            if (HM) {
                const cplx Dm = Dmloc[j - lo];
                const cplx da = (Dm * minv - D * minv2) * ida2, db = (D + m * Dm) * idb2;
                const double W = psi_p * chi_c - psi * chi_p;
                am = mk(-W * da.im, W * da.re);      // i W da
                bm = mk(-W * db.im, W * db.re);
            }
            double psix = 0.;
            if (HX) {
                psix = rxloc[j - lo] * psi_p + rj * psix_p;
                const cplx Dx = Dxloc[j - lo];
                const cplx zetal = mk(psix, chix_c), zetal_p = mk(psix_p, chix_p);
                const double tl = -tt * xinv * xl;
                const cplx c6 = Dx * minv - D * minv2 * ml + tl;
                ax = (c6 * psi + ca * psix - psix_p) * ida - na * ((c6 * zeta + ca * zetal - zetal_p) * ida2);
                const cplx c4 = ml * D + m * Dx + tl;
                bx = (c4 * psi + cb * psix - psix_p) * idb - nbq * ((c4 * zeta + cb * zetal - zetal_p) * idb2);
            }
            // sums of order j, and the asymmetry term of order j - 1 (it needs a_j, b_j)
            const double f1 = fv1[j], f4 = fv4[j];
            const double f3p = j >= 2 ? fv3[j - 1] : 0., f4p = j >= 2 ? fv4[j - 1] : 0.;
            const double sgn = (j & 1) ? -1. : 1.;
            acc[0] += f1 * (a.re + bb.re);
            acc[1] += f1 * (norm2(a) + norm2(bb));
            acc[2] += f1 * sgn * (a.re - bb.re);
            acc[3] += f1 * sgn * (a.im - bb.im);
            if (j >= 2) acc[4] += f3p * (re_mulc(ap, a) + re_mulc(bp, bb)) + f4p * re_mulc(ap, bp);
            if (HM) {
                // complex derivatives: the real part is d/dmr, the imaginary part d/dmi
                const cplx s = am + bm, d = am - bm, q2 = cmul(a, am) + cmul(bb, bm);
                accr[0] += f1 * s.re;
                acci[0] += f1 * s.im;
                accr[1] += f1 * 2. * q2.re;
                acci[1] += f1 * 2. * q2.im;
                accr[2] += f1 * sgn * d.re;
                accr[3] += f1 * sgn * d.im;
                if (j >= 2) {
                    const cplx g3 = cmul(a, amp) + cmul(ap, am) + cmul(bb, bmp) + cmul(bp, bm);
                    const cplx g4 = cmul(bp, amp) + cmul(ap, bmp);
                    accr[4] += f3p * g3.re + f4p * g4.re;
                    acci[4] += f3p * g3.im + f4p * g4.im;
                }
            }
            if (HX) {
                accx[0] += f1 * (ax.re + bx.re);
                accx[1] += f1 * 2. * (re_mulc(a, ax) + re_mulc(bb, bx));
                accx[2] += f1 * sgn * (ax.re - bx.re);
                accx[3] += f1 * sgn * (ax.im - bx.im);
                if (j >= 2)
                    accx[4] += f3p * (re_mulc(axp, a) + re_mulc(ap, ax) + re_mulc(bxp, bb) + re_mulc(bp, bx)) +
                               f4p * (re_mulc(axp, bp) + re_mulc(ap, bxp));
            }
            // coefficient columns of order j
            const int ek = oz_ek(j);
            auto put = [&](int col, cplx va, cplx vb) {
                const cplx cs = (va + vb) * f4, cd = (va - vb) * f4;
                cf[(size_t) col * tot + off + j - 1] = make_double4(cs.re, cs.im, cd.re, cd.im);
                if (re) track(mxe[col], cs, cd, ek);
            };
            if (to_tc) {
                tc_stage(tcbuf, n_tc, j, 0, (a + bb) * f4, (a - bb) * f4);
                for (int k = 0; k < B.nd1; ++k) {
                    cplx va = mk(0., 0.), vb = va;
                    if (HM) {
                        const cplx mk_ = B.m_l[C.ml_off + B.idx1[k]];
                        va = mk_ * am;
                        vb = mk_ * bm;
                    }
                    if (HX) {
                        const double xc = B.x_own ? 1. : B.xl[(size_t) k * R + r];
                        va = va + ax * xc;
                        vb = vb + bx * xc;
                    }
                    tc_stage(tcbuf, n_tc, j, 1 + k, (va + vb) * f4, (va - vb) * f4);
                }
                if (((j - 1) & 3) == 3 || j == n1) tc_flush(tcbuf, tcb, n_tc, j, tpos, j == n1 ? tgnk : 0);
            } else {
                put(0, a, bb);
                if (HM) put(1, am, bm);
                if (HX) put(1 + HM, ax, bx);
            }
            // upward: chi_{j+1} and its tangent; shift the previous order
            const double a1 = (2. * j + 1.) * xinv;
            const double chi_n = a1 * chi_c - chi_p;
            if (HX) {
                const double a2l = -a1 * xl * xinv;
                const double chix_n = a2l * chi_c + a1 * chix_c - chix_p;
                chix_p = chix_c;
                chix_c = chix_n;
                psix_p = psix;
                axp = ax;
                bxp = bx;
            }
            chi_p = chi_c;
            chi_c = chi_n;
            psi_p = psi;
            ap = a;
            bp = bb;
            amp = am;
            bmp = bm;
        }
    }
    auto put_sums = [&](int col, const double (&v)[5]) {
#pragma unroll
        for (int q = 0; q < 5; ++q) rs[((size_t) col * 5 + q) * R + r] = v[q];
    };
    put_sums(0, acc);
    if (HM) {
        // sb is complex itself: its derivative w.r.t. mi is -i times the one w.r.t. mr
        acci[2] = accr[3];
        acci[3] = -accr[2];
        put_sums(1, accr);
        put_sums(2, acci);
    }
    if (HX) put_sums(1 + 2 * HM, accx);
    if (re) {
#pragma unroll
        for (int c = 0; c < 1 + HM + HX; ++c)
            *(int4 *) (re + ((size_t) c * R + r) * 4) = make_int4(mxe[c][0], mxe[c][1], mxe[c][2], mxe[c][3]);
    }
}

template <bool HM, bool HX>
int launch(cudaStream_t s, const DevBatch &B, double *ck, double *coef, float *bop, double *rs) {
    if (bop)
        k_mie<HM, HX, true><<<ceil_div(B.R, 64), 64, 4 * 8 * (1 + B.nd1) * 64 * sizeof(float), s>>>(B, ck, coef, bop, rs);
    else
        k_mie<HM, HX, false><<<ceil_div(B.R, 64), 64, 0, s>>>(B, ck, coef, nullptr, rs);
    LMIEB_CUDA_TRY(cudaGetLastError());
    return 0;
}

}  // namespace

int launch_coef(cudaStream_t s, const DevBatch &B, double *ck, double *coef, float *bop, double *rs) {
    const bool hm = B.t_m > 0, hx = B.t_x > 0;
    if (hm) return hx ? launch<true, true>(s, B, ck, coef, bop, rs) : launch<true, false>(s, B, ck, coef, bop, rs);
    return hx ? launch<false, true>(s, B, ck, coef, bop, rs) : launch<false, false>(s, B, ck, coef, bop, rs);
}
