// oz_layout.cuh -- operands of the fixed-point angular contraction on the
// int8 tensor cores, shared by its operand kernels and its product kernel
// (k_oz.cu), K1 (which tracks the column exponents) and the driver.  Two
// formats: six digits (LMIEB_PRECISION_INT8) and seven (the large angular
// sums of LMIEB_PRECISION_FP64).
//
// The S1/S2 sums of a case are the dense products of tc_layout.cuh,
//     C[row, n] = sum_k A+[row, k] Bop[k, n],
// rows 2h / 2h+1 = (pi_k + tau_k)(mu_h) / s_k (pi_k - tau_k)(mu_h), columns
// the real and imaginary parts of S = fv4 (a + b) and D' = s_k fv4 (a - b) of
// the radii of a group.  Here every operand value becomes a signed integer of
// 8 ND - 1 fractional bits (47 with six digits, 55 with seven) and the integer
// products are summed exactly:
//   - order k gets the power of two 2^e_k, e_k = 2 ceil(log2 2k) (constant over
//     each chunk of 32 orders after the first): A+ is divided by it and Bop
//     multiplied by it, and each row r and column n gets its own power of two,
//     g_r and f_n, the smallest that bring every value of the row (all orders
//     of its case) or of the column to at most 1/2 in magnitude.  |pi +- tau|
//     grows like k^2 at the poles and slower elsewhere, so with the scale k^2
//     a row is largest at its first orders and g_r does not grow with the
//     case's order count: the small radii of a case keep their bits next to
//     the large ones (scale k instead, seven digits, x = 5 in a case of 950
//     orders: 1.7e-14 of |S|^2 against 3.9e-16; the FP64 sums: 5.5e-16);
//   - the scaled value x becomes V = round(x 2^(8 ND - 1)), |V| <= 2^(8 ND - 2),
//     written as ND balanced base-256 digits d_0 (most significant) .. in
//     [-128, 128), V = sum_i d_i 2^(8 (ND - 1 - i)): one int8 slice per digit;
//   - the product of A digit i and B digit j has the weight 2^(8 (2 ND - 2 - i - j));
//     the ND (ND + 1) / 2 products with i + j < ND are summed by tcgen05.mma
//     kind::i8 into ND int32 accumulators, one per diagonal i + j; the dropped
//     products (i + j >= ND) are below 2^-46 (six digits) or 2^-54 (seven) of
//     the largest term each;
//   - A and B digits are signed bytes; every int32 sum is exact (below
//     7 * 128 * 128 * 5120 < 2^31 for groups of up to 5120 orders);
//   - C = 2^(g_r + f_n - 14) sum_d 2^(-8 d) ACC_d, formed in int64 (to 2^-49 of
//     the largest term of the longest sums, 2^-57 of the shortest) and rounded
//     once to FP64.
// Each product then carries ~2^-46 (six digits) or ~2^-54 (seven; FP64: 2^-53
// and the rounding of every partial sum) of the largest term of its row and
// column.
//
// The pi/tau rows come from a recurrence in t = 1 - |mu| and the differences
// pi_k - pi_{k-1} (oz_rec): a rounding of mu pi_k near the pole, where
// pi_k ~ k^2 / 2 and its differences ~ k, is what limits the plain recurrence
// (relative error of |S|^2 summed exactly, plain / in t: x = 50 3.9e-14 /
// 7.7e-16, x = 900 2.0e-12 / 3.4e-15; the FP64 K3's 1.5e-14 / 7.7e-13).
//
// The A operand of a chunk of an angle tile is the same for every radius
// group of its case (the row exponent g_r is taken over all the case's
// orders): it is formed once per (case, tile, chunk) into memory, 32 ND bytes
// per product row -- slice s at 32 s, order 4 j + u in byte u of its 32-bit
// word j -- kept as 16-byte pieces with the rows of a piece consecutive
// (piece i of row r at 16 (i OZ_M + r)), and the product kernel stores it into
// tensor memory as it is.
//
// Layout of one chunk (OZ_KC orders) of the B operand in memory: ND slices,
// slice s holding digit s of every row, each slice in the tensor cores'
// K-major, no-swizzle core-matrix layout for 8-bit elements: 8 rows x 16
// orders (128 bytes) per core matrix, row groups 128 bytes apart, the two
// order groups rows / 8 * 128 bytes apart.  The A operand of a chunk lives in
// tensor memory: row r in lane r, slice s in 8 columns (4 orders per 32-bit
// column, order 4 j + u in byte u of column j).
#pragma once

#include <stdint.h>

constexpr int OZ_KC = 32;                            // orders per chunk (the K of one kind::i8 product)
constexpr int OZ_M = 128;                            // product rows: 64 half-angles and their mirrors
constexpr int OZ_HALF = OZ_M / 2;
constexpr int OZ_MAX_ND1 = 4;                        // index1 derivatives the kernel is built for
constexpr int OZ_MAX_ND2 = 3;                        // index2 derivatives the kernel is built for
constexpr int OZ_MAX_NK = 160;                       // chunks per group (5120 orders; int32 sums are exact to 18 thousand)
constexpr int OZ_MIN_N1 = 16;                        // smaller cases keep the FP64 angular stage

// whether the stage takes a case of truncation n1 whose radii reach n1max orders: at least OZ_MIN_N1, and
// radius groups that fit its exact int32 sums
inline bool oz_takes_orders(int n1, int n1max) {
    return n1 >= OZ_MIN_N1 && (n1max + OZ_KC - 1) / OZ_KC <= OZ_MAX_NK;
}

// The sizes of the two formats.  Tensor memory holds ND accumulators of NP
// columns and the A stages of 8 ND columns (512 in all): six digits leave
// room for 64 columns and two stages, seven for 48 columns (M 128, N 48 runs
// at 24.5 cycles per product: the rate of N 64, 32.1) and three stages.
template <int ND_>
struct Oz {
    static_assert(ND_ == 6 || ND_ == 7, "digits per value");
    static constexpr int ND = ND_;                        // base-256 digits per value
    static constexpr int NPROD = ND * (ND + 1) / 2;       // digit products per chunk (i + j < ND)
    static constexpr int NP = ND == 6 ? 64 : 48;          // operand rows (product N) per radius group
    static constexpr int NHALF = NP / 2;                  // rows of S (then D')
    static constexpr int ASTAGES = ND == 6 ? 2 : 3;       // A operand stages (tensor memory)
    static constexpr int ASLOTS = ND == 6 ? 2 : 3;        // A operand slots in shared memory (bulk copies)
    static constexpr int BSLOTS = 4;                      // B operand slots (bulk copies)
    static constexpr uint32_t BSLICE = NP * OZ_KC;        // bytes of one B slice of a chunk
    static constexpr uint32_t BSTAGE = ND * BSLICE;       // one B chunk of a group
    static constexpr uint32_t LBO_B = (NP / 8) * 128;     // order-group stride of a B slice
    static constexpr int AROW = ND * OZ_KC;               // bytes of one product row of an A chunk
    static constexpr int ACHUNK = OZ_M * AROW;            // bytes of one A chunk of an angle tile
    static constexpr int FRAC = 8 * ND - 1;               // fractional bits of the fixed-point values
    // exponent of the combination's row- and column-independent factor:
    // V_A V_B = 2^(16 (ND - 1)) sum_d 2^(-8 d) ACC_d, and the sums are kept in
    // units of 2^-16 of that sum (times 2^oz_sum_shift)
    static constexpr int CSHIFT = 16 * (ND - 1) - 2 * FRAC - 16;
};

// Bits kept below the unit of ACC_2 in the int64 sums of a group of nk chunks:
// |ACC_0 2^16 + ACC_1 2^8 + ACC_2| < 1.01 2^33 nk, so the sums stay below 2^63.
__host__ __device__ inline int oz_sum_shift(int nk) {
#ifdef __CUDA_ARCH__
    return 29 - (32 - __clz(nk - 1));
#else
    return 29 - (nk > 1 ? 32 - __builtin_clz((unsigned) (nk - 1)) : 0);
#endif
}

// the same for code that picks the format at run time
inline int oz_np(int nd) { return nd == 6 ? Oz<6>::NP : Oz<7>::NP; }
inline size_t oz_bstage(int nd) { return nd == 6 ? Oz<6>::BSTAGE : Oz<7>::BSTAGE; }
inline size_t oz_achunk(int nd) { return nd == 6 ? Oz<6>::ACHUNK : Oz<7>::ACHUNK; }
inline int oz_nprod(int nd) { return nd * (nd + 1) / 2; }
// radii per group for nt tangent columns (at most 2)
inline int oz_rg(int nd, int nt) { return oz_np(nd) / 2 / (2 * (1 + nt)); }

// Bound on |beta_l(fixed point) - beta_l(FP64)| / (2l + 1) of the expansion
// coefficients near the truncation threshold (|beta_l| within 1e-9 .. 1e-5 of
// 2l + 1), for a case reaching n1 orders.  Measured at most, with seven digits
// and with six: up to 1152 orders 7.3e-14 and 9.8e-14 (2000 single radii, 4600
// cases of 2 to 2000 radii in narrow and in broad ranges, 9000 distributions of
// every width); beyond, 1.4e-13 (880 cases of x from 1120 to 5000, 1 to 300 radii).
// Averaging over many radii does not lower it -- the largest values with seven
// digits belong to 500 radii over x up to 980, and most of them are the FP64
// kernel's -- although it is small (8.4e-15, 1.1e-14) in 8192 uneven cases.  A
// case with some |beta_l| within oz_trunc_band (2l + 1) of `accuracy` before its
// truncation point is solved again in FP64, which costs a batch the time of its
// largest such case: 3 of 1531 cases 2.0 ms.
__host__ __device__ inline double oz_trunc_band(int n1) { return n1 > 1152 ? 5e-13 : 2.5e-13; }
// 1.5 * 2^52 + 0x808080808080: see oz_digits
constexpr double OZ_MAGIC = 6896688841130112.0;

// e_c = 2 (6 + bit length of c): the order exponent of every order of chunk
// c >= 1 (orders 32 c + 1 .. 32 c + 32: ceil(log2 2k) is constant there)
__host__ __device__ inline int oz_ec(int c) {
#ifdef __CUDA_ARCH__
    return 2 * (6 + (32 - __clz(c)));
#else
    return 2 * (6 + (c ? 32 - __builtin_clz((unsigned) c) : 0));
#endif
}

// e_k = 2 ceil(log2 2k), k >= 1
__host__ __device__ inline int oz_ek(int k) {
#ifdef __CUDA_ARCH__
    return 2 * (32 - __clz(2 * k - 1));
#else
    return 2 * (32 - __builtin_clz((unsigned) (2 * k - 1)));
#endif
}

#ifdef __CUDACC__
// 2^e as a double, -1022 <= e <= 1023
__device__ __forceinline__ double oz_pow2(int e) { return __hiloint2double((1023 + e) << 20, 0); }

// The digits of V = round(x s), |x s| <= 2^(8 ND - 2), as bytes of V + B with
// B = 0x80 in each of the ND low bytes: V + B > 0, and its byte i is digit
// ND - 1 - i plus 128 (adding 128 to each balanced digit makes it a plain byte
// with no carries).  lo gets bytes 0..3, hi the others; a byte xor 0x80 is the
// digit as a two's-complement int8.  Six digits: t = x s + 1.5 2^52 + B is an
// integer in [2^52, 2^53) formed with one rounding, so the low 48 bits of its
// significand are V + B; seven digits exceed the significand and round to a
// 64-bit integer.
template <int ND>
__device__ __forceinline__ void oz_digits(double x, double s, uint32_t &lo, uint32_t &hi) {
    if (ND == 6) {
        const double t = fma(x, s, OZ_MAGIC);
        lo = (uint32_t) __double2loint(t);
        hi = (uint32_t) __double2hiint(t);
    } else {
        const unsigned long long u = (unsigned long long) __double2ll_rn(x * s) + 0x0080808080808080ull;
        lo = (uint32_t) u;
        hi = (uint32_t) (u >> 32);
    }
}

// Byte transpose of four words (consecutive orders): b_i = byte i of w0..w3.
__device__ __forceinline__ void oz_t4(uint32_t w0, uint32_t w1, uint32_t w2, uint32_t w3, uint32_t &b0,
                                      uint32_t &b1, uint32_t &b2, uint32_t &b3) {
    const uint32_t t0 = __byte_perm(w0, w1, 0x5140), t1 = __byte_perm(w2, w3, 0x5140);
    const uint32_t t2 = __byte_perm(w0, w1, 0x7362), t3 = __byte_perm(w2, w3, 0x7362);
    b0 = __byte_perm(t0, t1, 0x5410);
    b1 = __byte_perm(t0, t1, 0x7632);
    b2 = __byte_perm(t2, t3, 0x5410);
    b3 = __byte_perm(t2, t3, 0x7632);
}

// Digit slices of four consecutive orders of one row: w[s] holds digit s of
// the four orders (byte u = order u) as int8.
template <int ND>
__device__ __forceinline__ void oz_slices4(const uint32_t (&lo)[4], const uint32_t (&hi)[4], uint32_t (&w)[ND]) {
    uint32_t b[8];
    oz_t4(lo[0], lo[1], lo[2], lo[3], b[0], b[1], b[2], b[3]);
    oz_t4(hi[0], hi[1], hi[2], hi[3], b[4], b[5], b[6], b[7]);
#pragma unroll
    for (int s = 0; s < ND; ++s) w[s] = b[ND - 1 - s] ^ 0x80808080u;
}

// The pi/tau recurrence of one half-angle (reference src/lmie_core.c:658-721)
// at |mu|, in t = 1 - |mu| and d_k = pi_k - pi_{k-1}: with w = t pi_k and
// q = mu pi_k - pi_{k-1} = d_k - w,
//     tau_k = k q - pi_{k-1},  d_{k+1} = (k + 1) / k q - w,  pi_{k+1} = pi_k + d_{k+1}.
// Near the pole, where the pi_k agree in their leading digits, nothing larger
// than the differences is rounded.
struct oz_rec {
    double t, p0, p1, d, k;             // t, pi_{k-1}, pi_k, d_k, k
    __device__ __forceinline__ void start(double mu) {
        t = 1. - fabs(mu);
        p0 = 0.;
        p1 = d = k = 1.;
    }
    // tau_k and (in pk) pi_k of the current order; then on to order k + 1
    // (f2 = (k + 1) / k)
    __device__ __forceinline__ double step(double f2, double &pk) {
        const double w = t * p1, q = d - w, tau = fma(k, q, -p0);
        pk = p1;
        d = fma(q, f2, -w);
        p0 = p1;
        p1 += d;
        k += 1.;
        return tau;
    }
};

// smallest g with m <= 2^(g - 1) (m > 0): one bit of headroom; 0 for m = 0
__device__ __forceinline__ int oz_exp_of(double m) { return m > 0. ? ilogb(m) + 2 : 0; }
#endif
