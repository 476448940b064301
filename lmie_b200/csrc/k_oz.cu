// k_oz.cu -- K3 as an exact fixed-point contraction on the int8 tensor cores
// (operand formats in oz_layout.cuh): six digits for LMIEB_PRECISION_INT8,
// seven for the large angular sums of LMIEB_PRECISION_FP64.
//
// The S1/S2 sums over orders (reference src/lmie_core.c:658-721) of one case
// are the product A+ [S | D'] of 128 rows (64 half-angles of a tile and their
// mirrors, interleaved) by the NP operand rows of a radius group, over the
// orders.  Three kernels:
//   - k_oz_aop: per product row of every angle tile, the pi/tau recurrence
//     over the case's orders, once for the row exponent and once for the row's
//     digit slices of every chunk (the A operand is the same for all radius
//     groups of the case);
//   - k_oz_bop: per radius group, the column exponents f_n and the digit
//     slices of the B operand, chunk by chunk, from K1's FP64 coefficient
//     columns;
//   - k_angular_oz: a block owns one angle tile of one case and a range of its
//     radius groups; per group, chunks of OZ_KC orders flow through the
//     pipeline:
//       * lane 0 of warp 14 brings the chunks' A digit slices -- formed once per
//         (case, angle tile, chunk) by k_oz_aop -- and the group's B chunks into
//         shared memory with bulk copies running ahead of the products;
//       * warps 16-19 (one thread per row, the row's tensor-memory lane) store
//         A from there into its stage in tensor memory.  (Loads of A by these
//         threads hold an SM to what they keep in flight: 31 bytes per cycle,
//         1.6K cycles for a chunk of uneven batches, whose products take 0.7K.
//         tcgen05.cp from shared memory takes its time from the products, 7 x
//         34 cycles per chunk; these stores do not.  Six digits, 1000 cases
//         without index1 derivatives: 1262 us with loads, 987 with
//         tcgen05.cp, 834 this way; seven digits, 900 cases, one: 3193, 2351,
//         2006.);
//       * warps 12 and 13 issue the digit products of a chunk (21 or 28),
//         tcgen05.mma kind::i8 with A in tensor memory and B in shared memory
//         (M 128, N NP, K 32, int32 accumulation in tensor memory), one
//         accumulator per digit diagonal: one warp the even diagonals, the
//         other the odd ones.  The tensor pipe queues hardly any products
//         behind the one it runs, so a single issuing warp leaves it idle
//         while it waits for and sets up the next chunk (about 280 cycles per
//         chunk: 33.5 cycles per product of M 128, N 48 instead of 24.5, 43
//         instead of 32 at N 64); with two, each one's set-up falls into the
//         other's products (24.3 and 32.2 measured in a loop of this shape);
//       * during a group's last chunk warps 4-7 (S columns) and 0-3 (D'
//         columns) read the accumulators of their row (tensor-memory
//         lane = row) phase by phase -- diagonals 0-2, 3-4, 5 on -- as each
//         phase's products complete, add them up in int64 and hand the phase's
//         accumulators back, so the next group's products of that phase start.
//         The products go out by ascending diagonal, so while one group's
//         later diagonals run its first ones are read, and while the last ones
//         are read the next group's first ones run: tensor memory has no room
//         for a second accumulator set, and reading a whole group between its
//         last product and the next group's first one left the tensor pipe
//         idle for 2.2K cycles per group (a chunk's products take 0.7K).  The
//         sums then go to a shared-memory buffer as doubles;
//       * warps 8-11 form, from the buffer and while the next group's
//         products run, the phase-matrix quadratic forms and their
//         linearisations per radius (reference src/lmie_core.c:723-790; sm of
//         a row is in its pair row), accumulated over the block's radii in
//         registers.
// FP64 arithmetic waits for the products: a DFMA beside a running kind::i8
// stream completes every 128 cycles (2.5 without one), while integer, FP32 and
// conversion instructions are not slowed.  So the sums and their scaling are
// integer arithmetic and one conversion each, and what is left in FP64 is the
// quadratic forms, kept short: the sums over radii are formed for the complex
// tangent column (k_mie.cu) with the weight folded into the value's side, and
// turned into derivatives once at the end.
// The integer sums are exact, so nothing is drained during a group.
// Partials go to the same per-group buffer as the FP64 K3.
//
// Tensor memory: the accumulator of diagonal d at columns [d NP, (d + 1) NP);
// A stage s at ACOL + s ACOLS, slice i at +8 i.
//
// Every wait is bounded (about 1 s of clock, or until another block has
// failed); a block that gives up sets the error word, waits (bounded) for
// its tensor-core work and copies in flight, releases its tensor memory and
// returns.
#include <climits>
#include <cstdio>

#include "kernels.h"
#include "oz_layout.cuh"
#include "tc_ptx.cuh"

namespace {

constexpr int OZ_T = 640;                     // warps 0-7: sums (0-3 D', 4-7 S); 8-11: quadratic forms;
                                              // 12, 13: products; 14: operand copies; 16-19: A stages
constexpr int OZ_QUAD_WARP = 8, OZ_MMA_WARP = 12, OZ_COPY_WARP = 14, OZ_STAGE_WARP = 16;
// Registers a thread of each group of four warps: 96 at launch (640 threads),
// then 2 x 128 + 144 + 2 x 40 = 5 x 96.
constexpr int OZ_REG_SUMS = 128, OZ_REG_QUAD = 144, OZ_REG_REST = 40;
static_assert(2 * OZ_REG_SUMS + OZ_REG_QUAD + 2 * OZ_REG_REST <= 5 * 96, "no more registers than at launch");
constexpr uint32_t OZ_TMEM_COLS = 512;

// sizes and shared-memory offsets of the product kernel
template <int ND>
struct OzK : Oz<ND> {
    using F = Oz<ND>;
    static constexpr int MAX_GN = F::NHALF / 2;                        // radii of a group (oz_rg(nd, 0))
    static constexpr int MAX_W = 128;                                  // weights of a group: one per thread
    static constexpr uint32_t ACOLS = ND * OZ_KC / 4;                  // tensor-memory columns of an A stage
    static constexpr uint32_t ACOL = ND * F::NP;                       // first A stage column
    // barriers: afull[BSLOTS], bfull[BSLOTS], done[BSLOTS], ain[ASLOTS], accfull[3], accfree[3], hready[2],
    // hfree[2], fin
    static constexpr int NBAR = 3 * F::BSLOTS + F::ASLOTS + 11;
    static constexpr uint32_t O_ARING = F::BSLOTS * F::BSTAGE, RING = O_ARING + F::ASLOTS * F::ACHUNK;
    static constexpr int HB = F::NP * OZ_M;                            // doubles of one sums buffer
    static constexpr uint32_t HBUF = 2 * HB * 8;                       // two groups' sums, unscaled, [column][row]
    static constexpr uint32_t WBUF = MAX_W * 8;                        // a group's radius weights
    static constexpr uint32_t CBUF = F::NP * 4;                        // a group's column exponents
    static constexpr uint32_t O_HBUF = RING, O_WBUF = O_HBUF + HBUF, O_CBUF = O_WBUF + WBUF, O_BARS = O_CBUF + CBUF;
    static constexpr uint32_t SMEM = O_BARS + NBAR * 8 + 16;

    static_assert(F::BSTAGE % 128 == 0 && O_HBUF % 128 == 0, "B stages and sums start on 128-byte boundaries");
    static_assert(F::NP % 16 == 0 && F::NP >= 16 && F::NP <= 256, "N of an M=128 kind::i8 product");
    static_assert(ACOL + F::ASTAGES * ACOLS <= OZ_TMEM_COLS, "accumulators and A stages in tensor memory");
    static_assert(F::ASTAGES <= F::BSLOTS && F::ASLOTS <= F::BSLOTS, "a chunk's barriers outlive its stages");
    static_assert(WBUF % 16 == 0 && CBUF % 16 == 0, "barriers stay 8-byte aligned");
    static_assert(SMEM <= 227 * 1024, "shared memory per block");
    // weights per radius: value, index2, and with tangent columns index1 (twice with the x column)
    static_assert(MAX_GN * (1 + OZ_MAX_ND2 + OZ_MAX_ND1) <= MAX_W &&
                  MAX_GN / 2 * (1 + OZ_MAX_ND2 + 2 * OZ_MAX_ND1) <= MAX_W, "one weight per thread");
    // |V| <= 2^(FRAC - 1) must stay inside the balanced digits (-0x8080.. .. 0x7f7f..)
    static_assert(F::FRAC - 1 <= 8 * ND - 2, "digit weights: the top digit holds at most 64");
};

// instruction descriptor of kind::i8: D int32, A and B signed 8-bit, both K-major
__host__ __device__ constexpr uint32_t idesc_i8(int m, int n) {
    return (2u << 4) | (1u << 7) | (1u << 10) | ((uint32_t) (n >> 3) << 17) | ((uint32_t) (m >> 4) << 24);
}

// The registers a thread of the caller's four warps (a multiple of four) may
// use from here on.
template <int N>
__device__ __forceinline__ void reg_inc() {
    asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(N));
}
template <int N>
__device__ __forceinline__ void reg_dec() {
    asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(N));
}

// lane 0's value, which the compiler then knows to be the same in the whole
// (converged) warp
template <class T>
__device__ __forceinline__ T warp_uniform(T v) {
    return __shfl_sync(0xffffffffu, v, 0);
}

// 1 in one lane of a converged warp (the lowest), 0 in the others
__device__ __forceinline__ uint32_t elect_one() {
    uint32_t pred = 0;
    asm volatile(
        "{\n\t.reg .pred P;\n\t"
        "elect.sync _|P, 0xffffffff;\n\t"
        "selp.u32 %0, 1, 0, P;\n\t}"
        : "=r"(pred));
    return pred;
}

// A from tensor memory (column address a), B from shared memory; issued by the
// lane whose `on` is set.  The lane is picked by a guard on the instruction,
// not by a branch: outside a divergent branch the operands stay in uniform
// registers, from which the instruction takes them (one warp issues a product
// every 24 cycles or less this way, every 47 in a branch for one lane).
__device__ __forceinline__ void mma_i8_ts(uint32_t d, uint32_t a, uint64_t b, uint32_t idesc, uint32_t accumulate,
                                          uint32_t on) {
    asm volatile(
        "{\n\t.reg .pred p, q;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "setp.ne.b32 q, %5, 0;\n\t"
        "@q tcgen05.mma.cta_group::1.kind::i8 [%0], [%1], %2, %3, p;\n\t}" ::"r"(d),
        "r"(a), "l"(b), "r"(idesc), "r"(accumulate), "r"(on)
        : "memory");
}

// mma_commit by the lane whose `on` is set
__device__ __forceinline__ void mma_commit_on(uint32_t bar, uint32_t on) {
    asm volatile(
        "{\n\t.reg .pred q;\n\t"
        "setp.ne.b32 q, %1, 0;\n\t"
        "@q tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];\n\t}" ::"r"(bar),
        "r"(on)
        : "memory");
}

// warp-wide: four consecutive 32-bit columns of this thread's lane
__device__ __forceinline__ void tmem_st4(uint32_t taddr, uint32_t a, uint32_t b, uint32_t c, uint32_t d) {
    asm volatile("tcgen05.st.sync.aligned.32x32b.x4.b32 [%0], {%1, %2, %3, %4};" ::"r"(taddr), "r"(a), "r"(b),
                 "r"(c), "r"(d)
                 : "memory");
}

// Read-out phases of the accumulators: diagonals [oz_ph(p), oz_ph(p + 1)).
constexpr int OZ_NPH = 3;
template <int ND>
__host__ __device__ constexpr int oz_ph(int p) { return p == 0 ? 0 : (p == 1 ? 3 : (p == 2 ? 5 : ND)); }

// The digit products of diagonals D0, D0 + STEP, ... below D1 of one chunk
// by the lane with `on` (warp-wide): a0 the tensor-memory column of the
// chunk's A stage, b0 the shared address of its B stage, acc the
// tensor-memory column of diagonal 0; `first`: the chunk opens the group's
// sums.
template <int ND, int D0, int D1, int STEP>
__device__ __forceinline__ void issue_products_i8(uint32_t a0, uint32_t b0, uint32_t acc, bool first, uint32_t on) {
    using F = Oz<ND>;
    constexpr uint32_t idesc = idesc_i8(OZ_M, F::NP);
    const uint64_t db = sdesc(b0, F::LBO_B, 128);
#pragma unroll
    for (int d = D0; d < D1; d += STEP)
#pragma unroll
        for (int i = 0; i <= d; ++i) {
            const int j = d - i;
            mma_i8_ts(acc + d * F::NP, a0 + i * (OZ_KC / 4), db + (uint64_t) ((j * F::BSLICE) >> 4), idesc,
                      (first && i == 0) ? 0u : 1u, on);
        }
}

// One issuing warp's products of one chunk: its diagonals (parity PAR) phase by
// phase.  open: the chunk opens its group's sums; held: the previous group's
// accumulators of a phase must have been read first (accfree, parity fpar);
// close: it ends them, and the products of a phase complete the group's sums
// of it (accfull).  Returns whether a wait gave up (warp-uniform).
template <int ND, int PAR, int PH>
__device__ __forceinline__ bool oz_issue_phase(uint32_t a0, uint32_t b0, uint32_t acc, bool open, bool held,
                                               bool close, uint32_t accfull0, uint32_t accfree0, uint32_t fpar,
                                               uint32_t done, uint32_t on, const int *err) {
    constexpr int P0 = oz_ph<ND>(PH), D0 = P0 + ((P0 ^ PAR) & 1);
    if (held) {
        if (__any_sync(0xffffffffu, !mbar_wait(accfree0 + 8 * PH, fpar, err))) return true;
        tc_fence_after();
    }
    issue_products_i8<ND, D0, oz_ph<ND>(PH + 1), 2>(a0, b0, acc, open, on);
    if (PH == OZ_NPH - 1) mma_commit_on(done, on);
    if (close) mma_commit_on(accfull0 + 8 * PH, on);
    return false;
}

template <int ND, int PAR>
__device__ __forceinline__ bool oz_issue_chunk(uint32_t a0, uint32_t b0, uint32_t acc, bool open, bool held, bool close,
                                               uint32_t accfull0, uint32_t accfree0, uint32_t fpar, uint32_t done,
                                               uint32_t on, const int *err) {
    return oz_issue_phase<ND, PAR, 0>(a0, b0, acc, open, held, close, accfull0, accfree0, fpar, done, on, err) ||
           oz_issue_phase<ND, PAR, 1>(a0, b0, acc, open, held, close, accfull0, accfree0, fpar, done, on, err) ||
           oz_issue_phase<ND, PAR, 2>(a0, b0, acc, open, held, close, accfull0, accfree0, fpar, done, on, err);
}

// Phase PH's part of the sums V[c] (units of 2^-sh of ACC_2's) of one half's
// columns in this thread's lane, from tensor memory (taddr: the lane's first
// column of diagonal 0; warp-wide).  The loads of a batch of columns go out
// before one wait.
template <int ND, int PH>
__device__ __forceinline__ void oz_read_phase(uint32_t taddr, int sh, long long (&V)[Oz<ND>::NHALF]) {
    constexpr int D0 = oz_ph<ND>(PH), NA = oz_ph<ND>(PH + 1) - D0, NHALF = Oz<ND>::NHALF;
    constexpr int NC = 8;                               // columns per batch
    static_assert(NHALF % NC == 0, "whole batches");
#pragma unroll
    for (int c = 0; c < NHALF; c += NC) {
        uint32_t a[NA][NC];
#pragma unroll
        for (int d = 0; d < NA; ++d) tmem_ld8(taddr + (D0 + d) * Oz<ND>::NP + c, a[d]);
        tmem_wait_ld();
#pragma unroll
        for (int i = 0; i < NC; ++i) {
#pragma unroll
            for (int d = 0; d < NA; ++d) reg_after_wait(a[d][i]);
            if (PH == 0) {
                V[c + i] = ((long long) (int) a[0][i] * 65536 + (long long) (int) a[1][i] * 256 + (int) a[2][i]) << sh;
            } else if (PH == 1) {
                V[c + i] += ((long long) (int) a[0][i] * 256 + (int) a[1][i]) << (sh - 16);
            } else if (ND == 6) {
                // unit 2^-24: sh is 21 .. 29
                const long long v = (int) a[0][i];
                V[c + i] += sh >= 24 ? v << (sh - 24) : (v + (1 << (23 - sh))) >> (24 - sh);
            } else {
                // unit 2^-32
                const long long v = (long long) (int) a[0][i] * 256 + (int) a[NA - 1][i];
                V[c + i] += (v + (1 << (31 - sh))) >> (32 - sh);
            }
        }
    }
}

// One thread's part of taking a group's sums out of tensor memory: every phase
// as its products complete (accfull), handing it back (accfree) for the next
// group.  Returns whether a wait gave up (warp-uniform: the tensor-memory
// accesses are warp-wide).
template <int ND>
__device__ __forceinline__ bool oz_take(uint32_t taddr, int sh, long long (&V)[Oz<ND>::NHALF], uint32_t accfull0,
                                        uint32_t accfree0, uint32_t parity, const int *err) {
    if (__any_sync(0xffffffffu, !mbar_wait(accfull0, parity, err))) return true;
    tc_fence_after();
    oz_read_phase<ND, 0>(taddr, sh, V);
    tc_fence_before();
    mbar_arrive(accfree0);
    if (__any_sync(0xffffffffu, !mbar_wait(accfull0 + 8, parity, err))) return true;
    tc_fence_after();
    oz_read_phase<ND, 1>(taddr, sh, V);
    tc_fence_before();
    mbar_arrive(accfree0 + 8);
    if (__any_sync(0xffffffffu, !mbar_wait(accfull0 + 16, parity, err))) return true;
    tc_fence_after();
    oz_read_phase<ND, 2>(taddr, sh, V);
    tc_fence_before();
    mbar_arrive(accfree0 + 16);
    return false;
}

// v 2^(e >> 20) for a value v that came from an integer (zero or normal)
__device__ __forceinline__ double oz_scaled(double v, int e) {
    const int hi = __double2hiint(v);
    return __hiloint2double(hi ? hi + e : 0, __double2loint(v));
}

// ---------------------------------------------------------------------------
// B operand of the radius groups: block per group, thread per operand row
// n = tid % NP (S re, S im, ..., then D' re, D' im, ...) and every fourth
// block of 16 orders.  The column exponent f_n (largest ilogb(|v| 2^e_k) + 2
// over the column) comes from the exponents K1 tracked while it wrote the
// coefficients; the kernel writes the digit slices of every chunk; rows and
// orders without a value get zero.
// ---------------------------------------------------------------------------
constexpr int OZ_BOP_J = 4;                           // threads per row

template <int ND>
__global__ void __launch_bounds__(OZ_BOP_J * Oz<ND>::NP) k_oz_bop(DevBatch B, const double *__restrict__ coef,
                                                      unsigned char *__restrict__ bop, int *__restrict__ colexp) {
    constexpr int OZ_NP = Oz<ND>::NP, OZ_NHALF = Oz<ND>::NHALF;
    const int g = blockIdx.x, tid = threadIdx.x;
    const int r0 = B.tg_r0[g], gn = B.tg_n[g], nk = B.tg_nk[g];
    const int C1 = 1 + (B.t_m > 0) + (B.t_x > 0), P = gn * C1;
    const int n = tid % OZ_NP, j0 = tid / OZ_NP;
    const int rp = (n % OZ_NHALF) >> 1;               // operand column pair (radius, Mie column)
    const int comp = (n >= OZ_NHALF ? 2 : 0) + (n & 1);   // re/im of S, then of D'
    const bool real = rp < P, dpart = n >= OZ_NHALF;
    const double *cf = coef + comp;                   // component `comp` of the double4 entries
    const size_t tot = (size_t) B.tot;
    int n1 = 0, f = 0;
    size_t base = 0;
    if (real) {
        const int p = rp / C1, col = rp - p * C1, r = r0 + p;
        n1 = B.n1r[r];
        base = ((size_t) col * tot + B.off[r]) * 4;
        // largest biased exponent + e_k: f = that - 1021 (0: the column is zero)
        const int m = B.oz_radexp[((size_t) col * B.R + r) * 4 + comp];
        f = m ? max(m - 1021, -900) : 0;
    }
    if (j0 == 0) colexp[(size_t) g * OZ_NP + n] = f;
    // digits, 16 orders at a time
    unsigned char *rb = bop + B.tg_off[g] + (n >> 3) * 128 + (n & 7) * 16;
    for (int blk = j0; blk < 2 * nk; blk += OZ_BOP_J) {
        uint32_t w[ND][4];
#pragma unroll
        for (int qd = 0; qd < 4; ++qd) {
            uint32_t lo[4], hi[4];
#pragma unroll
            for (int u = 0; u < 4; ++u) {
                const int k = blk * 16 + qd * 4 + u + 1;
                double v = k <= n1 ? __ldg(cf + base + (size_t) (k - 1) * 4) : 0.;
                if (dpart && !(k & 1)) v = -v;        // s_k of D'
                oz_digits<ND>(v, oz_pow2(Oz<ND>::FRAC + oz_ek(k) - f), lo[u], hi[u]);
            }
            uint32_t s6[ND];
            oz_slices4<ND>(lo, hi, s6);
#pragma unroll
            for (int s = 0; s < ND; ++s) w[s][qd] = s6[s];
        }
        unsigned char *cb = rb + (size_t) (blk >> 1) * Oz<ND>::BSTAGE + (blk & 1) * Oz<ND>::LBO_B;
#pragma unroll
        for (int s = 0; s < ND; ++s)
            *(uint4 *) (cb + s * Oz<ND>::BSLICE) = make_uint4(w[s][0], w[s][1], w[s][2], w[s][3]);
    }
}

// ---------------------------------------------------------------------------
// A operand: thread per product row of every angle tile of every case (flat
// index space `start`, OZ_M rows per tile).  First the row exponent g_r over
// all the case's orders (rowexp[C.rx_off + 2h + mirror]), then the recurrence
// again: each chunk's row values scaled by 2^(FRAC - e_k - g_r), their digits
// and the row's digit slices, AROW bytes per chunk as AROW / 16 pieces of 16
// bytes, piece i (slice i / 2, orders 16 (i % 2) .. + 15) of the row at
// aop[C.a_off + (tile nkx + chunk) ACHUNK + (i OZ_M + row) 16]: the rows of a
// piece are consecutive, so the product kernel's warps read 512 contiguous
// bytes per load.  Rows past the case's angles get the digits of zero.
// A row is a serial chain of about 3 dependent FP64 operations per order and
// pass (x = 5000, 5077 orders: ~0.15 ms); it runs beside K1, whose chains are
// longer, so the second pass costs less than a table of the first one's
// values.
// ---------------------------------------------------------------------------
template <int ND>
__global__ void __launch_bounds__(128) k_oz_aop(DevBatch B, long long total, const long long *__restrict__ start,
                                                signed char *__restrict__ rowexp, unsigned char *__restrict__ aop) {
    const long long e = (long long) blockIdx.x * blockDim.x + threadIdx.x;
    if (e >= total) return;
    const int c = find_case(start, B.ncase, e);
    const DevCase &C = B.cs[c];
    const long long q = e - start[c];
    const int t = (int) (q / OZ_M), row = (int) (q % OZ_M);
    const int h = t * OZ_HALF + (row >> 1);
    const bool gact = h < C.nh;
    const double mu = gact ? B.mu_pool[C.mu_off + h] : 0.;
    // The recurrence runs at |mu|.  (pi + tau)(mu) and s_k (pi - tau)(mu), the
    // rows 2h and 2h + 1, change places for mu < 0: pi +- tau at -|mu| is
    // s_k (pi -+ tau) at |mu|.
    const bool minus = (mu < 0.) != ((row & 1) != 0);
    const double sg = minus ? -1. : 1.;
    oz_rec r;
    r.start(mu);
    double m = 0.;
    for (int kc = 0; kc < C.nkx; ++kc) {
        const double *f2 = B.oz_f2 + kc * OZ_KC + 1;
        double mc = 0.;
#pragma unroll 8
        for (int u = 0; u < OZ_KC; ++u) {
            double pk;
            const double tau = r.step(f2[u], pk);
            const double v = fabs(fma(sg, tau, pk));
            mc = fmax(mc, kc == 0 ? v * oz_pow2(-oz_ek(u + 1)) : v);
        }
        m = fmax(m, kc == 0 ? mc : mc * oz_pow2(-oz_ec(kc)));
    }
    const int gr = gact ? oz_exp_of(m) : 0;
    if (gact) rowexp[C.rx_off + 2 * (size_t) h + (row & 1)] = (signed char) gr;
    const double gsc = gact ? oz_pow2(Oz<ND>::FRAC - gr) : 0.;
    uint4 *dst = (uint4 *) (aop + C.a_off + (size_t) t * C.nkx * Oz<ND>::ACHUNK) + row;
    r.start(mu);
    for (int kc = 0; kc < C.nkx; ++kc) {
        // the chunk's scale 2^(FRAC - e_k - g_r); a minus row carries s_k
        const double sp = kc == 0 ? 0. : gsc * oz_pow2(-oz_ec(kc));
        const double *f2 = B.oz_f2 + kc * OZ_KC + 1;
        uint32_t w[ND][8];
#pragma unroll
        for (int qd = 0; qd < 8; ++qd) {
            uint32_t lo[4], hi[4];
#pragma unroll
            for (int u = 0; u < 4; ++u) {
                double pk;
                const double tau = r.step(f2[qd * 4 + u], pk);
                double sc = kc == 0 ? gsc * oz_pow2(-oz_ek(qd * 4 + u + 1)) : sp;
                if (minus && (u & 1)) sc = -sc;
                oz_digits<ND>(fma(sg, tau, pk), sc, lo[u], hi[u]);
            }
            uint32_t s6[ND];
            oz_slices4<ND>(lo, hi, s6);
#pragma unroll
            for (int sl = 0; sl < ND; ++sl) w[sl][qd] = s6[sl];
        }
        uint4 *dc = dst + (size_t) kc * (Oz<ND>::ACHUNK / 16);
#pragma unroll
        for (int sl = 0; sl < ND; ++sl) {
            dc[(2 * sl) * OZ_M] = make_uint4(w[sl][0], w[sl][1], w[sl][2], w[sl][3]);
            dc[(2 * sl + 1) * OZ_M] = make_uint4(w[sl][4], w[sl][5], w[sl][6], w[sl][7]);
        }
    }
}

// barrier 2 over the 128 threads of warps 8-11, OR-reducing v
__device__ __forceinline__ int oz_epi_sync_or(int v) {
    uint32_t r;
    asm volatile(
        "{\n\t.reg .pred p, q;\n\t"
        "setp.ne.u32 q, %1, 0;\n\t"
        "bar.red.or.pred p, 2, 128, q;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(r)
        : "r"(v)
        : "memory");
    return (int) r;
}

// ---------------------------------------------------------------------------
// The product kernel.
// ---------------------------------------------------------------------------
// TM: the m tangent column; TX: 0 no per-derivative sums, 1 those of index1
// derivatives that move the weights, 2 those and the x column.
template <int ND, int TM, int TX>
__global__ void __launch_bounds__(OZ_T, 1) k_angular_oz(DevBatch B, const AngItem *__restrict__ items,
                                                        const unsigned char *__restrict__ bop,
                                                        double *__restrict__ part, int *__restrict__ err) {
    using F = OzK<ND>;
    constexpr int NT = TM + (TX == 2), CPR = 2 * (1 + NT);   // columns of each half per radius
    constexpr int OZ_NP = F::NP, OZ_NHALF = F::NHALF, OZ_MAX_GN = F::MAX_GN, OZ_HB = F::HB;
    constexpr int OZ_ASTAGES = F::ASTAGES, OZ_BSLOTS = F::BSLOTS, OZ_ASLOTS = F::ASLOTS, OZ_NBAR = F::NBAR;
    constexpr uint32_t OZ_ACOL = F::ACOL, OZ_ACOLS = F::ACOLS, OZ_BSTAGE = F::BSTAGE, OZ_ACHUNK = F::ACHUNK;
    extern __shared__ __align__(1024) unsigned char smem[];
    double *hbuf = (double *) (smem + F::O_HBUF);            // [2][OZ_NP][OZ_M] sums of a group, unscaled
    double *wsh = (double *) (smem + F::O_WBUF);             // [radius][NS] weights
    int *csh = (int *) (smem + F::O_CBUF);                   // [OZ_NP] column exponents << 20
    uint64_t *bars = (uint64_t *) (smem + F::O_BARS);
    uint32_t *tmem_hold = (uint32_t *) (bars + OZ_NBAR);
    const uint32_t bring = smem_u32(smem);
    // chunk q: its A digits are in shared memory, ain[q % ASLOTS], and in tensor memory, afull[q % BSLOTS] (the
    // shared slot is then free again); its B digits are in shared memory, bfull[q % BSLOTS]; its products have
    // completed, done[q % BSLOTS] (both issuing warps)
    const uint32_t afull0 = smem_u32(bars), bfull0 = afull0 + 8 * OZ_BSLOTS, done0 = bfull0 + 8 * OZ_BSLOTS;
    const uint32_t ain0 = done0 + 8 * OZ_BSLOTS;
    const uint32_t accfull0 = ain0 + 8 * OZ_ASLOTS, accfree0 = accfull0 + 8 * OZ_NPH;
    const uint32_t hready0 = accfree0 + 8 * OZ_NPH, hfree0 = hready0 + 16, fin = hfree0 + 16;

    const int tid = threadIdx.x, warp = warp_uniform(tid >> 5);
    const AngItem it = items[blockIdx.x];
    const DevCase &C = B.cs[it.c];
    const int nh = C.nh, n_qang = C.n_qang, R = B.R;
    const int nd1 = B.nd1, nd2 = B.nd2, NS = 1 + nd2 + (TX > 0 ? nd1 : 0) + (TX == 2 ? nd1 : 0);

    // after a failure elsewhere the remaining blocks return at once
    __shared__ int s_skip;
    if (tid == 0) s_skip = *(volatile const int *) err;
    __syncthreads();
    if (s_skip) return;
    if (tid == 0) {
        for (int i = 0; i < OZ_BSLOTS; ++i) {
            mbar_init(afull0 + 8 * i, OZ_M);
            mbar_init(bfull0 + 8 * i, 1);
            mbar_init(done0 + 8 * i, 2);
        }
        for (int i = 0; i < OZ_ASLOTS; ++i) mbar_init(ain0 + 8 * i, 1);
        for (int i = 0; i < OZ_NPH; ++i) {
            mbar_init(accfull0 + 8 * i, 2);
            mbar_init(accfree0 + 8 * i, 256);
        }
        for (int i = 0; i < 2; ++i) {
            mbar_init(hready0 + 8 * i, 256);
            mbar_init(hfree0 + 8 * i, 128);
        }
        mbar_init(fin, 2);
        fence_mbar_init();
    }
    if (warp == 0) tmem_alloc(smem_u32(tmem_hold), OZ_TMEM_COLS);
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = *tmem_hold;
    int bad = 0;

    if (warp < OZ_QUAD_WARP) {
        reg_inc<OZ_REG_SUMS>();
        // ---------------- warps 0-7: the groups' sums, one row (lane) per thread ----------------
        // Warps 0-3 take the D' columns of a group's sums out of tensor memory,
        // warps 4-7 the S columns, and, once the quadratic forms are done with
        // the buffer's previous group, into the buffer.
        const int set = warp >> 2, row = tid & (OZ_M - 1);
        const int hcol = set == 0 ? OZ_NHALF : 0;            // first column of the set's half
        const uint32_t taddr = tmem + ((uint32_t) ((warp & 3) * 32) << 16) + hcol;
        int nk = it.rbeg < it.rend ? B.tg_nk[it.rbeg] : 1, gi = 0;
        for (int g = it.rbeg; g < it.rend; ++g, ++gi) {
            const int sh = oz_sum_shift(nk), b = gi & 1;
            if (g + 1 < it.rend) nk = B.tg_nk[g + 1];
            long long V[OZ_NHALF];
            if (oz_take<ND>(taddr, sh, V, accfull0, accfree0, gi & 1, err) ||
                __any_sync(0xffffffffu, gi >= 2 && !mbar_wait(hfree0 + 8 * b, ((gi >> 1) - 1) & 1, err))) {
                bad = 1;
                break;
            }
            double *hb = hbuf + b * OZ_HB + hcol * OZ_M + row;
#pragma unroll
            for (int i = 0; i < OZ_NHALF; ++i) hb[i * OZ_M] = (double) V[i];
            mbar_arrive(hready0 + 8 * b);
        }
    } else if (warp < OZ_MMA_WARP) {
        reg_inc<OZ_REG_QUAD>();
        // ---------------- warps 8-11: quadratic forms, one row per thread ----------------
        // A warp whose wait fails keeps taking the barriers of the four warps,
        // which stop together.
        const int t1 = tid - OZ_QUAD_WARP * 32;              // product row
        const int eh = t1 >> 1, emir = t1 & 1;
        const int ej = it.xt * OZ_HALF + eh;
        const bool eact = ej < nh;
        const signed char *gtab = B.oz_rowexp + C.rx_off + 2 * (size_t) (eact ? ej : 0) + emir;
        // f-weighted sums over radii: the value's four invariants, those of the
        // index2 columns, of the index1 derivatives' own weights and x column
        double rv[4] = {0., 0., 0., 0.}, r2[OZ_MAX_ND2][4], r1[TX ? OZ_MAX_ND1 : 1][4];
#pragma unroll
        for (int s = 0; s < OZ_MAX_ND2; ++s)
#pragma unroll
            for (int e = 0; e < 4; ++e) r2[s][e] = 0.;
#pragma unroll
        for (int s = 0; s < (TX ? OZ_MAX_ND1 : 1); ++s)
#pragma unroll
            for (int e = 0; e < 4; ++e) r1[s][e] = 0.;
        // with the m column: conj(sp) dsp, conj(sm) dsm, conj(sm) dsp, conj(sp) dsm
        cplx rm[TM ? 4 : 1];
#pragma unroll
        for (int e = 0; e < (TM ? 4 : 1); ++e) rm[e] = mk(0., 0.);
        // the scales of this row and of its pair row (which holds this row's sm)
        const double rsc = oz_pow2(eact ? (int) *gtab : 0);
        const double rsp = __shfl_xor_sync(0xffffffffu, rsc, 1);
        // A group's radius weights (gn NS <= MAX_W values, at most one per
        // thread) and column exponents (with the row-independent factor of the
        // combination), fetched into registers one group ahead so that their
        // loads overlap the previous group's forms.
        double wnext = 0.;
        int cnext = 0;
        auto fetch = [&](int g) {
            const int gn = B.tg_n[g];
            if (t1 < gn * NS && gn <= OZ_MAX_GN) {
                const int p = t1 / NS, s = t1 - p * NS, rad = B.tg_r0[g] + p;
                if (s <= nd2) {
                    wnext = B.w[(size_t) (s == 0 ? 0 : 1 + B.idx2[s - 1]) * R + rad];
                } else if (s <= nd2 + nd1) {
                    wnext = B.w[(size_t) (1 + B.idx1[s - 1 - nd2]) * R + rad];
                } else {
                    wnext = B.x_own ? 1. : B.xl[(size_t) (s - 1 - nd2 - nd1) * R + rad];
                }
            }
            if (t1 < OZ_NP)
                cnext = (B.oz_colexp[(size_t) g * OZ_NP + t1] + F::CSHIFT - oz_sum_shift(B.tg_nk[g])) * (1 << 20);
        };
        if (it.rbeg < it.rend) fetch(it.rbeg);
        int gi = 0;
        for (int g = it.rbeg; g < it.rend; ++g, ++gi) {
            const int gn = B.tg_n[g];
            // the previous group's weights and exponents have been read by all four warps
            if (oz_epi_sync_or(bad || gn > OZ_MAX_GN)) {
                bad = 1;
                break;
            }
            if (t1 < gn * NS) wsh[t1] = wnext;
            if (t1 < OZ_NP) csh[t1] = cnext;
            oz_epi_sync_or(0);
            // the next group's loads, in flight during this group's forms (a
            // barrier waits for the loads issued before it)
            if (g + 1 < it.rend) fetch(g + 1);
            // both halves of the group's sums are in its buffer
            const double *hb = hbuf + (gi & 1) * OZ_HB;
            if (__any_sync(0xffffffffu, !mbar_wait(hready0 + 8 * (gi & 1), (gi >> 1) & 1, err))) {
                bad = 1;
                continue;
            }
            // The row scales are left out here: every term of an invariant 0
            // (|sp|^2 and its tangents) carries rsc^2, of an invariant 1 rsp^2
            // and of the others rsc rsp (powers of two, applied once at the
            // end).
#pragma unroll (TM ? 2 : 4)
            for (int p = 0; p < gn; ++p) {
                // columns of S (i < CPR, this row) and D' (i >= CPR, the pair row: sm)
                double v[2 * CPR];
#pragma unroll
                for (int i = 0; i < CPR; ++i) {
                    const int cs = p * CPR + i, cd = OZ_NHALF + p * CPR + i;
                    v[i] = oz_scaled(hb[cs * OZ_M + t1], csh[cs]);
                    v[CPR + i] = oz_scaled(hb[cd * OZ_M + (t1 ^ 1)], csh[cd]);
                }
                const double *wp = wsh + p * NS;
                const double f = wp[0];
                // invariants of (sp, sm): |sp|^2, |sm|^2, Re(sp sm*), Im(sm sp*)
                const double spr = v[0], spi = v[1], smr = v[CPR], smi = v[CPR + 1];
                const double inv[4] = {spr * spr + spi * spi, smr * smr + smi * smi, spr * smr + spi * smi,
                                       smi * spr - smr * spi};
#pragma unroll
                for (int e = 0; e < 4; ++e) rv[e] += f * inv[e];
#pragma unroll
                for (int k = 0; k < OZ_MAX_ND2; ++k)
                    if (k < nd2) {
                        const double fl = wp[1 + k];
#pragma unroll
                        for (int e = 0; e < 4; ++e) r2[k][e] += fl * inv[e];
                    }
                // the weighted value, for the products with its tangents
                const double gpr = f * spr, gpi = f * spi, gmr = f * smr, gmi = f * smi;
                if (TM) {
                    const double dpr = v[2], dpi = v[3], dmr = v[CPR + 2], dmi = v[CPR + 3];
                    rm[0].re += gpr * dpr;  rm[0].re += gpi * dpi;
                    rm[0].im += gpr * dpi;  rm[0].im -= gpi * dpr;
                    rm[1].re += gmr * dmr;  rm[1].re += gmi * dmi;
                    rm[1].im += gmr * dmi;  rm[1].im -= gmi * dmr;
                    rm[2].re += gmr * dpr;  rm[2].re += gmi * dpi;
                    rm[2].im += gmr * dpi;  rm[2].im -= gmi * dpr;
                    rm[3].re += gpr * dmr;  rm[3].re += gpi * dmi;
                    rm[3].im += gpr * dmi;  rm[3].im -= gpi * dmr;
                }
                if (TX) {
                    double dx[4] = {0., 0., 0., 0.};
                    if (TX == 2) {
                        constexpr int X = 2 + 2 * TM;
                        const double plr = v[X], pli = v[X + 1], mlr = v[CPR + X], mli = v[CPR + X + 1];
                        dx[0] = 2. * (plr * gpr + pli * gpi);
                        dx[1] = 2. * (mlr * gmr + mli * gmi);
                        dx[2] = plr * gmr + pli * gmi + gpr * mlr + gpi * mli;
                        dx[3] = mli * gpr - mlr * gpi + gmi * plr - gmr * pli;
                    }
#pragma unroll
                    for (int k = 0; k < OZ_MAX_ND1; ++k)
                        if (k < nd1) {
                            const double fl = wp[1 + nd2 + k], xc = TX == 2 ? wp[1 + nd2 + nd1 + k] : 0.;
#pragma unroll
                            for (int e = 0; e < 4; ++e) {
                                r1[k][e] += fl * inv[e];
                                if (TX == 2) r1[k][e] += xc * dx[e];
                            }
                        }
                }
            }
            // the buffer is free for the group after next
            mbar_arrive(hfree0 + 8 * (gi & 1));
        }
        if (oz_epi_sync_or(bad)) bad = 1;
        if (!bad && eact) {
            // phase-matrix elements: ((A + B) / 4, (A - B) / 4, -C / 2, D / 2),
            // with the row scales
            const int jj = emir ? n_qang - 1 - ej : ej;
            const int Q = 4 * (1 + B.nd);
            double *pc = part + C.part_off + (size_t) it.g * Q * n_qang;
            const double ss = rsc * rsc, mm = rsp * rsp, sm = rsc * rsp;
            auto put = [&](int slot, const double (&q)[4]) {
                double *o = pc + (size_t) slot * 4 * n_qang + jj;
                const double a = q[0] * ss, b = q[1] * mm;
                o[0] = .25 * (a + b);
                o[(size_t) n_qang] = .25 * (a - b);
                o[(size_t) 2 * n_qang] = -.5 * (q[2] * sm);
                o[(size_t) 3 * n_qang] = .5 * (q[3] * sm);
            };
            put(0, rv);
#pragma unroll
            for (int k = 0; k < OZ_MAX_ND2; ++k)
                if (k < nd2) put(1 + B.idx2[k], r2[k]);
#pragma unroll
            for (int k = 0; k < OZ_MAX_ND1; ++k)
                if (k < nd1) {
                    double d[4];
#pragma unroll
                    for (int e = 0; e < 4; ++e) d[e] = TX ? r1[TX ? k : 0][e] : 0.;
                    if (TM) {
                        // d|sp|^2 = 2 Re(m_l conj(sp) dsp) and so on
                        const cplx ml = B.m_l[C.ml_off + B.idx1[k]];
                        const cplx u = rm[TM ? 2 : 0] + rm[TM ? 3 : 0], w = rm[TM ? 2 : 0] - rm[TM ? 3 : 0];
                        d[0] += 2. * (ml.re * rm[0].re - ml.im * rm[0].im);
                        d[1] += 2. * (ml.re * rm[TM ? 1 : 0].re - ml.im * rm[TM ? 1 : 0].im);
                        d[2] += ml.re * u.re - ml.im * u.im;
                        d[3] -= ml.re * w.im + ml.im * w.re;
                    }
                    put(1 + B.idx1[k], d);
                }
        }
    } else if (warp >= OZ_STAGE_WARP) {
        reg_dec<OZ_REG_REST>();
        // ---------------- warps 16-19: A stages, from shared to tensor memory, one row (lane) per thread ----------------
        const int row = tid & (OZ_M - 1);
        const uint32_t taddr = tmem + ((uint32_t) ((warp & 3) * 32) << 16) + OZ_ACOL;
        const uint4 *aring = (const uint4 *) (smem + F::O_ARING) + row;
        int q = 0;
        for (int g = it.rbeg; g < it.rend && !bad; ++g) {
            const int nk = B.tg_nk[g];
            for (int kc = 0; kc < nk; ++kc, ++q) {
                // the digits are there, and the stage's previous chunk has been multiplied
                const int as = q % OZ_ASLOTS, qp = q - OZ_ASTAGES;
                const bool ok = mbar_wait(ain0 + 8 * as, (q / OZ_ASLOTS) & 1, err) &&
                                (qp < 0 || mbar_wait(done0 + 8 * (qp % OZ_BSLOTS), (qp / OZ_BSLOTS) & 1, err));
                if (__any_sync(0xffffffffu, !ok)) {
                    bad = 1;
                    break;
                }
                tc_fence_after();
                const uint4 *ac = aring + as * (OZ_ACHUNK / 16);
                const uint32_t acol = taddr + (q % OZ_ASTAGES) * OZ_ACOLS;
#pragma unroll
                for (int i = 0; i < 2 * ND; ++i) {
                    const uint4 v = ac[i * OZ_M];
                    tmem_st4(acol + i * (OZ_KC / 8), v.x, v.y, v.z, v.w);
                }
                tmem_wait_st();
                tc_fence_before();
                mbar_arrive(afull0 + 8 * (q % OZ_BSLOTS));
            }
        }
    } else {
        reg_dec<OZ_REG_REST>();
        if (warp >= OZ_COPY_WARP) {
            // ---------------- warp 14, lane 0: operand copies, ahead of the products ----------------
            if (tid == OZ_COPY_WARP * 32) {
                const unsigned char *asrc = B.oz_aop + C.a_off + (size_t) it.xt * C.nkx * OZ_ACHUNK;
                int pq = 0, acopied = 0;
                for (int g = it.rbeg; g < it.rend && !bad; ++g) {
                    const int nk = B.tg_nk[g];
                    const unsigned char *src = bop + B.tg_off[g];
                    for (int kc = 0; kc < nk; ++kc, ++pq) {
                        const int ps = pq % OZ_BSLOTS, as = pq % OZ_ASLOTS, pa = pq - OZ_ASLOTS;
                        // the slots' previous chunks must have been copied on and consumed
                        if (pa >= 0 && !mbar_wait(afull0 + 8 * (pa % OZ_BSLOTS), (pa / OZ_BSLOTS) & 1, err)) {
                            bad = 1;
                            break;
                        }
                        mbar_expect_tx(ain0 + 8 * as, OZ_ACHUNK);
                        bulk_g2s(bring + F::O_ARING + as * OZ_ACHUNK, asrc + (size_t) kc * OZ_ACHUNK, OZ_ACHUNK, ain0 + 8 * as);
                        acopied = pq + 1;
                        if (pq >= OZ_BSLOTS && !mbar_wait(done0 + 8 * ps, ((pq / OZ_BSLOTS) - 1) & 1, err)) {
                            bad = 1;
                            break;
                        }
                        mbar_expect_tx(bfull0 + 8 * ps, OZ_BSTAGE);
                        bulk_g2s(bring + ps * OZ_BSTAGE, src, OZ_BSTAGE, bfull0 + 8 * ps);
                        src += OZ_BSTAGE;
                    }
                }
                // the copies in flight land before the block ends
                for (int c = acopied > OZ_ASLOTS ? acopied - OZ_ASLOTS : 0; c < acopied; ++c)
                    mbar_wait(ain0 + 8 * (c % OZ_ASLOTS), (c / OZ_ASLOTS) & 1, nullptr);
                for (int c = pq > OZ_BSLOTS ? pq - OZ_BSLOTS : 0; c < pq; ++c)
                    mbar_wait(bfull0 + 8 * (c % OZ_BSLOTS), (c / OZ_BSLOTS) & 1, nullptr);
            }
        } else {
            // ---------------- warps 12, 13: the products of the even / odd diagonals ----------------
            // The whole warp runs the loop and one elected lane issues; the decisions
            // to stop are warp-uniform, and so is, visibly to the compiler, what
            // the products' operands are made of: they are taken from uniform
            // registers, and moving each operand of each product there costs more
            // than the product takes.
            const uint32_t tm = warp_uniform(tmem), b0 = warp_uniform(bring);
            const int rend = warp_uniform(it.rend);
            const uint32_t on = elect_one();
            int q = 0, gi = 0;
            for (int g = warp_uniform(it.rbeg); g < rend && !bad; ++g, ++gi) {
                const int nk = warp_uniform(B.tg_nk[g]);
                for (int kc = 0; kc < nk; ++kc, ++q) {
                    const int sb = q % OZ_BSLOTS;
                    const bool ok = mbar_wait(afull0 + 8 * sb, (q / OZ_BSLOTS) & 1, err) &&
                                    mbar_wait(bfull0 + 8 * sb, (q / OZ_BSLOTS) & 1, err);
                    if (__any_sync(0xffffffffu, !ok)) {
                        bad = 1;
                        break;
                    }
                    tc_fence_after();
                    const uint32_t ac = tm + OZ_ACOL + (q % OZ_ASTAGES) * OZ_ACOLS, bc = b0 + sb * OZ_BSTAGE;
                    const bool open = kc == 0, close = kc == nk - 1, held = open && gi >= 1;
                    const uint32_t fpar = (gi - 1) & 1, done = done0 + 8 * sb;
                    if (warp == OZ_MMA_WARP ? oz_issue_chunk<ND, 0>(ac, bc, tm, open, held, close, accfull0, accfree0, fpar,
                                                                    done, on, err)
                                            : oz_issue_chunk<ND, 1>(ac, bc, tm, open, held, close, accfull0, accfree0, fpar,
                                                                    done, on, err)) {
                        bad = 1;
                        break;
                    }
                }
            }
            // all products of this warp have completed
            mma_commit_on(fin, on);
            mbar_wait(fin, 0u, nullptr);
        }
    }
    if (bad) atomicExch(err, 1);
    tc_fence_before();
    __syncthreads();
    if (warp == 0) {
        tc_fence_after();
        tmem_dealloc(tmem, OZ_TMEM_COLS);
    }
}

// ---------------------------------------------------------------------------
// Self-test of the fixed-point machinery: D[128 x NP] = A[128 x K] B^T (six digits),
// A, B given in FP64 (row-major, K contiguous), K a multiple of OZ_KC up to
// OZ_MAX_NK chunks; one block of 128 threads, the per-chunk, row and column
// scaling, digit slices (A in tensor memory, B in shared memory),
// descriptors, products, accumulators and exact combination of the product
// kernel.  Its waits for the products give up after `wait_cycles`; with
// `withhold` the first chunk's products are never issued, so that wait runs
// out: the block then releases its tensor memory and sets *err (the failure
// path of the product kernel, without a fault).
// ---------------------------------------------------------------------------
__global__ void __launch_bounds__(128, 1) k_oz_selftest(int K, const double *__restrict__ A,
                                                         const double *__restrict__ Bm, double *__restrict__ D,
                                                         int *__restrict__ err, long long wait_cycles,
                                                         int withhold) {
    constexpr int ND = 6;
    using F = OzK<ND>;
    constexpr int OZ_NP = F::NP;
    extern __shared__ __align__(1024) unsigned char smem[];
    uint64_t *bars = (uint64_t *) (smem + F::BSTAGE);
    uint32_t *tmem_hold = (uint32_t *) (bars + 2);
    __shared__ int fB[OZ_NP];
    const uint32_t b0 = smem_u32(smem), done = smem_u32(bars);
    const int tid = threadIdx.x, warp = tid >> 5;
    if (tid == 0) {
        mbar_init(done, 1);
        fence_mbar_init();
    }
    if (warp == 0) tmem_alloc(smem_u32(tmem_hold), OZ_TMEM_COLS);
    // row exponent of A row tid, column exponents of B rows
    double ma = 0.;
    for (int k = 0; k < K; ++k) ma = fmax(ma, fabs(A[(size_t) tid * K + k]) * oz_pow2(-oz_ek(k + 1)));
    const int gA = oz_exp_of(ma);
    if (tid < OZ_NP) {
        double mb = 0.;
        for (int k = 0; k < K; ++k) mb = fmax(mb, fabs(Bm[(size_t) tid * K + k]) * oz_pow2(oz_ek(k + 1)));
        fB[tid] = oz_exp_of(mb);
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = *tmem_hold;
    const uint32_t tlane = tmem + ((uint32_t) (warp * 32) << 16);
    unsigned char *bs = smem;
    uint32_t ph = 0;
    int bad = 0;
    for (int kc = 0; kc * OZ_KC < K && !bad; ++kc) {
        for (int hf = 0; hf < 2; ++hf) {
            uint32_t wa[ND][4], wb[ND][4];
            for (int qd = 0; qd < 4; ++qd) {
                uint32_t lo[4], hi[4], lb[4], hb[4];
                for (int u = 0; u < 4; ++u) {
                    const int k = kc * OZ_KC + hf * 16 + qd * 4 + u;
                    const int ek = oz_ek(k + 1);
                    oz_digits<ND>(A[(size_t) tid * K + k], oz_pow2(F::FRAC - ek - gA), lo[u], hi[u]);
                    const int n = tid & (OZ_NP - 1);
                    oz_digits<ND>(Bm[(size_t) n * K + k], oz_pow2(F::FRAC + ek - fB[n]), lb[u], hb[u]);
                }
                uint32_t s6[ND], t6[ND];
                oz_slices4<ND>(lo, hi, s6);
                oz_slices4<ND>(lb, hb, t6);
                for (int s = 0; s < ND; ++s) {
                    wa[s][qd] = s6[s];
                    wb[s][qd] = t6[s];
                }
            }
            for (int s = 0; s < ND; ++s)
                tmem_st4(tlane + F::ACOL + s * (OZ_KC / 4) + hf * 4, wa[s][0], wa[s][1], wa[s][2], wa[s][3]);
            if (tid < OZ_NP) {
                const uint32_t rb = (tid >> 3) * 128 + (tid & 7) * 16 + hf * F::LBO_B;
                for (int s = 0; s < ND; ++s)
                    *(uint4 *) (bs + s * F::BSLICE + rb) = make_uint4(wb[s][0], wb[s][1], wb[s][2], wb[s][3]);
            }
        }
        tmem_wait_st();
        fence_proxy_async();
        tc_fence_before();
        __syncthreads();
        if (tid == 0 && !(withhold && kc == 0)) {
            tc_fence_after();
            issue_products_i8<ND, 0, ND, 1>(tmem + F::ACOL, b0, tmem, kc == 0, 1u);
            mma_commit(done);
        }
        const int lbad = !mbar_wait_for(done, ph, err, wait_cycles);
        ph ^= 1u;
        bad = __syncthreads_or(lbad);
        tc_fence_after();
    }
    if (!bad) {
        const uint32_t trow = tmem + ((uint32_t) (warp * 32) << 16);
        for (int c = 0; c < OZ_NP; c += 16) {
            uint32_t a[ND][16];
            for (int d = 0; d < ND; ++d) tmem_ld16(trow + d * OZ_NP + c, a[d]);
            tmem_wait_ld();
            for (int i = 0; i < 16; ++i) {
                const int sh = oz_sum_shift(K / OZ_KC);
                for (int d = 0; d < ND; ++d) reg_after_wait(a[d][i]);
                long long v = ((long long) (int) a[0][i] * 65536 + (long long) (int) a[1][i] * 256 + (int) a[2][i]) << sh;
                v += ((long long) (int) a[3][i] * 256 + (int) a[4][i]) << (sh - 16);
                v += sh >= 24 ? (long long) (int) a[5][i] << (sh - 24)
                              : ((long long) (int) a[5][i] + (1 << (23 - sh))) >> (24 - sh);
                D[(size_t) tid * OZ_NP + c + i] = oz_scaled((double) v, (gA + fB[c + i] + F::CSHIFT - sh) * (1 << 20));
            }
        }
    } else if (tid == 0) {
        atomicExch(err, 1);
    }
    tc_fence_before();
    __syncthreads();
    if (warp == 0) {
        tc_fence_after();
        tmem_dealloc(tmem, OZ_TMEM_COLS);
    }
}

template <int ND, int TM, int TX>
int launch_oz(cudaStream_t s, const DevBatch &B, int nitems, const AngItem *items, const unsigned char *bop,
              double *part, int *err) {
    constexpr int smem = (int) OzK<ND>::SMEM;
    static bool attr = false;
    if (!attr) {
        LMIEB_CUDA_TRY(cudaFuncSetAttribute(k_angular_oz<ND, TM, TX>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
        attr = true;
    }
    k_angular_oz<ND, TM, TX><<<nitems, OZ_T, smem, s>>>(B, items, bop, part, err);
    LMIEB_CUDA_TRY(cudaGetLastError());
    return 0;
}

template <int ND>
int launch_oz_basis(cudaStream_t s, const DevBatch &B, int nitems, const AngItem *items, const unsigned char *bop,
                    double *part, int *err) {
    if (B.nd1 > OZ_MAX_ND1 || B.nd2 > OZ_MAX_ND2) {
        fprintf(stderr, "ERROR: lmie_b200: fixed-point angular stage built for at most %d + %d derivatives\n", OZ_MAX_ND1,
                OZ_MAX_ND2);
        return -1;
    }
    const int tx = B.t_x ? 2 : (B.oz_wl ? 1 : 0);
    if (B.t_m) {
        if (tx == 0) return launch_oz<ND, 1, 0>(s, B, nitems, items, bop, part, err);
        if (tx == 1) return launch_oz<ND, 1, 1>(s, B, nitems, items, bop, part, err);
        return launch_oz<ND, 1, 2>(s, B, nitems, items, bop, part, err);
    }
    if (tx == 0) return launch_oz<ND, 0, 0>(s, B, nitems, items, bop, part, err);
    if (tx == 1) return launch_oz<ND, 0, 1>(s, B, nitems, items, bop, part, err);
    return launch_oz<ND, 0, 2>(s, B, nitems, items, bop, part, err);
}

template <int ND>
int launch_operands(cudaStream_t s, const DevBatch &B, long long narow, const long long *arow_start,
                    signed char *rowexp, unsigned char *aop, int ngroups, const double *coef, unsigned char *bop,
                    int *colexp) {
    if (narow > 0) {
        k_oz_aop<ND><<<ceil_div(narow, 128), 128, 0, s>>>(B, narow, arow_start, rowexp, aop);
        LMIEB_CUDA_TRY(cudaGetLastError());
    }
    if (ngroups > 0) {
        k_oz_bop<ND><<<ngroups, OZ_BOP_J * Oz<ND>::NP, 0, s>>>(B, coef, bop, colexp);
        LMIEB_CUDA_TRY(cudaGetLastError());
    }
    return 0;
}

}  // namespace

int launch_oz_operands(cudaStream_t s, const DevBatch &B, int digits, long long narow, const long long *arow_start,
                       signed char *rowexp, unsigned char *aop, int ngroups, const double *coef, unsigned char *bop,
                       int *colexp) {
    return digits == 6 ? launch_operands<6>(s, B, narow, arow_start, rowexp, aop, ngroups, coef, bop, colexp)
                       : launch_operands<7>(s, B, narow, arow_start, rowexp, aop, ngroups, coef, bop, colexp);
}

int launch_angular_oz(cudaStream_t s, const DevBatch &B, int digits, int nitems, const AngItem *items,
                      const unsigned char *bop, double *part, int *err) {
    if (nitems <= 0) return 0;
    return digits == 6 ? launch_oz_basis<6>(s, B, nitems, items, bop, part, err)
                       : launch_oz_basis<7>(s, B, nitems, items, bop, part, err);
}

int launch_oz_selftest(cudaStream_t s, int K, const double *A, const double *Bm, double *D, int *err,
                       long long wait_cycles, int withhold) {
    static bool attr = false;
    const int smem = (int) (Oz<6>::BSTAGE + 64);
    if (!attr) {
        LMIEB_CUDA_TRY(cudaFuncSetAttribute(k_oz_selftest, cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
        attr = true;
    }
    k_oz_selftest<<<1, 128, smem, s>>>(K, A, Bm, D, err, wait_cycles, withhold);
    LMIEB_CUDA_TRY(cudaGetLastError());
    return 0;
}
