// k_noalloc.cu -- per-radius cross sections with no device allocation.
//
// Some callers of this library cannot call cudaMalloc: a radiative-transfer
// model embedded in a host application whose memory pool has already claimed
// the whole GPU, or a retrieval loop that must not pay cudaMalloc's implicit
// device-wide synchronisation on every call.  They own their input and output
// buffers and need the Mie work done without the library touching the
// allocator.  lmie_cross_sections_noalloc serves them: it runs the recurrences
// and formulas of the drop-in solve (mie_radius.cuh; value only, no
// derivatives) with a block per radius, whose scratch is the block's shared
// memory, and takes the truncation orders as a kernel argument: no device
// memory of the library's, and calls that overlap share nothing.
//
// Limits: at most NA_MAX_RADII = 1024 radii per call and size parameters
// 0 < x = 2 pi r / lambda <= NA_MAX_X = 900 (so n1(x) < NA_MAX_ORDER = 1024).
//
// The truncation orders n1, n2 of every radius (reference
// src/lmie_core.c:18-38) are computed on the host with the host's libm, as
// everywhere else in this library: the device's pow may differ from the host's
// in the last place and move an (int) cast across an integer.
#include <cmath>
#include <cstdio>

#include "dev_common.cuh"
#include "mie_radius.cuh"
#include "../../include/lmie_b200.h"

extern "C" int lmieb_calc_n1(double x);
extern "C" int lmieb_calc_n2(int n1, double zr, double zi);

namespace {

constexpr int NA_MAX_RADII = 1024;
constexpr int NA_MAX_ORDER = 1024;
constexpr double NA_MAX_X = 900.;

// (n1, n2) of every radius of the call; n1 = 0: out of range
struct Trunc {
    int2 n[NA_MAX_RADII];
};
static_assert(mie_block_smem(mie_block_rows(NA_MAX_ORDER), false, false) <= 48 * 1024, "shared memory of a block");

// Bound by FP64 latency: the three chains of the largest radius (n1 dependent
// pairs of FMAs), then n1 / 128 rounds of orders.  1000 radii up to x = 880: 45 us, the
// whole call: 110 us (a thread per radius with D and psi in device memory: 1770).
__global__ void __launch_bounds__(MIE_BLOCK_T) k_cross_sections(int n, const double *__restrict__ radius,
                                                                double lambda, cplx m, cplx minv, int rows,
                                                                const __grid_constant__ Trunc trunc,
                                                                double *__restrict__ out) {
    extern __shared__ __align__(16) unsigned char smem[];
    const int i = blockIdx.x;
    const int2 nn = trunc.n[i];
    if (nn.x < 1) {
        // out of range: write NaN (the host reports it)
        if (threadIdx.x < 4) out[(size_t) threadIdx.x * n + i] = __longlong_as_double(0x7ff8000000000000LL);
        return;
    }
    mie_block<false, false, MIE_BLOCK_T>(
        smem, rows, false, 1,
        [&](MieRadius<false> &c) { c.set_m(m, minv, mk(0., 0.)); },
        [&](int, MieRadius<false> &c, int &n1, int &n2) {
            c.set_x(2. * LMIEB_PI * radius[i] / lambda, 0.);
            n1 = nn.x;
            n2 = nn.y;
        },
        [](int n, double &f3, double &f4) {
            f3 = (double) (n - 1) * (n + 1) / n;
            f4 = n >= 2 ? (2. * n - 1.) / ((double) n * (n - 1)) : 0.;
        },
        [](int) {}, [](int, const MieAB &) {},
        [&](const MieSums<false, false> &sums) {
            if (threadIdx.x == 0) {
                const double lam2 = lambda * lambda / (2. * LMIEB_PI);
                out[i] = sums.v[0] * lam2;
                out[(size_t) n + i] = sums.v[1] * lam2;
                out[(size_t) 2 * n + i] = norm2(mk(sums.v[2], sums.v[3])) * lam2 / (2. * 4. * LMIEB_PI);
                out[(size_t) 3 * n + i] = sums.v[4] / sums.v[1] * 2.;
            }
        });
}

}  // namespace

extern "C" int lmie_cross_sections_noalloc(int n_radii, const double *radius, double lambda, double mr,
                                           double mi, double *out, void *stream) {
    if (n_radii < 1 || n_radii > NA_MAX_RADII) {
        fprintf(stderr, "ERROR: lmie_cross_sections_noalloc: n_radii = %d, must be in 1..%d\n", n_radii,
                NA_MAX_RADII);
        return -1;
    }
    if (!radius || !out) {
        fprintf(stderr, "ERROR: lmie_cross_sections_noalloc: radius and out must be device pointers\n");
        return -1;
    }
    if (!(lambda > 0.)) {
        fprintf(stderr, "ERROR: lmie_cross_sections_noalloc: lambda = %g must be positive\n", lambda);
        return -1;
    }
    cudaStream_t s = (cudaStream_t) stream;
    const cplx m = mk(mr, -mi);
    // truncation orders on the host (host libm): the radii come down to this
    // thread's stack, n1 and n2 go up with the launch
    double rad[NA_MAX_RADII];
    Trunc trunc;
    LMIEB_CUDA_TRY(cudaMemcpyAsync(rad, radius, sizeof(double) * n_radii, cudaMemcpyDeviceToHost, s));
    LMIEB_CUDA_TRY(cudaStreamSynchronize(s));
    int bad = 0, n1max = 1;
    for (int i = 0; i < n_radii; ++i) {
        const double x = 2. * LMIEB_PI * rad[i] / lambda;
        int n1 = 0, n2 = 0;
        if (x > 0. && x <= NA_MAX_X) {
            n1 = lmieb_calc_n1(x);
            n2 = lmieb_calc_n2(n1, mr * x, -mi * x);
        }
        if (n1 < 1 || n1 >= NA_MAX_ORDER || n2 < n1) {
            n1 = 0;
            bad = i + 1;
        }
        trunc.n[i] = make_int2(n1, n2);
        n1max = n1 > n1max ? n1 : n1max;
    }
    const int rows = mie_block_rows(n1max);
    k_cross_sections<<<n_radii, MIE_BLOCK_T, mie_block_smem(rows, false, false), s>>>(n_radii, radius, lambda, m, 1. / m, rows,
                                                                               trunc, out);
    LMIEB_CUDA_TRY(cudaGetLastError());
    LMIEB_CUDA_TRY(cudaStreamSynchronize(s));
    if (bad) {
        fprintf(stderr, "ERROR: lmie_cross_sections_noalloc: radius %d gives a size parameter outside "
                "(0, %g] (lambda = %g)\n", bad - 1, NA_MAX_X, lambda);
        return -1;
    }
    return 0;
}
