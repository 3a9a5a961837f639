// Plain-FP64 Gaussian and Laplacian kernel matrices by direct differences,
// the FP64 parity path of fkernels.f90:317-377.
//
// K_s[j, i] = exp(scale_s * sum_k f(A[j,k] - B[i,k])), f = square (Gaussian,
// scale = -0.5/sigma^2) or abs (Laplacian, scale = -1/sigma). Every sigma is
// emitted from one pass over the descriptors.
//
// Tiles of 64 x 64 outputs (32 x 64 and 16 x 64 for small problems) per 128-thread CTA,
// dist_tile.cuh. Symmetric mode launches only the tiles on or below the
// diagonal and writes the mirror through a shared-memory transpose.
#include <math.h>

#include "common.cuh"
#include "dist_tile.cuh"

namespace fmlb {
namespace {

constexpr int BN = dist::DT_N, TPB = dist::DT_TPB, MAXSIG = 32;

// Few tiles leave an SM one warp per FP64 unit, which cannot keep it busy: 16-row
// tiles up to one per SM, 32-row ones up to two 64-row tiles per SM. us on d = 276
// with 16, 32 and 64 rows: 1 x 1000 17, 23, 68; 128 x 2000 34, 26, 50; 1000 x 1000
// symmetric 97, 39, 70; 1600 symmetric 222, 85, 84; 2000 x 2000 350, 216, 179.
constexpr int kSmallTilesPerSm = 1, kHalfTilesPerSm = 2;

struct SigmaScales {
    double s[MAXSIG];
};

// Tiles of 16 RI x 64. Symmetric: the tiles of the 64 x 64 blocks on or below the
// diagonal, one or two (RI = 2) to a block.
template <bool kL1, int RI>
__global__ void __launch_bounds__(TPB, RI == 4 ? 4 : RI == 2 ? 6 : 8)
distance_kernel_f64(const double *__restrict__ A, int na, int lda, const double *__restrict__ B,
                    int nb, int ldb, int d, const __grid_constant__ SigmaScales sc, int nsig,
                    double *__restrict__ K, long long ldk, long long sstride, int symmetric) {
    // the stage and the transpose share one buffer
    constexpr int BM = 16 * RI, kT = BN * (BM + 1), kPerBlock = BN / BM;
    constexpr int kStage = dist::stage_doubles<RI>();
    __shared__ double smem[RI > 1 && kT > kStage ? kT : kStage];
    double(*T)[BM + 1] = reinterpret_cast<double(*)[BM + 1]>(smem);

    int by, bx, row0;
    if (symmetric) {
        const long long t = blockIdx.x / kPerBlock;
        by = (int)((sqrt(8.0 * (double)t + 1.0) - 1.0) * 0.5);
        while ((long long)by * (by + 1) / 2 > t) --by;
        while ((long long)(by + 1) * (by + 2) / 2 <= t) ++by;
        bx = (int)(t - (long long)by * (by + 1) / 2);
        row0 = by * BN + blockIdx.x % kPerBlock * BM;
        if (row0 >= na) return;
    } else {
        bx = blockIdx.x;
        by = blockIdx.y;
        row0 = by * BM;
    }
    const int col0 = bx * BN;
    const int nr = min(BM, na - row0), nc = min(BN, nb - col0);
    double acc[RI][8];
    dist::dist_tile<kL1 ? dist::kAbs : dist::kSquare, RI>(
        acc, smem, [&](int r) { return A + (size_t)(row0 + r) * lda; },
        [&](int c) { return B + (size_t)(col0 + c) * ldb; }, nr, nc, d);

    const int r0 = dist::first_row<RI>(), c0 = dist::first_col();
    const bool mirror = RI > 1 && symmetric && by > bx;
    if (mirror) __syncthreads();  // the stage becomes the transpose
    for (int s = 0; s < nsig; ++s) {
        double *Ks = K + s * sstride;
        const double scale = sc.s[s];
#pragma unroll
        for (int i = 0; i < RI; ++i) {
            const int r = r0 + 4 * i;
#pragma unroll
            for (int j = 0; j < 8; ++j) {
                const int c = c0 + 8 * j;
                if (r < nr && c < nc) {
                    const double v = exp(scale * acc[i][j]);
                    Ks[(size_t)(row0 + r) * ldk + col0 + c] = v;
                    if (mirror) T[c][r] = v;
                }
            }
        }
        if (mirror) {
            __syncthreads();
            // T[c][r] -> K[col0 + c][row0 + r], coalesced in r
            for (int t = threadIdx.x; t < BN * BM; t += TPB) {
                const int c = t / BM, r = t % BM;
                if (c < nc && r < nr) Ks[(size_t)(col0 + c) * ldk + row0 + r] = T[c][r];
            }
            __syncthreads();
        }
    }
}

template <bool kL1>
int launch_distance(const double *A, int na, int lda, const double *B, int nb, int ldb, int d,
                    const double *sigmas, int nsigma, double *K, long long ldk, long long sstride,
                    int symmetric, cudaStream_t st, const char *name) {
    FMLB_REQUIRE(na >= 0 && nb >= 0 && d >= 1, "%s: bad sizes na=%d nb=%d d=%d", name, na, nb, d);
    FMLB_REQUIRE(lda >= d && ldb >= d, "%s: leading dimension < d", name);
    FMLB_REQUIRE(ldk >= nb, "%s: ldk < nb", name);
    FMLB_REQUIRE(nsigma >= 1 && sigmas, "%s: need at least one sigma", name);
    FMLB_REQUIRE(nsigma == 1 || sstride >= (long long)na * ldk || sstride <= -(long long)na * ldk,
                 "%s: sigma_stride overlaps matrices", name);
    if (symmetric) FMLB_REQUIRE(A == B && na == nb && lda == ldb, "%s: symmetric needs A == B", name);
    if (na == 0 || nb == 0) return FMLB_OK;
    for (int s0 = 0; s0 < nsigma; s0 += MAXSIG) {
        const int ns = nsigma - s0 < MAXSIG ? nsigma - s0 : MAXSIG;
        SigmaScales sc;
        for (int s = 0; s < ns; ++s) {
            const double sg = sigmas[s0 + s];
            sc.s[s] = kL1 ? -1.0 / sg : -0.5 / (sg * sg);  // fkernels.f90:334 / :367
        }
        double *Ks = K + s0 * sstride;
        // only the tiles on or below the diagonal where symmetric; the whole matrix
        // in 16-row tiles, where the k-loop's latency counts and not the work
        const long long nt = ceil_div(na, BN), ntc = ceil_div(nb, BN);
        const long long nblk = symmetric ? nt * (nt + 1) / 2 : nt * ntc;
        if (4 * nt * ntc <= kSmallTilesPerSm * sm_count()) {
            const dim3 grid((unsigned)ntc, ceil_div(na, 16));
            distance_kernel_f64<kL1, 1><<<grid, TPB, 0, st>>>(A, na, lda, B, nb, ldb, d, sc, ns,
                                                              Ks, ldk, sstride, 0);
        } else if (nblk <= kHalfTilesPerSm * sm_count()) {
            const dim3 grid = symmetric ? dim3((unsigned)(2 * nblk))
                                        : dim3((unsigned)ntc, ceil_div(na, 32));
            distance_kernel_f64<kL1, 2><<<grid, TPB, 0, st>>>(A, na, lda, B, nb, ldb, d, sc, ns,
                                                              Ks, ldk, sstride, symmetric);
        } else if (symmetric) {
            FMLB_REQUIRE(nblk < (1LL << 31), "%s: too many tiles", name);
            distance_kernel_f64<kL1, 4><<<(unsigned)nblk, TPB, 0, st>>>(
                A, na, lda, B, nb, ldb, d, sc, ns, Ks, ldk, sstride, 1);
        } else {
            const dim3 grid((unsigned)ntc, (unsigned)nt);
            FMLB_REQUIRE(grid.y <= 65535, "%s: na too large for one launch", name);
            distance_kernel_f64<kL1, 4><<<grid, TPB, 0, st>>>(A, na, lda, B, nb, ldb, d, sc, ns,
                                                              Ks, ldk, sstride, 0);
        }
        FMLB_TRY(launch_status(name));
    }
    return FMLB_OK;
}

}  // namespace
}  // namespace fmlb

extern "C" int fmlb_gaussian_kernel_f64(const double *A, int na, int lda, const double *B, int nb,
                                        int ldb, int d, const double *sigmas_host, int nsigma,
                                        double *K, long long ldk, long long sigma_stride,
                                        int symmetric, void *stream) {
    return fmlb::launch_distance<false>(A, na, lda, B, nb, ldb, d, sigmas_host, nsigma, K, ldk,
                                        sigma_stride, symmetric, FMLB_STREAM(stream),
                                        "fmlb_gaussian_kernel_f64");
}

extern "C" int fmlb_laplacian_kernel_f64(const double *A, int na, int lda, const double *B, int nb,
                                         int ldb, int d, const double *sigmas_host, int nsigma,
                                         double *K, long long ldk, long long sigma_stride,
                                         int symmetric, void *stream) {
    return fmlb::launch_distance<true>(A, na, lda, B, nb, ldb, d, sigmas_host, nsigma, K, ldk,
                                       sigma_stride, symmetric, FMLB_STREAM(stream),
                                       "fmlb_laplacian_kernel_f64");
}
