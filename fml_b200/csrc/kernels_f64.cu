// Plain-FP64 Gaussian and Laplacian kernel matrices by direct differences,
// the FP64 parity path of fkernels.f90:317-377.
//
// K_s[j, i] = exp(scale_s * sum_k f(A[j,k] - B[i,k])), f = square (Gaussian,
// scale = -0.5/sigma^2) or abs (Laplacian, scale = -1/sigma). Every sigma is
// emitted from one pass over the descriptors.
//
// Tiles of 64 x 64, 32 x 64 or 16 x 64 outputs per 128-thread CTA, dist_tile.cuh.
// Symmetric mode launches only the tiles on or below the diagonal and writes the
// mirror through a shared-memory transpose.
#include <math.h>

#include "common.cuh"
#include "dist_tile.cuh"

namespace fmlb {
namespace {

constexpr int BN = dist::DT_N, TPB = dist::DT_TPB, MAXSIG = 32;

// 32-row tiles of 4 x 4 pairs per thread, or 64-row ones of 4 x 8: the former leave
// finer remainders, the latter load less per pair. A call whose busiest SM gets k
// 32-row or m 64-row tiles takes about k + 0.7 or 1.87 m + 1 times 12.6 us at d = 276 (19.7
// at d = 435). us of 32-row and 64-row tiles, and of the 64 x 64 tiles with 256 threads and
// a single buffer that these replaced, symmetric, d = 276, one sigma: 635 rows 23, 38, 35;
// 1019 35, 39, 35; 1403 60, 61, 60; 1659 72, 84, 86; 1915 98, 109, 112; 2427 147, 152,
// 162; 2875 187, 179, 191; 4475 441, 415, 455. 2 x 8 pairs instead of 4 x 4 need more
// shared loads than there are cycles: 39 for 1019 rows, 70 for 1403.
bool half_tiles(long long nhalf, long long nblk) {
    const long long s = sm_count(), k = (nhalf + s - 1) / s, m = (nblk + s - 1) / s;
    return 100 * k < 187 * m + 30;
}

struct SigmaScales {
    double s[MAXSIG];
};

// RI x CJ pairs per thread. Symmetric: the tiles of the 64 x 64 blocks on or below the
// diagonal, one or (of 32 rows) two to a block; of the last row of blocks one where
// that covers its rows.
template <bool kL1, int RI, int CJ>
__global__ void __launch_bounds__(TPB, RI == 1 ? 5 : 4)
distance_kernel_f64(const double *__restrict__ A, int na, int lda, const double *__restrict__ B,
                    int nb, int ldb, int d, const __grid_constant__ SigmaScales sc, int nsig,
                    double *__restrict__ K, long long ldk, long long sstride, int symmetric) {
    // the stage and the transpose share one buffer
    constexpr int BM = dist::tile_rows<RI, CJ>(), kT = BN * (BM + 1), kPerBlock = BN / BM;
    constexpr int kStage = dist::stage_doubles<RI, CJ>();
    __shared__ double smem[RI > 1 && kT > kStage ? kT : kStage];
    double(*T)[BM + 1] = reinterpret_cast<double(*)[BM + 1]>(smem);

    int by, bx, row0;
    if (symmetric) {
        const long long nt = (na + BN - 1) / BN, above = nt * (nt - 1) / 2;
        const bool one = blockIdx.x >= kPerBlock * above && (na - 1) % BN < BM;
        const long long t = one ? blockIdx.x - (kPerBlock - 1) * above : blockIdx.x / kPerBlock;
        by = (int)((sqrt(8.0 * (double)t + 1.0) - 1.0) * 0.5);
        while ((long long)by * (by + 1) / 2 > t) --by;
        while ((long long)(by + 1) * (by + 2) / 2 <= t) ++by;
        bx = (int)(t - (long long)by * (by + 1) / 2);
        row0 = by * BN + (one ? 0 : blockIdx.x % kPerBlock) * BM;
    } else {
        bx = blockIdx.x;
        by = blockIdx.y;
        row0 = by * BM;
    }
    const int col0 = bx * BN;
    const int nr = min(BM, na - row0), nc = min(BN, nb - col0);
    double acc[RI][CJ];
    dist::dist_tile<kL1 ? dist::kAbs : dist::kSquare, RI == 1>(
        acc, smem, [&](int r) { return A + (size_t)(row0 + r) * lda; },
        [&](int c) { return B + (size_t)(col0 + c) * ldb; }, nr, nc, d);

    const int r0 = dist::first_row<RI, CJ>(), c0 = dist::first_col<CJ>();
    const bool mirror = RI > 1 && symmetric && by > bx;
    if (mirror) __syncthreads();  // the stage becomes the transpose
    for (int s = 0; s < nsig; ++s) {
        double *Ks = K + s * sstride;
        const double scale = sc.s[s];
#pragma unroll
        for (int i = 0; i < RI; ++i) {
            const int r = r0 + 4 * i;
#pragma unroll
            for (int j = 0; j < CJ; ++j) {
                const int c = c0 + 8 * j;
                const double v = exp(scale * acc[i][j]);  // before the test: several side by side
                if (r < nr && c < nc) Ks[(size_t)(row0 + r) * ldk + col0 + c] = v;
                if (mirror) T[c][r] = v;
            }
        }
        if (mirror) {
            __syncthreads();
            // T[c][r] -> K[col0 + c][row0 + r], coalesced in r
            const int r = threadIdx.x % BM, first = threadIdx.x / BM;
            double *out = Ks + (size_t)(col0 + first) * ldk + row0 + r;
            if (r < nr) {
#pragma unroll 8
                for (int c = first; c < nc; c += TPB / BM, out += (TPB / BM) * ldk) *out = T[c][r];
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
        // in 16-row tiles, where the k-loop's latency counts and not the work (379
        // rows symmetric, d = 276: 19 us, 23 in 32-row ones; 640 rows 43 and 22)
        const long long nt = ceil_div(na, BN), ntc = ceil_div(nb, BN);
        const long long nblk = symmetric ? nt * (nt + 1) / 2 : nt * ntc;
        const long long nhalf = symmetric ? 2 * nblk - ((na - 1) % BN < BN / 2 ? nt : 0)
                                          : ntc * ceil_div(na, BN / 2);
        if (4 * nt * ntc <= sm_count()) {
            const dim3 grid((unsigned)ntc, ceil_div(na, 16));
            distance_kernel_f64<kL1, 1, 8><<<grid, TPB, 0, st>>>(A, na, lda, B, nb, ldb, d, sc, ns,
                                                              Ks, ldk, sstride, 0);
        } else if (half_tiles(nhalf, nblk)) {
            const dim3 grid = symmetric ? dim3((unsigned)nhalf)
                                        : dim3((unsigned)ntc, ceil_div(na, 32));
            distance_kernel_f64<kL1, 4, 4><<<grid, TPB, 0, st>>>(A, na, lda, B, nb, ldb, d, sc, ns,
                                                              Ks, ldk, sstride, symmetric);
        } else if (symmetric) {
            FMLB_REQUIRE(nblk < (1LL << 31), "%s: too many tiles", name);
            distance_kernel_f64<kL1, 4, 8><<<(unsigned)nblk, TPB, 0, st>>>(
                A, na, lda, B, nb, ldb, d, sc, ns, Ks, ldk, sstride, 1);
        } else {
            const dim3 grid((unsigned)ntc, (unsigned)nt);
            FMLB_REQUIRE(grid.y <= 65535, "%s: na too large for one launch", name);
            distance_kernel_f64<kL1, 4, 8><<<grid, TPB, 0, st>>>(A, na, lda, B, nb, ldb, d, sc, ns,
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
