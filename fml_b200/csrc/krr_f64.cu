// KRR helpers on the FP64 path:
//   * fmlb_add_diagonal_f64: A[i, i] += lambda (the user-side K + lambda*I);
//   * fmlb_kernel_predict_f64: y_s[q] = sum_t k_s(Xq[q], Xt[t]) alpha_s[t] for
//     every sigma, with the kernel matrix never written to memory (the user-side
//     prediction K_test @ alpha, fused; reference pattern fget_prediction,
//     fml/kernels/fkernels.f90:480-539);
//   * fmlb_gemv_f64: y = M x for a stored kernel matrix (the user-side
//     K_test @ alpha when the test kernel was built separately, e.g. ARAD).
// The prediction is split over the training set into fixed chunks whose
// partial sums are reduced in a second pass in a fixed order (deterministic).
// A chunk is worked by a cluster of eight CTAs, 128 training points each, whose
// sums meet in distributed shared memory: with one CTA per chunk, 1000 queries
// against 1000 training points ran on 16 of the SMs (600 us, now 75).
#include <cooperative_groups.h>
#include <limits.h>
#include <math.h>

#include <algorithm>

#include "common.cuh"
#include "dist_tile.cuh"

namespace fmlb {
namespace {

constexpr int BN = dist::DT_N, TPB = dist::DT_TPB, MAXSIG = 8;
constexpr int CHUNK = 1024;  // training points per split
constexpr int PARTS = 8, PART = CHUNK / PARTS;  // CTAs of a cluster, training points of each

struct Scales {
    double s[MAXSIG];
};

__global__ void add_diagonal_kernel(double *A, long long lda, int n, double lam) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) A[(size_t)i * lda + i] += lam;
}

// 16 RI queries x CHUNK training points per cluster. A query's sums are formed
// in the same order whatever RI and the queries beside it are.
template <bool kL1, int RI>
__global__ void __cluster_dims__(1, 1, PARTS) __launch_bounds__(TPB, RI == 4 ? 4 : RI == 2 ? 6 : 5)
predict_partial_kernel(const double *__restrict__ Q, int nq, int ldq, const double *__restrict__ T,
                       int nt, int ldt, int d, const __grid_constant__ Scales sc, int nsig,
                       const double *__restrict__ alpha, long long lda_alpha,
                       double *__restrict__ partial) {
    constexpr int BM = 16 * RI;
    __shared__ double stage[dist::stage_doubles<RI, 8>()];
    __shared__ double red[MAXSIG][BM];
    const int row0 = blockIdx.x * BM, nr = min(BM, nq - row0);
    const int split = blockIdx.y;
    const int t_begin = split * CHUNK + blockIdx.z * PART, t_end = min(nt, t_begin + PART);
    const int r0 = dist::first_row<RI, 8>(), c0 = dist::first_col<8>();
    for (int t = threadIdx.x; t < nsig * BM; t += TPB) red[t / BM][t % BM] = 0.0;
    // (the first barrier inside dist_tile orders these before their use)
    for (int col0 = t_begin; col0 < t_end; col0 += BN) {
        const int nc = min(BN, t_end - col0);
        double acc[RI][8];
        dist::dist_tile<kL1 ? dist::kAbs : dist::kSquare, true>(
            acc, stage, [&](int r) { return Q + (size_t)(row0 + r) * ldq; },
            [&](int c) { return T + (size_t)(col0 + c) * ldt; }, nr, nc, d);
        for (int s = 0; s < nsig; ++s) {
            const double scale = sc.s[s];
            double v[RI];
#pragma unroll
            for (int i = 0; i < RI; ++i) v[i] = 0.0;
#pragma unroll
            for (int j = 0; j < 8; ++j) {
                const int c = c0 + 8 * j;
                if (c < nc) {
                    const double a = alpha[s * lda_alpha + col0 + c];
#pragma unroll
                    for (int i = 0; i < RI; ++i) v[i] = fma(exp(scale * acc[i][j]), a, v[i]);
                }
            }
#pragma unroll
            for (int i = 0; i < RI; ++i) {  // over the 8 lanes of a row, in a fixed order
#pragma unroll
                for (int o = 4; o; o >>= 1) v[i] += __shfl_xor_sync(0xffffffffu, v[i], o);
                if (c0 == 0) red[s][r0 + 4 * i] += v[i];
            }
        }
    }
    cooperative_groups::cluster_group cluster = cooperative_groups::this_cluster();
    cluster.sync();
    if (blockIdx.z == 0) {
        for (int t = threadIdx.x; t < nsig * BM; t += TPB) {
            const int s = t / BM, r = t % BM;
            if (r < nr) {
                double v = 0.0;
                for (int p = 0; p < PARTS; ++p) v += *cluster.map_shared_rank(&red[s][r], p);
                partial[((size_t)split * nsig + s) * nq + row0 + r] = v;
            }
        }
    }
    cluster.sync();  // no CTA leaves while its sums are read
}

// The partial sums of every chunk, in tiles of 16, 32 or 64 queries by the number
// of CTAs that the largest would give. us for 16, 32, 64 queries, d = 276: 200 x 1000
// 41, 52, 70; 500 x 1000 64, 71, 70; 1000 x 1000 114, 76, 113; 2000 x 1000 213, 134,
// 117; 1000 x 2000 214, 134, 117; 2000 x 2000 392, 249, 211.
int launch_predict_partial(int kind, const double *Xq, int nq, int ldq, const double *Xt, int nt,
                           int ldt, int d, const Scales &sc, int nsigma, const double *alpha,
                           long long lda_alpha, double *partial, cudaStream_t st) {
    const int nsplit = ceil_div(nt, CHUNK);
    const long long tiles = (long long)ceil_div(nq, 64) * ceil_div(nt, PART);
    const int ri = 2 * tiles <= sm_count() ? 1 : 2 * tiles <= 3 * sm_count() ? 2 : 4;
    const dim3 grid(ceil_div(nq, 16 * ri), nsplit, PARTS);
#define FMLB_PREDICT(L1, RI)                                                                   \
    predict_partial_kernel<L1, RI><<<grid, TPB, 0, st>>>(Xq, nq, ldq, Xt, nt, ldt, d, sc,     \
                                                         nsigma, alpha, lda_alpha, partial)
    if (kind == 0) {
        if (ri == 1) FMLB_PREDICT(false, 1);
        else if (ri == 2) FMLB_PREDICT(false, 2);
        else FMLB_PREDICT(false, 4);
    } else {
        if (ri == 1) FMLB_PREDICT(true, 1);
        else if (ri == 2) FMLB_PREDICT(true, 2);
        else FMLB_PREDICT(true, 4);
    }
#undef FMLB_PREDICT
    return launch_status("predict_partial_kernel");
}

__global__ void reduce_splits_kernel(const double *__restrict__ partial, int nsplit, int nsig,
                                     int nq, double *__restrict__ y, long long ldy) {
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= nsig * nq) return;
    const int s = t / nq, q = t % nq;
    double v = 0.0;
    for (int p = 0; p < nsplit; ++p) v += partial[((size_t)p * nsig + s) * nq + q];
    y[s * ldy + q] = v;
}

// one warp per row, lanes stride the columns, fixed shuffle tree (deterministic)
__global__ void gemv_rows_kernel(const double *__restrict__ M, long long ldm, int rows, int cols,
                                 const double *__restrict__ x, double *__restrict__ y) {
    const int warp = (int)((blockIdx.x * (size_t)blockDim.x + threadIdx.x) >> 5);
    const int lane = threadIdx.x & 31;
    if (warp >= rows) return;
    const double *m = M + (size_t)warp * ldm;
    double v = 0.0;
    for (int t = lane; t < cols; t += 32) v = fma(m[t], x[t], v);
#pragma unroll
    for (int o = 16; o; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    if (lane == 0) y[warp] = v;
}

}  // namespace
}  // namespace fmlb

extern "C" int fmlb_gemv_f64(const double *M, long long ldm, int rows, int cols, const double *x,
                             double *y, void *stream) {
    using namespace fmlb;
    FMLB_REQUIRE(rows >= 0 && cols >= 0 && ldm >= cols, "fmlb_gemv_f64: bad sizes");
    if (rows == 0) return FMLB_OK;
    FMLB_REQUIRE(M && x && y, "fmlb_gemv_f64: null pointer");
    gemv_rows_kernel<<<ceil_div(rows, 8), 256, 0, FMLB_STREAM(stream)>>>(M, ldm, rows, cols, x, y);
    return launch_status("gemv_rows_kernel");
}

extern "C" int fmlb_add_diagonal_f64(double *A, long long lda, int n, double lam, void *stream) {
    using namespace fmlb;
    FMLB_REQUIRE(n >= 0 && lda >= n, "fmlb_add_diagonal_f64: bad sizes");
    if (n == 0) return FMLB_OK;
    add_diagonal_kernel<<<ceil_div(n, 256), 256, 0, FMLB_STREAM(stream)>>>(A, lda, n, lam);
    return launch_status("add_diagonal_kernel");
}

extern "C" size_t fmlb_kernel_predict_workspace_bytes(int nq, int nt, int nsigma) {
    if (nq <= 0 || nt <= 0 || nsigma <= 0) return 256;
    const size_t nsplit = (size_t)(nt + fmlb::CHUNK - 1) / fmlb::CHUNK;
    return nsplit * nsigma * nq * sizeof(double);
}

extern "C" int fmlb_kernel_predict_f64(int kind, const double *Xq, int nq, int ldq,
                                       const double *Xt, int nt, int ldt, int d,
                                       const double *sigmas_host, int nsigma, const double *alpha,
                                       long long lda_alpha, double *y, long long ldy,
                                       void *workspace, size_t ws_bytes, void *stream) {
    using namespace fmlb;
    cudaStream_t st = FMLB_STREAM(stream);
    FMLB_REQUIRE(kind == 0 || kind == 1, "fmlb_kernel_predict_f64: kind must be 0 (gaussian) "
                                         "or 1 (laplacian)");
    FMLB_REQUIRE(nq >= 0 && nt >= 0 && d >= 1 && ldq >= d && ldt >= d,
                 "fmlb_kernel_predict_f64: bad sizes");
    FMLB_REQUIRE(nsigma >= 1 && nsigma <= MAXSIG && sigmas_host,
                 "fmlb_kernel_predict_f64: nsigma must be 1..%d", MAXSIG);
    FMLB_REQUIRE(lda_alpha >= nt && ldy >= nq, "fmlb_kernel_predict_f64: bad alpha / y stride");
    FMLB_REQUIRE((long long)nsigma * nq < INT_MAX,
                 "fmlb_kernel_predict_f64: nsigma * nq = %lld must stay below 2^31",
                 (long long)nsigma * nq);
    if (nq == 0) return FMLB_OK;
    if (nt == 0) {
        for (int s = 0; s < nsigma; ++s)
            FMLB_TRY(cuda_status(cudaMemsetAsync(y + s * ldy, 0, sizeof(double) * nq, st),
                                 "fmlb_kernel_predict_f64: memset"));
        return FMLB_OK;
    }
    const size_t need = fmlb_kernel_predict_workspace_bytes(nq, nt, nsigma);
    if (ws_bytes < need || !workspace) {
        set_error("fmlb_kernel_predict_f64: workspace %zu < %zu bytes", ws_bytes, need);
        return FMLB_ENOMEM;
    }
    Scales sc;
    for (int s = 0; s < nsigma; ++s) {
        const double sg = sigmas_host[s];
        sc.s[s] = kind == 1 ? -1.0 / sg : -0.5 / (sg * sg);
    }
    const int nsplit = ceil_div(nt, CHUNK);
    double *partial = static_cast<double *>(workspace);
    FMLB_REQUIRE(nsplit <= 65535, "fmlb_kernel_predict_f64: training set too large");
    FMLB_TRY(launch_predict_partial(kind, Xq, nq, ldq, Xt, nt, ldt, d, sc, nsigma, alpha,
                                    lda_alpha, partial, st));
    reduce_splits_kernel<<<ceil_div((long)nsigma * nq, 256), 256, 0, st>>>(partial, nsplit, nsigma,
                                                                          nq, y, ldy);
    return launch_status("reduce_splits_kernel");
}

// ---------------------------------------------------------------------------
// Allocation-free prediction.
//
// Some callers cannot allocate device memory on the call path: an inference
// server whose memory is reserved up front by its own arena, a host library
// that receives only its input and output buffers from a framework that owns
// all device allocations, or code that must not reach cudaMalloc's implicit
// synchronisation. For them this variant keeps its split partial sums in the
// file-scope array below instead of a caller-provided workspace. The array is
// part of the module image: every GPU that loads the library holds it
// (8 MiB) until the process exits.
//
// The array's name in host code is only a host-side stand-in, so its device
// address is looked up once per device with cudaGetSymbolAddress, with that
// device current, on the first call made on that device. Make that first call
// before any stream capture. All calls share the array; a call fully
// overwrites the part it reads, so nothing needs clearing between calls, but
// calls that overlap on the GPU (different streams, or host threads) race on
// it and must be serialised by the caller. The looked-up address is cached per
// device for the life of the process: it does not survive cudaDeviceReset
// (after which the module may load at another address), so a process that
// resets a device must not call this entry point on it again.
// ---------------------------------------------------------------------------
#include <mutex>

namespace fmlb {
namespace {

constexpr size_t kNoAllocScratchDoubles = (size_t)1 << 20;  // 8 MiB
__device__ __align__(256) double g_predict_scratch[kNoAllocScratchDoubles];

constexpr int kMaxDevices = 64;
double *g_scratch_ptr[kMaxDevices] = {nullptr};
std::mutex g_scratch_mutex;

int noalloc_scratch(double **out) {
    int dev = 0;
    FMLB_TRY(cuda_status(cudaGetDevice(&dev), "fmlb_kernel_predict_f64_noalloc: cudaGetDevice"));
    FMLB_REQUIRE(dev >= 0 && dev < kMaxDevices,
                 "fmlb_kernel_predict_f64_noalloc: device %d out of range", dev);
    std::lock_guard<std::mutex> lock(g_scratch_mutex);
    if (!g_scratch_ptr[dev]) {
        void *p = nullptr;
        FMLB_TRY(cuda_status(cudaGetSymbolAddress(&p, g_predict_scratch),
                             "fmlb_kernel_predict_f64_noalloc: cudaGetSymbolAddress"));
        g_scratch_ptr[dev] = static_cast<double *>(p);
    }
    *out = g_scratch_ptr[dev];
    return FMLB_OK;
}

}  // namespace
}  // namespace fmlb

extern "C" int fmlb_kernel_predict_f64_noalloc(int kind, const double *Xq, int nq, int ldq,
                                               const double *Xt, int nt, int ldt, int d,
                                               const double *sigmas_host, int nsigma,
                                               const double *alpha, long long lda_alpha,
                                               double *y, long long ldy, void *stream) {
    using namespace fmlb;
    cudaStream_t st = FMLB_STREAM(stream);
    FMLB_REQUIRE(kind == 0 || kind == 1, "fmlb_kernel_predict_f64_noalloc: kind must be 0 "
                                         "(gaussian) or 1 (laplacian)");
    FMLB_REQUIRE(nq >= 0 && nt >= 0 && d >= 1 && ldq >= d && ldt >= d,
                 "fmlb_kernel_predict_f64_noalloc: bad sizes");
    FMLB_REQUIRE(nsigma >= 1 && nsigma <= MAXSIG && sigmas_host,
                 "fmlb_kernel_predict_f64_noalloc: nsigma must be 1..%d", MAXSIG);
    FMLB_REQUIRE(lda_alpha >= nt && ldy >= nq,
                 "fmlb_kernel_predict_f64_noalloc: bad alpha / y stride");
    if (nq == 0) return FMLB_OK;
    if (nt == 0) {
        for (int s = 0; s < nsigma; ++s)
            FMLB_TRY(cuda_status(cudaMemsetAsync(y + s * ldy, 0, sizeof(double) * nq, st),
                                 "fmlb_kernel_predict_f64_noalloc: memset"));
        return FMLB_OK;
    }
    const int nsplit = ceil_div(nt, CHUNK);
    const size_t need = (size_t)nsplit * nsigma * nq;
    FMLB_REQUIRE(need <= kNoAllocScratchDoubles,
                 "fmlb_kernel_predict_f64_noalloc: ceil(nt/%d) * nsigma * nq = %zu exceeds the "
                 "fixed scratch of %zu doubles (8 MiB); split the queries or use "
                 "fmlb_kernel_predict_f64 with a workspace",
                 CHUNK, need, kNoAllocScratchDoubles);
    double *partial = nullptr;
    FMLB_TRY(noalloc_scratch(&partial));
    Scales sc;
    for (int s = 0; s < nsigma; ++s) {
        const double sg = sigmas_host[s];
        sc.s[s] = kind == 1 ? -1.0 / sg : -0.5 / (sg * sg);
    }
    FMLB_REQUIRE(nsplit <= 65535, "fmlb_kernel_predict_f64_noalloc: training set too large");
    FMLB_TRY(launch_predict_partial(kind, Xq, nq, ldq, Xt, nt, ldt, d, sc, nsigma, alpha,
                                    lda_alpha, partial, st));
    reduce_splits_kernel<<<ceil_div((long)nsigma * nq, 256), 256, 0, st>>>(partial, nsplit, nsigma,
                                                                          nq, y, ldy);
    return launch_status("reduce_splits_kernel");
}
