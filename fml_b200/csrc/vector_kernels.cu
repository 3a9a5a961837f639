// Atomic vector kernels over per-atom descriptors (local / atomic Coulomb
// matrices):
//
//   K[k, i, j] = sum_{ia < n1[i], ja < n2[j]} exp(c_k * d(x1[i, ia], x2[j, ja]))
//
//   Gaussian  (fkernels.f90:106-162): d = sum_f (a_f - b_f)^2, c_k = -0.5 / sigma_k^2
//   Laplacian (fkernels.f90:23-104):  d = sum_f |a_f - b_f|,   c_k = -1 / sigma_k
//
// Layout: X (nm, amax, d) row-major FP64 (molecule, atom, feature); K
// (nsig, nm1, nm2) row-major, the reference's kernels(k, i, j) order.
//
// A CTA takes a group of molecules of each side. Their atoms, packed into one
// row and one column list, form a dense block that is worked through in 64 x 64
// distance tiles (dist_tile.cuh). A tile's distances go to shared memory, each
// row is summed over the columns of one molecule and these sums over the rows
// of one molecule, in a fixed order, so the result does not depend on
// scheduling. (Small sets of short descriptors: vector_pair_kernel.)
//
// Bound by FP64 issue: subtract, multiply, add per feature and atom pair, as
// the reference rounds them (a contracted FMA moves kernels of 1e-100 by more
// than the 1e-13 they agree with it to). A CTA per molecule pair with one atom
// pair per thread and load pair was bound by shared memory (300 x 401 molecules
// of up to 23 atoms, d = 276, 3 sigmas: 6.27 ms, now 2.17 ms).
#include <math.h>

#include <algorithm>

#include "common.cuh"
#include "dist_tile.cuh"
#include "fmlb.h"

namespace fmlb {
namespace {

constexpr int VK_TPB = dist::DT_TPB;
constexpr int VK_T = dist::DT_N;      // tile rows and columns
constexpr int VK_P = VK_T + 1;        // row pitch of the distance tile
constexpr int VK_MAX_GROUP = 8;
constexpr int VK_ROWS = 160;   // atoms of a group: group size x amax stays below, or one molecule
constexpr int VK_MAX_ATOMS = 128;
constexpr int VK_MAX_SIGMAS = 32;

struct Coefs {
    double c[VK_MAX_SIGMAS];
};

struct VkSide {
    const double *X;
    const int *N, *O;  // atoms per molecule, or (packed) the molecules' first rows
    int nm, amax, group;
};

// Atoms of molecule m and its first row in X.
__device__ __forceinline__ int vk_molecule(const VkSide &s, int m, long long &first, int *status) {
    int n = s.O ? s.O[m + 1] - s.O[m] : s.N[m];
    first = s.O ? s.O[m] : (long long)m * s.amax;  // 2^24 molecules x 128 atoms pass 32 bits
    if (n < 0 || n > s.amax) {  // rejected on the host as well
        if (status) atomicCAS(status, 0, 1);
        n = min(max(n, 0), s.amax);
    }
    return n;
}

// Atom list of molecules [m0, m0 + group): seg[q] = first list entry of
// molecule m0 + q, row[] = its rows in X. One whole warp.
__device__ __forceinline__ void vk_list(const VkSide &s, int m0, int *seg, long long *row,
                                        int *status) {
    const int lane = threadIdx.x & 31;
    int n = 0;
    long long first = 0;
    if (lane < s.group && m0 + lane < s.nm) n = vk_molecule(s, m0 + lane, first, status);
    int incl = n;
    for (int d = 1; d <= VK_MAX_GROUP; d <<= 1) {
        const int o = __shfl_up_sync(0xffffffffu, incl, d);
        if (lane >= d) incl += o;
    }
    if (lane <= s.group) seg[lane] = incl - n;
    for (int q = 0; q < s.group; ++q) {
        const int nq = __shfl_sync(0xffffffffu, n, q);
        const long long f = __shfl_sync(0xffffffffu, first, q);
        const int at = __shfl_sync(0xffffffffu, incl - n, q);
        for (int a = lane; a < nq; a += 32) row[at + a] = f + a;
    }
}

// Sum of f(x), beg <= x < end, in four interleaved partial sums: a quarter of the
// roundings one after the other (mean relative error of a kernel of up to 23 x 23 atoms
// 4.9e-17, 8.2e-17 with one sum), and four exponentials side by side.
template <typename F>
__device__ __forceinline__ double sum4(int beg, int end, F f) {
    double s[4] = {0.0, 0.0, 0.0, 0.0};
    int x = beg;
    for (; x + 3 < end; x += 4)
#pragma unroll
        for (int i = 0; i < 4; ++i) s[i] += f(x + i);
#pragma unroll
    for (int i = 0; i < 3; ++i)
        if (x + i < end) s[i] += f(x + i);
    return (s[0] + s[1]) + (s[2] + s[3]);
}

// Packed mode (O set): molecule m's atoms are rows O[m] .. O[m+1] of a
// (total_atoms, d) matrix; amax then bounds the counts only.
template <int KIND>
__global__ void __launch_bounds__(VK_TPB, 4)
vector_kernels_kernel(const VkSide s1, const VkSide s2, int d, const __grid_constant__ Coefs coef,
                      int nsig, double *__restrict__ K, int *__restrict__ status) {
    extern __shared__ double ksum[];  // [nsig][group1][group2]
    __shared__ double stage[dist::stage_doubles<4, 8>()];  // features, then the distance tile
    __shared__ double part[VK_T][VK_MAX_GROUP + 1];
    __shared__ int seg1[VK_MAX_GROUP + 1], seg2[VK_MAX_GROUP + 1];
    __shared__ long long row1[VK_ROWS], row2[VK_ROWS];
    static_assert(VK_T * VK_P <= dist::stage_doubles<4, 8>(), "the tile fits");
    double(*D)[VK_P] = reinterpret_cast<double(*)[VK_P]>(stage);
    const int tid = threadIdx.x, warp = tid >> 5;
    const int nb2 = (s2.nm - 1) / s2.group + 1;
    const int m1 = (int)(blockIdx.x / nb2) * s1.group, m2 = (int)(blockIdx.x % nb2) * s2.group;
    const int g12 = s1.group * s2.group;
    if (warp == 0) vk_list(s1, m1, seg1, row1, status);
    if (warp == 1) vk_list(s2, m2, seg2, row2, status);
    for (int t = tid; t < nsig * g12; t += VK_TPB) ksum[t] = 0.0;
    __syncthreads();
    const int R1 = seg1[s1.group], R2 = seg2[s2.group];
    const int tr = dist::first_row<4, 8>(), tc = dist::first_col<8>();

    for (int r0 = 0; r0 < R1; r0 += VK_T) {
        for (int c0 = 0; c0 < R2; c0 += VK_T) {
            const int nr = min(VK_T, R1 - r0), nc = min(VK_T, R2 - c0);
            double acc[4][8];
            dist::dist_tile<KIND == 0 ? dist::kSquareUnfused : dist::kAbs, true>(
                acc, stage, [&](int r) { return s1.X + row1[r0 + r] * d; },
                [&](int c) { return s2.X + row2[c0 + c] * d; }, nr, nc, d);
            __syncthreads();  // the stage becomes the distance tile
#pragma unroll
            for (int i = 0; i < 4; ++i)
#pragma unroll
                for (int j = 0; j < 8; ++j) D[tr + 4 * i][tc + 8 * j] = acc[i][j];
            __syncthreads();
            for (int k = 0; k < nsig; ++k) {
                const double c = coef.c[k];
                // rows of the tile x molecules of the second side
                for (int t = tid; t < VK_T * s2.group; t += VK_TPB) {
                    const int r = t & (VK_T - 1), q = t / VK_T;
                    if (r < nr) {
                        part[r][q] = sum4(max(seg2[q] - c0, 0), min(seg2[q + 1] - c0, nc),
                                          [&](int x) { return exp(D[r][x] * c); });
                    }
                }
                __syncthreads();
                for (int t = tid; t < g12; t += VK_TPB) {
                    const int p = t / s2.group, q = t - p * s2.group;
                    ksum[k * g12 + t] += sum4(max(seg1[p] - r0, 0), min(seg1[p + 1] - r0, nr),
                                              [&](int x) { return part[x][q]; });
                }
                __syncthreads();
            }
        }
    }
    for (int t = tid; t < nsig * g12; t += VK_TPB) {
        const int k = t / g12, p = (t - k * g12) / s2.group, q = t % s2.group;
        if (m1 + p < s1.nm && m2 + q < s2.nm)
            K[((size_t)k * s1.nm + m1 + p) * s2.nm + m2 + q] = ksum[t];
    }
}

// Small sets of short descriptors: a CTA per molecule pair, two atom pairs at most per
// thread, 32 features of all atoms in shared memory at a time. What counts there is the
// time of one CTA from its start to its end, of which the tile takes 2 to 4 us more. us
// with a CTA per pair and with tiles: 30 x 36 molecules of 7 atoms, d = 28, 6, 10; 10
// atoms, d = 55, 9, 12; 45 x 54 of 11, d = 120, 23, 25; 52 x 62 of 11, d = 66, 19, 19, d =
// 100, 29, 27; 1 and 100 atoms, d = 30, 19, 27, 100 x 120 of these 57, 67.
constexpr int VP_TPB = 64, VP_ATOM_PAIRS = 2 * VP_TPB, VP_FEATURES = 32, VP_PITCH = 33;
constexpr int VP_MAX_D = 128, VP_PAIRS_PER_SM = 24;

template <int KIND>
__global__ void __launch_bounds__(VP_TPB)
vector_pair_kernel(const VkSide s1, const VkSide s2, int d, const __grid_constant__ Coefs coef,
                   int nsig, double *__restrict__ K, int *__restrict__ status) {
    extern __shared__ double ksum[];  // features of the first side's atoms, then the second's
    __shared__ double half[VK_MAX_SIGMAS];
    double *A = ksum, *B = A + s1.amax * VP_PITCH;
    const int i = (int)(blockIdx.x / (unsigned)s2.nm), j = (int)(blockIdx.x % (unsigned)s2.nm);
    const int t = threadIdx.x, lane = t & 31;
    int *stat = t == 0 ? status : nullptr;
    long long f1, f2;
    const int ni = vk_molecule(s1, i, f1, stat), nj = vk_molecule(s2, j, f2, stat), np = ni * nj;
    const double *x1 = s1.X + f1 * d, *x2 = s2.X + f2 * d;
    int at[2], bt[2];
    double dist[2] = {0.0, 0.0};
#pragma unroll
    for (int q = 0; q < 2; ++q) {  // atom pair t + 64 q; past the last: the last once more
        const int p = max(min(t + q * VP_TPB, np - 1), 0), b = ni ? p / ni : 0;
        at[q] = (p - b * ni) * VP_PITCH;
        bt[q] = b * VP_PITCH;
    }
    for (int c = 0; c < d && np > 0; c += VP_FEATURES) {
        const int nf = min(VP_FEATURES, d - c);
        __syncthreads();
        for (int e = t; e < ni * VP_FEATURES; e += VP_TPB) {
            const int a = e / VP_FEATURES, f = e % VP_FEATURES;
            if (f < nf) A[a * VP_PITCH + f] = x1[(size_t)a * d + c + f];
        }
        for (int e = t; e < nj * VP_FEATURES; e += VP_TPB) {
            const int b = e / VP_FEATURES, f = e % VP_FEATURES;
            if (f < nf) B[b * VP_PITCH + f] = x2[(size_t)b * d + c + f];
        }
        __syncthreads();
#pragma unroll 4
        for (int k = 0; k < nf; ++k)
#pragma unroll
            for (int q = 0; q < 2; ++q)
                dist[q] = dist::add_term<KIND == 0 ? dist::kSquareUnfused : dist::kAbs>(
                    dist[q], A[at[q] + k], B[bt[q] + k]);
    }
    double mine = 0.0;  // lane k's: the first warp's sum of sigma k
#pragma unroll 1
    for (int k = 0; k < nsig; ++k) {
        double v = 0.0;
#pragma unroll
        for (int q = 0; q < 2; ++q)
            if (t + q * VP_TPB < np) v += exp(dist[q] * coef.c[k]);
        for (int o = 16; o; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
        if (t == VP_TPB / 2) half[k] = v;
        if (lane == k) mine = v;
    }
    __syncthreads();
    if (t < nsig) K[((size_t)t * s1.nm + i) * s2.nm + j] = mine + half[t];
}

bool vk_small(const VkSide &s1, const VkSide &s2, int d) {
    return s1.amax * s2.amax <= VP_ATOM_PAIRS && d <= VP_MAX_D &&
           (long long)s1.nm * s2.nm <= (long long)VP_PAIRS_PER_SM * sm_count();
}

// Molecules per group: about 80 atoms at the usual fill of a padded row (the
// tile's unused rows and columns then cost a sixth), fewer while the blocks
// would not fill the GPU a few times over: a side of more than one tile is halved until
// there are eight blocks per SM, one within a tile only until there are two, since that
// leaves more of the tile empty. us for groups of 1 x 1, 2 x 1 and 2 x 2 of 23 atoms, d =
// 276, one sigma: 30 x 30 molecules 73, 62, -; 40 x 40 105, 95, 76; 60 x 60 (2 x 1, 2 x 2)
// 159, 122. 100 x 120 of 4 and 30 atoms, d = 100: 8 x 2 molecules 53, 2 x 2 126. With a CTA
// per molecule pair: 74, 113, 215 and 84 us.
void vk_groups(VkSide &s1, VkSide &s2) {
    auto most = [](const VkSide &s) { return std::max(1, std::min(VK_MAX_GROUP, VK_ROWS / s.amax)); };
    s1.group = most(s1);
    s2.group = most(s2);
    auto blocks = [&] {
        return (long long)ceil_div(s1.nm, s1.group) * ceil_div(s2.nm, s2.group);
    };
    for (;;) {
        const bool first = s2.group == 1 || (s1.group > 1 && s1.group * s1.amax >= s2.group * s2.amax);
        VkSide &s = first ? s1 : s2;
        if (s.group == 1 || blocks() >= (s.group * s.amax > VK_T ? 8LL : 2LL) * sm_count()) break;
        s.group = (s.group + 1) / 2;
    }
}

template <int KIND>
int launch_vk(VkSide s1, VkSide s2, int d, const Coefs &coef, int nsig, double *K, int *status,
              cudaStream_t st) {
    if (vk_small(s1, s2, d)) {
        const size_t smem = sizeof(double) * VP_PITCH * (s1.amax + s2.amax);  // at most 34 KB
        vector_pair_kernel<KIND><<<(unsigned)(s1.nm * s2.nm), VP_TPB, smem, st>>>(s1, s2, d, coef,
                                                                                 nsig, K, status);
        return launch_status("vector_pair_kernel");
    }
    vk_groups(s1, s2);
    // at most 16 KB, but beside 41 KB of static shared memory: with many sigmas the two
    // pass the 48 KB that a launch gets without the attribute
    const size_t smem = sizeof(double) * (size_t)nsig * s1.group * s2.group;
    FMLB_TRY(cuda_status(cudaFuncSetAttribute(vector_kernels_kernel<KIND>,
                                              cudaFuncAttributeMaxDynamicSharedMemorySize,
                                              (int)smem),
                         "cudaFuncSetAttribute"));
    const long long blocks = (long long)ceil_div(s1.nm, s1.group) * ceil_div(s2.nm, s2.group);
    vector_kernels_kernel<KIND><<<(unsigned)blocks, VK_TPB, smem, st>>>(s1, s2, d, coef, nsig, K,
                                                                      status);
    return launch_status(KIND == 0 ? "vector_kernels_kernel<gaussian>"
                                   : "vector_kernels_kernel<laplacian>");
}

}  // namespace
}  // namespace fmlb

static int vector_kernels_impl(int kind, const double *X1, const int *N1, int nm1, int amax1,
                               const double *X2, const int *N2, int nm2, int amax2, int d,
                               const double *sigmas_host, int nsig, double *K, int *status,
                               const int *O1, const int *O2, void *stream) {
    using namespace fmlb;
    FMLB_REQUIRE(kind == 0 || kind == 1, "fmlb_vector_kernels_f64: kind must be 0 or 1");
    FMLB_REQUIRE(nm1 >= 0 && nm2 >= 0 && d >= 0, "fmlb_vector_kernels_f64: bad sizes");
    FMLB_REQUIRE(amax1 >= 1 && amax1 <= VK_MAX_ATOMS && amax2 >= 1 && amax2 <= VK_MAX_ATOMS,
                 "fmlb_vector_kernels_f64: atoms per molecule must be 1..%d", VK_MAX_ATOMS);
    FMLB_REQUIRE(nsig >= 1 && nsig <= VK_MAX_SIGMAS,
                 "fmlb_vector_kernels_f64: nsig=%d outside 1..%d", nsig, VK_MAX_SIGMAS);
    FMLB_REQUIRE(sigmas_host, "fmlb_vector_kernels_f64: null sigmas");
    if ((long long)nm1 * nm2 == 0) return FMLB_OK;
    FMLB_REQUIRE(X1 && (N1 || O1) && X2 && (N2 || O2) && K,
                 "fmlb_vector_kernels_f64: null pointer");
    Coefs coef;
    for (int k = 0; k < nsig; ++k) {
        FMLB_REQUIRE(sigmas_host[k] > 0.0, "fmlb_vector_kernels_f64: sigma %d not positive", k);
        coef.c[k] = kind == 0 ? -0.5 / (sigmas_host[k] * sigmas_host[k]) : -1.0 / sigmas_host[k];
    }
    cudaStream_t st = FMLB_STREAM(stream);
    FMLB_REQUIRE((long long)nm1 * nm2 < 0x7fffffffLL,
                 "fmlb_vector_kernels_f64: too many molecule pairs");
    const VkSide s1 = {X1, N1, O1, nm1, amax1, 1}, s2 = {X2, N2, O2, nm2, amax2, 1};
    return kind == 0 ? launch_vk<0>(s1, s2, d, coef, nsig, K, status, st)
                     : launch_vk<1>(s1, s2, d, coef, nsig, K, status, st);
}

extern "C" int fmlb_vector_kernels_f64(int kind, const double *X1, const int *N1, int nm1,
                                       int amax1, const double *X2, const int *N2, int nm2,
                                       int amax2, int d, const double *sigmas_host, int nsig,
                                       double *K, int *status, void *stream) {
    return vector_kernels_impl(kind, X1, N1, nm1, amax1, X2, N2, nm2, amax2, d, sigmas_host,
                               nsig, K, status, nullptr, nullptr, stream);
}

// Packed form: X (total_atoms, d) rows with molecule offsets O (nm + 1);
// amax bounds the atoms of one molecule (checked on the device through
// status). The molecule kernel of fget_alpha (fkernels.f90:380-440) is the
// Laplacian form with X1 = X2.
extern "C" int fmlb_vector_kernels_packed_f64(int kind, const double *X1, const int *O1, int nm1,
                                              int amax1, const double *X2, const int *O2, int nm2,
                                              int amax2, int d, const double *sigmas_host,
                                              int nsig, double *K, int *status, void *stream) {
    using namespace fmlb;
    FMLB_REQUIRE(nm1 == 0 || O1, "fmlb_vector_kernels_packed_f64: null offsets");
    FMLB_REQUIRE(nm2 == 0 || O2, "fmlb_vector_kernels_packed_f64: null offsets");
    return vector_kernels_impl(kind, X1, nullptr, nm1, amax1, X2, nullptr, nm2, amax2, d,
                               sigmas_host, nsig, K, status, O1, O2, stream);
}
