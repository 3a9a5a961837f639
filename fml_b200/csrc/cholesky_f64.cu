// Plain-FP64 blocked right-looking Cholesky factorisation and solve, the
// replacement for LAPACK dpotrf('U') / dpotrs('U') as fcho_solve calls them
// (fml/math/fcho_solve.f90:35-42).
//
// Storage: row-major (n, n), factor L in the triangle i >= j (A = L L^T); the
// other triangle is never read or written. For the reference's C-order
// argument this is its dpotrf('U') factor U = L^T.
//
// Two levels of blocking. Inner panels of NB = 128 columns:
//   1. potf2 of the diagonal block in shared memory (one CTA), with the inverses
//      of its 32 x 32 diagonal sub-blocks; a
//      non-positive pivot records the LAPACK info (1-based column) and every
//      later kernel of the factorisation returns at once;
//   2. panel solve L21 = A21 L11^-T by 32-column blocks with those inverses;
// outer panels of 256, 512 or 1024 columns (wider at larger n):
//   3. trailing update A22 -= L21 L21^T with k = the outer width, on the FP64
//      tensor cores (mma.sync m8n8k4 f64), 128x64 tiles on or below the
//      diagonal, operands streamed through a 3-stage cp.async pipeline;
// with the next outer panel factored on a second stream under step 3.
// The inverses of the 128 x 128 diagonal blocks, formed at the end for all
// blocks side by side, stay in the workspace for the solve (section 4).
#include <math.h>
#include <stdint.h>

#include <algorithm>

#include "common.cuh"
#include "ozaki.cuh"
#include "tc_common.cuh"

namespace fmlb {
namespace {

constexpr int NB = 128;  // panel width
constexpr int TPB = 256;

__device__ __forceinline__ bool failed(const int *info) {
    return info && *(volatile const int *)info != 0;
}

// Programmatic dependent launch (kernels launched with programmatic stream
// serialization; in a kernel launched without it both are no-ops).
// griddepcontrol.wait returns once the previous kernel of the stream has
// completed and its writes are visible, so every read of data that kernel
// may write comes after it. The panel chain (diagonal block, panel solve,
// update inside the outer panel) signals its dependent only at its end, so
// the next kernel's CTAs do not sit on SMs the concurrent bulk update needs.
__device__ __forceinline__ void pdl_launch_dependents() {
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
}
__device__ __forceinline__ void pdl_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }

__device__ __forceinline__ void cp_async_16(void *smem, const void *gmem, int src_bytes) {
    const unsigned s = (unsigned)__cvta_generic_to_shared(smem);
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(s), "l"(gmem),
                 "r"(src_bytes));
}
__device__ __forceinline__ void cp_async_8(void *smem, const void *gmem, int src_bytes) {
    const unsigned s = (unsigned)__cvta_generic_to_shared(smem);
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;\n" ::"r"(s), "l"(gmem),
                 "r"(src_bytes));
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;\n"); }
template <int N>
__device__ __forceinline__ void cp_async_wait() {
    asm volatile("cp.async.wait_group %0;\n" ::"n"(N));
}

// ---- 1. diagonal block ----------------------------------------------------
// The 128 x 128 block is factored in four 32-column steps:
//   warp 0 factors the 32 x 32 diagonal sub-block in registers, warp 1 follows it
//   by eight columns with the sub-block's inverse, and the other warps meanwhile
//   do what is left of the update by the step before;
//   all warps: the 32-column sub-panel below it (a product with the inverse), then
//   the update of the next diagonal sub-block, on the FP64 tensor cores.
// Only the four 32 x 32 inverses are formed here: the panel solve needs no more,
// and the block inverses of the triangular solves come from block_inverse_kernel,
// once, for all blocks side by side.
//
// Bound by the latency of the 128 serial pivots, about 190 cycles each. 24 us a
// block; 36 with the inverse's updates and the whole block's behind the pivots on
// the one warp's path and the column's stores, with their bank conflicts, among them;
// 190 with factor and inverse in separate passes and the block products as
// shared-memory FMA loops.
constexpr int LDL = NB + 4;  // row pitch: the fragments' rows fall in distinct banks
constexpr int SB = 32, NSB = NB / SB, LDW = SB + 4;
constexpr size_t kPotf2Smem =  // the block, two inverses, the sub-block's columns and roots
    ((size_t)NB * LDL + 2 * (size_t)(SB * LDW + SB * SB + 2 * SB)) * sizeof(double);

__device__ __forceinline__ void dmma_8x8x4(double (&d)[2], double a, double b) {
    asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0,%1}, {%2}, {%3}, {%0,%1};\n"
                 : "+d"(d[0]), "+d"(d[1])
                 : "d"(a), "d"(b));
}

// 1 / sqrt(x) for normal x by a third-order step from the hardware's approximation
// (Householder's method: e = 1 - x y^2, y (1 + e / 2 + 3 e^2 / 8)), without branches.
__device__ __forceinline__ double rsqrt_normal(double x) {
    double y;
    asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(x));
    const double e = fma(-(x * y), y, 1.0);
    return fma(fma(0.375, e, 0.5), y * e, y);
}

// Named barriers between warps 0 and 1, one for each eight columns.
__device__ __forceinline__ void columns_done(int id) {
    asm volatile("bar.arrive %0, 64;" ::"r"(id) : "memory");
}
__device__ __forceinline__ void columns_wait(int id) {
    asm volatile("bar.sync %0, 64;" ::"r"(id) : "memory");
}

// What a column step of the sub-block's factorisation hands to the next, the same
// in every lane: column J's pivot and its reciprocal root, the entry below the pivot
// (unscaled) and the diagonal entry after that one, both as the steps before J left
// them.
struct PotrfStep {
    double piv, inv, below, diag;
};

// Eight column steps, `WIDTH` columns left at the first: a[c] holds the lane's
// (row's) entry of column J + c. A step scales column J by inv, stores it and
// updates the columns after it into the registers one place down. Every lane forms
// the next pivot by itself from `below` and `diag`, which were broadcast a step
// ahead, so that a column's chain is the reciprocal root and two operations, with
// the broadcasts and the updates beside it. The column goes through shared memory
// (two entries to a load, where a shuffle takes two instructions each). Entries above
// the diagonal and past the last column hold values that nothing reads.
template <int WIDTH, bool kCareful>
__device__ __forceinline__ void potrf_steps(double (&a)[SB], PotrfStep &s, int J0, double *cols,
                                            double *invs, double &mine) {
    const int lane = threadIdx.x & 31;
#pragma unroll 1
    for (int q = 0; q < 8; ++q) {
        const int J = J0 + q;
        const double lij = a[0] * s.inv, l1 = s.below * s.inv, piv = fma(-l1, l1, s.diag);
        double *col = cols + J * SB;  // L[J + c][J] at c
        col[(lane - J) & 31] = lij;
        invs[J] = s.inv;
        if (lane == J) mine = s.piv;
        a[1] = fma(-lij, l1, a[1]);
        s.below = __shfl_sync(0xffffffffu, a[1], (J + 2) & 31);
        s.diag = __shfl_sync(0xffffffffu, fma(-lij, lij, a[2]), (J + 2) & 31);
        __syncwarp();
        s.piv = piv;
        s.inv = kCareful ? rsqrt(piv) : rsqrt_normal(piv);
        a[0] = a[1];
#pragma unroll
        for (int c = 2; c < WIDTH; c += 2) {
            const double2 l = *reinterpret_cast<const double2 *>(col + c);
            a[c - 1] = fma(-lij, l.x, a[c]);
            a[c] = fma(-lij, l.y, a[c + 1 < SB ? c + 1 : c]);
        }
    }
    columns_done(1 + J0 / 8);
}

// Warp 0: factors the 32 x 32 sub-block at L[b0.., b0..] into cols, with the pivots
// and their reciprocal roots in pivs and invs. Returns the 1-based failing column, 0
// or, unless kCareful, -1 (the same in every lane) for a pivot that is not a normal
// number: the library's reciprocal root then has to be used.
template <bool kCareful>
__device__ __forceinline__ int warp_potrf32(double (*L)[LDL], int b0, double *cols, double *invs,
                                            double *pivs) {
    const int lane = threadIdx.x & 31;
    double a[SB];
#pragma unroll
    for (int c = 0; c < SB; ++c) a[c] = c <= lane ? L[b0 + lane][b0 + c] : 0.0;
    PotrfStep s;
    s.piv = __shfl_sync(0xffffffffu, a[0], 0);
    s.inv = rsqrt(s.piv);
    s.below = __shfl_sync(0xffffffffu, a[0], 1);
    s.diag = __shfl_sync(0xffffffffu, a[1], 1);
    double mine = 0.0;
    static_assert(SB == 32, "four times eight steps");
    potrf_steps<32, kCareful>(a, s, 0, cols, invs, mine);
    potrf_steps<24, kCareful>(a, s, 8, cols, invs, mine);
    potrf_steps<16, kCareful>(a, s, 16, cols, invs, mine);
    potrf_steps<8, kCareful>(a, s, 24, cols, invs, mine);
    pivs[lane] = mine;
    const bool normal = mine >= 2.2250738585072014e-308 && mine <= 1.7976931348623157e308;
    const unsigned other = __ballot_sync(0xffffffffu, kCareful ? !(mine > 0.0) : !normal);
    if (!other) return 0;
    const int first = __ffs(other) - 1;
    if (!kCareful && __shfl_sync(0xffffffffu, mine, first) > 0.0) return -1;
    return first + 1;
}

// Eight row steps of the forward substitution for the inverse: v[c] holds the
// lane's (column's) entry of row J + c, moved down as above.
template <int WIDTH>
__device__ __forceinline__ void inverse_steps(double (&v)[SB], int J0, double (*W)[LDW],
                                              const double *cols, const double *invs) {
    const int lane = threadIdx.x & 31;
    columns_wait(1 + J0 / 8);
#pragma unroll 1
    for (int J = J0; J < J0 + 8; ++J) {
        const double vj = v[0] * invs[J];
        W[J][lane] = vj;
#pragma unroll
        for (int c = 0; c < WIDTH; c += 2) {
            const double2 l = *reinterpret_cast<const double2 *>(cols + J * SB + c);
            if (c > 0) v[c - 1] = fma(-l.x, vj, v[c]);
            v[c] = fma(-l.y, vj, v[c + 1 < SB ? c + 1 : c]);
        }
    }
}

// Warp 1: the inverse of the sub-block that warp 0 factors, into W (row-major, zeros
// above the diagonal).
__device__ __forceinline__ void warp_inverse32(double (*W)[LDW], const double *cols,
                                               const double *invs) {
    const int lane = threadIdx.x & 31;
    double v[SB];
#pragma unroll
    for (int c = 0; c < SB; ++c) v[c] = c == lane ? 1.0 : 0.0;
    inverse_steps<32>(v, 0, W, cols, invs);
    inverse_steps<24>(v, 8, W, cols, invs);
    inverse_steps<16>(v, 16, W, cols, invs);
    inverse_steps<8>(v, 24, W, cols, invs);
}

// A factored sub-block to its place in the block, its diagonal as the root of the
// pivot, corrected once, and its inverse to its place in the block inverse: rows
// `part`, part + parts and so on.
__device__ __forceinline__ void put_subblock(double (*L)[LDL], double *__restrict__ Linv, int b0,
                                             const double *step, int part, int parts) {
    const int lane = threadIdx.x & 31;
    const double *W = step, *cols = W + SB * LDW, *pivs = cols + SB * SB, *invs = pivs + SB;
#pragma unroll 4
    for (int r = part; r < SB; r += parts) {
        const double piv = pivs[r], inv = invs[r], root = piv * inv;
        // an infinite pivot (its reciprocal root is zero) is its own root
        const double diag = inv > 0.0 ? fma(0.5 * inv, fma(-root, root, piv), root) : piv;
        const double v = lane == r ? diag : cols[lane * SB + ((r - lane) & 31)];
        if (lane <= r) L[b0 + r][b0 + lane] = v;
        Linv[(size_t)(b0 + r) * NB + b0 + lane] = W[r * LDW + lane];
    }
}

// T 8 x 8 tiles of the block side by side: L[m.., c..] -= L[m.., b0..] L[c.., b0..]^T
template <int T>
__device__ __forceinline__ void update_tiles(double (*L)[LDL], int m, int c, int b0) {
    const int lane = threadIdx.x & 31, g = lane >> 2, tq = lane & 3;
    double o[T][4][2];
#pragma unroll
    for (int t = 0; t < T; ++t)
#pragma unroll
        for (int q = 0; q < 4; ++q) o[t][q][0] = o[t][q][1] = 0.0;
#pragma unroll
    for (int k = 0; k < SB; k += 4) {
        const double x = L[m + g][b0 + k + tq];
#pragma unroll
        for (int t = 0; t < T; ++t) dmma_8x8x4(o[t][k / 4 % 4], x, L[c + 8 * t + g][b0 + k + tq]);
    }
#pragma unroll
    for (int t = 0; t < T; ++t)
#pragma unroll
        for (int q = 0; q < 2; ++q)
            L[m + g][c + 8 * t + 2 * tq + q] -=
                (o[t][0][q] + o[t][1][q]) + (o[t][2][q] + o[t][3][q]);
}

__global__ void __launch_bounds__(TPB, 1)
potf2_block_kernel(double *__restrict__ A, long long lda, int k0, int kn,
                   double *__restrict__ Linv, int *__restrict__ info) {
    extern __shared__ __align__(16) double potf2_smem[];
    double(*L)[LDL] = reinterpret_cast<double(*)[LDL]>(potf2_smem);
    constexpr int kWarps = TPB / 32, kStep = SB * LDW + SB * SB + 2 * SB;
    const auto step = [&](int J) {  // two buffers: inverse, columns, pivots, their roots
        return potf2_smem + NB * LDL + (J & 1) * kStep;
    };
    __shared__ int bad;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int g = lane >> 2, tq = lane & 3;  // fragment row / k (A, B), row / column pair (C)
    double *Ak = A + (size_t)k0 * lda + k0;
    const bool wide = (uintptr_t)Ak % 16 == 0 && lda % 2 == 0;
    if (tid == 0) bad = 0;
    pdl_wait();
    if (wide) {
        for (int r = warp; r < kn; r += kWarps)  // all loads in flight together
#pragma unroll
            for (int c = 2 * lane; c < NB; c += 64)
                if (c <= r) cp_async_16(&L[r][c], Ak + (size_t)r * lda + c, c < r ? 16 : 8);
    } else {
        for (int r = warp; r < kn; r += kWarps)
#pragma unroll
            for (int c = lane; c < NB; c += 32)
                if (c <= r) cp_async_8(&L[r][c], Ak + (size_t)r * lda + c, 8);
    }
    for (int r = kn + warp; r < NB; r += kWarps)  // identity past kn keeps the block SPD
        for (int c = lane; c <= r; c += 32) L[r][c] = r == c ? 1.0 : 0.0;
    cp_async_commit();
    const bool stop = failed(info);
    cp_async_wait<0>();
    if (stop) return;
    __syncthreads();
    for (int J = 0; J < NSB; ++J) {
        const int b0 = J * SB, r0 = b0 + SB, p0 = b0 - SB;
        double(*W)[LDW] = reinterpret_cast<double(*)[LDW]>(step(J));
        double *cols = step(J) + SB * LDW, *pivs = cols + SB * SB, *invs = pivs + SB;
        if (warp == 0) {
            const int f = warp_potrf32<false>(L, b0, cols, invs, pivs);
            if (f && lane == 0) bad = f > 0 ? b0 + f : f;
        } else if (warp == 1) {
            warp_inverse32(W, cols, invs);
        } else if (J > 0 && (warp & 2)) {
            // the rest of the update by step J - 1, two 8 x 8 tiles at a time (the
            // second may lie above the diagonal), by the warps that share no
            // scheduler with warps 0 and 1
            const int nt = (NB - b0) / 8, turn = (warp & 1) + (warp >> 2) * 2;
            int item = 0;
            for (int ti = SB / 8; ti < nt; ++ti)
                for (int tj = 0; tj <= ti; tj += 2)
                    if ((item++ & 3) == turn) update_tiles<2>(L, b0 + 8 * ti, b0 + 8 * tj, p0);
        } else if (J > 0) {
            put_subblock(L, Linv, p0, step(J - 1), warp & 1, 2);
        }
        __syncthreads();
        if (bad < 0) {  // a pivot outside the normal numbers
            __syncthreads();
            if (warp == 0) {
                const int f = warp_potrf32<true>(L, b0, cols, invs, pivs);
                if (lane == 0) bad = f ? b0 + f : 0;
            } else if (warp == 1) {
                warp_inverse32(W, cols, invs);
            }
            __syncthreads();
        }
        if (bad) {
            if (tid == 0) atomicCAS(info, 0, k0 + bad);
            return;
        }
        if (J == NSB - 1) break;
        // sub-panel solve, 8 rows per warp and turn: X <- X inv(D)^T
        for (int m = r0 + warp * 8; m < NB; m += 8 * kWarps) {
            double x[SB / 4], o[SB / 8][2];
#pragma unroll
            for (int k = 0; k < SB / 4; ++k) x[k] = L[m + g][b0 + 4 * k + tq];
#pragma unroll
            for (int c = 0; c < SB / 8; ++c) {
                o[c][0] = o[c][1] = 0.0;
#pragma unroll
                for (int k = 0; k < 2 * c + 2; ++k)  // inv(D) is lower triangular
                    dmma_8x8x4(o[c], x[k], W[8 * c + g][4 * k + tq]);
            }
            __syncwarp();
#pragma unroll
            for (int c = 0; c < SB / 8; ++c) {
                L[m + g][b0 + 8 * c + 2 * tq] = o[c][0];
                L[m + g][b0 + 8 * c + 2 * tq + 1] = o[c][1];
            }
        }
        __syncthreads();
        // update of the next diagonal sub-block: its ten tiles on or below the diagonal
        for (int t = warp; t < 10; t += kWarps) {
            const int ti = (t > 0) + (t > 2) + (t > 5), tj = t - ti * (ti + 1) / 2;
            update_tiles<1>(L, r0 + 8 * ti, r0 + 8 * tj, b0);
        }
        __syncthreads();
    }
    put_subblock(L, Linv, NB - SB, step(NSB - 1), warp, kWarps);
    __syncthreads();
    // factor back to global (16-byte stores took 4500 cycles, these 2700)
#pragma unroll 4
    for (int r = warp; r < kn; r += kWarps)
#pragma unroll
        for (int c = lane; c < NB; c += 32)
            if (c <= r) Ak[(size_t)r * lda + c] = L[r][c];
    pdl_launch_dependents();
}

// ---- 2. panel solve: rows [r0, n) of columns [k0, k0+kn): X <- X L11^-T ----
// Forward substitution by 32-column blocks on the FP64 tensor cores: X_J <-
// (X_J - sum_{K < J} X_K L_JK^T) W_J^T with the factored diagonal block and its
// 32 x 32 inverses W_J. Chunks of 32 rows, one CTA per SM taking them in turn
// with the diagonal block kept in shared memory; warp w owns 8 rows and 16 of
// each block's 32 columns.
constexpr int TRSM_ROWS = 32;
constexpr int TRSM_BLK = SB * LDW;  // doubles of a 32 x 32 block of the lower triangle
constexpr size_t kTrsmSmem =
    ((size_t)TRSM_ROWS * LDL + (size_t)NSB * (NSB + 1) / 2 * TRSM_BLK) * sizeof(double);

__global__ void __launch_bounds__(TPB)
panel_trsm_kernel(double *__restrict__ A, long long lda, int n, int k0,
                  const double *__restrict__ Linv, const int *__restrict__ info) {
    extern __shared__ __align__(16) double trsm_smem[];
    double(*X)[LDL] = reinterpret_cast<double(*)[LDL]>(trsm_smem);
    double *blocks = trsm_smem + TRSM_ROWS * LDL;  // (R, C) at R (R + 1) / 2 + C
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int g = lane >> 2, tq = lane & 3;
    const bool wide = ((uintptr_t)A | (uintptr_t)Linv) % 16 == 0 && lda % 2 == 0;
    pdl_wait();
    const auto place = [&](int r, int c) {
        const int R = r / SB, C = c / SB;
        return blocks + (R * (R + 1) / 2 + C) * TRSM_BLK + (r % SB) * LDW + c % SB;
    };
    const double *Ak = A + (size_t)k0 * lda + k0;
    if (wide) {
        for (int t = tid; t < NB * NB / 2; t += TPB) {
            const int r = t / (NB / 2), c = t % (NB / 2) * 2;
            if (c / SB <= r / SB)
                cp_async_16(place(r, c), c / SB == r / SB ? Linv + 2 * t : Ak + (size_t)r * lda + c,
                            16);
        }
    } else {
        for (int t = tid; t < NB * NB; t += TPB) {
            const int r = t / NB, c = t % NB;
            if (c / SB <= r / SB)
                cp_async_8(place(r, c), c / SB == r / SB ? Linv + t : Ak + (size_t)r * lda + c, 8);
        }
    }
    const bool stop = failed(info);
    const int m = (warp & 3) * 8, h = (warp >> 2) * 16;  // rows m.., columns h.. of each block
    for (int r0 = k0 + NB + blockIdx.x * TRSM_ROWS; r0 < n && !stop;
         r0 += gridDim.x * TRSM_ROWS) {
        if (wide) {
            for (int t = tid; t < TRSM_ROWS * NB / 2; t += TPB) {
                const int r = t / (NB / 2), c = t % (NB / 2) * 2;
                cp_async_16(&X[r][c], A + (size_t)min(r0 + r, n - 1) * lda + k0 + c,
                            r0 + r < n ? 16 : 0);
            }
        } else {
            for (int t = tid; t < TRSM_ROWS * NB; t += TPB) {
                const int r = t / NB, c = t % NB;
                cp_async_8(&X[r][c], A + (size_t)min(r0 + r, n - 1) * lda + k0 + c,
                           r0 + r < n ? 8 : 0);
            }
        }
        cp_async_commit();
        cp_async_wait<0>();
        for (int J = 0; J < NSB; ++J) {
            const double *row = blocks + J * (J + 1) / 2 * TRSM_BLK + (h + g) * LDW + tq;
            __syncthreads();
            double o[2][4][2] = {};  // four chains for each 8 x 8 tile
            for (int K = 0; K < J; ++K) {
#pragma unroll
                for (int k = 0; k < SB; k += 4) {
                    const double x = X[m + g][K * SB + k + tq];
#pragma unroll
                    for (int c = 0; c < 2; ++c)
                        dmma_8x8x4(o[c][k / 4 % 4], x, row[K * TRSM_BLK + 8 * c * LDW + k]);
                }
            }
#pragma unroll
            for (int c = 0; c < 2; ++c)
#pragma unroll
                for (int q = 0; q < 2; ++q) {
                    X[m + g][J * SB + h + 8 * c + 2 * tq + q] -=
                        (o[c][0][q] + o[c][1][q]) + (o[c][2][q] + o[c][3][q]);
                    o[c][0][q] = o[c][1][q] = 0.0;
                }
            __syncthreads();
            for (int k = 0; k < h + 16; k += 8) {  // W_J is lower triangular
#pragma unroll
                for (int e = 0; e < 2; ++e) {
                    const double x = X[m + g][J * SB + k + 4 * e + tq];
#pragma unroll
                    for (int c = 0; c < 2; ++c)
                        dmma_8x8x4(o[c][e], x, row[J * TRSM_BLK + 8 * c * LDW + k + 4 * e]);
                }
            }
            __syncthreads();
#pragma unroll
            for (int c = 0; c < 2; ++c)
#pragma unroll
                for (int q = 0; q < 2; ++q)
                    X[m + g][J * SB + h + 8 * c + 2 * tq + q] = o[c][0][q] + o[c][1][q];
        }
        __syncthreads();
        for (int t = tid; t < TRSM_ROWS * NB; t += TPB) {
            const int r = t / NB, c = t % NB;
            if (r0 + r < n) A[(size_t)(r0 + r) * lda + k0 + c] = X[r][c];
        }
        __syncthreads();
    }
    cp_async_wait<0>();
    pdl_launch_dependents();
}

// Inverses of the 128 x 128 diagonal blocks of the factor for the triangular
// solves, one CTA per block: from the 32 x 32 inverses that the factorisation
// left on their diagonal,
//   inv(L)_IJ = -inv(L_II) sum_{K=J}^{I-1} L_IK inv(L)_KJ,  I > J,
// block row by block row, and zeros above the diagonal.
constexpr int LDT = NB - SB + 4;  // a block row of L left of the diagonal: 32 x 96
constexpr size_t kBlockInvSmem = ((size_t)NB * LDL + (size_t)SB * LDT) * sizeof(double);

__global__ void __launch_bounds__(TPB)
block_inverse_kernel(const double *__restrict__ A, long long lda, int n, double *__restrict__ Linv,
                     const int *__restrict__ info) {
    extern __shared__ double potf2_smem[];
    double(*V)[LDL] = reinterpret_cast<double(*)[LDL]>(potf2_smem);  // the inverse
    double(*T)[LDT] = reinterpret_cast<double(*)[LDT]>(potf2_smem + NB * LDL);
    pdl_wait();
    if (failed(info)) return;
    const int k0 = blockIdx.x * NB, kn = min(NB, n - k0);
    double *Li = Linv + (size_t)blockIdx.x * NB * NB;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int g = lane >> 2, tq = lane & 3;
    for (int t = tid; t < NB * NB; t += TPB) {
        const int r = t >> 7, c = t & (NB - 1);
        if (c / SB == r / SB) cp_async_8(&V[r][c], Li + t, 8);
        else V[r][c] = 0.0;
    }
    for (int I = 1; I < NSB; ++I) {
        // T: block row I of L, then sum_K L_IK inv(L)_KJ in its place
        __syncthreads();
        for (int t = tid; t < SB * I * SB; t += TPB) {
            const int r = t / (I * SB), c = t % (I * SB);
            const bool in = I * SB + r < kn;
            cp_async_8(&T[r][c], in ? A + (size_t)(k0 + I * SB + r) * lda + k0 + c : A, in ? 8 : 0);
        }
        cp_async_commit();
        cp_async_wait<0>();
        __syncthreads();
        double o[6][2];  // 8 x 8 tiles of the (32 x 32 I) block row, 16 I of them over 8 warps
        for (int pass = 0; pass < 2; ++pass) {
            // pass 0: T <- T V_0..I-1,J;  pass 1: V_I <- -V_II T
#pragma unroll
            for (int q = 0; q < 6; ++q) {
                const int t = warp + q * (TPB / 32);
                if (t < 16 * I) {
                    const int m = (t & 3) * 8, c = (t >> 2) * 8;
                    o[q][0] = o[q][1] = 0.0;
                    if (pass == 0)
                        for (int k = c / SB * SB; k < I * SB; k += 4)
                            dmma_8x8x4(o[q], T[m + g][k + tq], V[k + tq][c + g]);
                    else
                        for (int k = 0; k < m + 8; k += 4)  // V_II is lower triangular
                            dmma_8x8x4(o[q], V[I * SB + m + g][I * SB + k + tq], T[k + tq][c + g]);
                }
            }
            __syncthreads();
#pragma unroll
            for (int q = 0; q < 6; ++q) {
                const int t = warp + q * (TPB / 32);
                if (t < 16 * I) {
                    const int m = (t & 3) * 8, c = (t >> 2) * 8 + 2 * tq;
                    if (pass == 0) {
                        T[m + g][c] = o[q][0];
                        T[m + g][c + 1] = o[q][1];
                    } else {
                        V[I * SB + m + g][c] = -o[q][0];
                        V[I * SB + m + g][c + 1] = -o[q][1];
                    }
                }
            }
            __syncthreads();
        }
    }
    for (int t = tid; t < NB * NB; t += TPB) Li[t] = V[t >> 7][t & (NB - 1)];
}

// Rows [0, rend) of columns [k0, k0 + kn): X <- X Linv^T (the inverse's
// column-block step, section 5): out[r][c] = sum_{k <= c} X[r][k] Linv[c][k].
constexpr int RTRSM_ROWS = 64, LDR = NB + 1;
constexpr size_t kRowsTrsmSmem = (size_t)(NB + RTRSM_ROWS) * LDR * sizeof(double);
__global__ void __launch_bounds__(TPB)
rows_trsm_kernel(double *__restrict__ A, long long lda, int rend, int k0, int kn,
                 const double *__restrict__ Linv, const int *__restrict__ info) {
    extern __shared__ double trsm_smem[];
    if (failed(info)) return;
    const int r0 = blockIdx.x * RTRSM_ROWS;
    double(*Li)[LDR] = reinterpret_cast<double(*)[LDR]>(trsm_smem);
    double(*P)[LDR] = reinterpret_cast<double(*)[LDR]>(trsm_smem + NB * LDR);
    const int tid = threadIdx.x;
    for (int t = tid; t < NB * NB; t += TPB) Li[t / NB][t % NB] = Linv[t];
    for (int t = tid; t < RTRSM_ROWS * NB; t += TPB) {
        const int r = t / NB, c = t % NB;
        P[r][c] = (r0 + r < rend && c < kn) ? A[(size_t)(r0 + r) * lda + k0 + c] : 0.0;
    }
    __syncthreads();
    const int c = tid & (NB - 1), rq = tid / NB;  // 2 row groups of 32 rows
    double out[32];
#pragma unroll
    for (int i = 0; i < 32; ++i) out[i] = 0.0;
    for (int k = 0; k <= c; ++k) {
        const double l = Li[c][k];
#pragma unroll
        for (int i = 0; i < 32; ++i) out[i] = fma(P[rq * 32 + i][k], l, out[i]);
    }
#pragma unroll
    for (int i = 0; i < 32; ++i) {
        const int r = r0 + rq * 32 + i;
        if (r < rend && c < kn) A[(size_t)r * lda + k0 + c] = out[i];
    }
}

// ---- 3. trailing update on the FP64 tensor cores ---------------------------
// C (m x m, stride ldc) -= P P^T on the triangle c <= r, P is (m x k).
// CTA tile 128 rows x 64 columns, 4 warps as 2 x 2, warp tile 64x32 =
// 8 x 4 m8n8 fragments; two CTAs fit per SM so one CTA's prologue and
// read-modify-write epilogue overlap the other's tensor-core work.
constexpr int SY_TM = 128, SY_TN = 64, SY_TK = 16, SY_LD = 20, SY_STAGES = 3, SY_TPB = 128;
constexpr int SY_STAGE_DOUBLES = (SY_TM + SY_TN) * SY_LD;
constexpr int SY_CLD = SY_TN + 8;  // row pitch of the epilogue's C tile in shared memory
static_assert(SY_TM * SY_CLD <= SY_STAGES * SY_STAGE_DOUBLES, "C tile must fit in the stages");
constexpr size_t kSyrkSmem = (size_t)SY_STAGES * SY_STAGE_DOUBLES * sizeof(double);

// Loads rows [row0, row0+ROWS) x k-columns [kc0, kc0+16) of P into a ROWS x
// SY_LD stage buffer; out-of-range rows / columns are zero-filled.
template <int ROWS, bool kAligned16>
__device__ __forceinline__ void syrk_load_tile(double *dst, const double *__restrict__ P,
                                               long long ldp, int m, int k, int row0, int kc0) {
    const int tid = threadIdx.x;
    if (kAligned16) {
#pragma unroll
        for (int i = 0; i < (ROWS * SY_TK / 2) / SY_TPB; ++i) {
            const int c = tid + i * SY_TPB;
            const int r = c >> 3, kc = (c & 7) * 2;
            const int gr = row0 + r, gk = kc0 + kc;
            int bytes = 0;
            if (gr < m) bytes = min(max(k - gk, 0), 2) * 8;
            const double *src = bytes ? P + (size_t)gr * ldp + gk : P;
            cp_async_16(dst + r * SY_LD + kc, src, bytes);
        }
    } else {
#pragma unroll
        for (int i = 0; i < (ROWS * SY_TK) / SY_TPB; ++i) {
            const int c = tid + i * SY_TPB;
            const int r = c >> 4, kc = c & 15;
            const int gr = row0 + r, gk = kc0 + kc;
            const bool ok = gr < m && gk < k;
            cp_async_8(dst + r * SY_LD + kc, ok ? P + (size_t)gr * ldp + gk : P, ok ? 8 : 0);
        }
    }
}

// Tile of TM x TN = TM/2 of the trailing update; a warp holds TM/2 x TN/2.
template <int TM>
struct SyTile {
    static constexpr int kM = TM, kN = TM / 2, kFr = TM / 16, kFc = TM / 32;
    static constexpr int kStage = (kM + kN) * SY_LD, kCld = kN + 8;
    static constexpr size_t kSmem = (size_t)SY_STAGES * kStage * sizeof(double);
    static_assert(kM * kCld <= SY_STAGES * kStage, "C tile must fit in the stages");
};

template <bool kAligned16, int TM>
__global__ void __launch_bounds__(SY_TPB, TM == 128 ? 2 : 4)
syrk_dmma_kernel(double *__restrict__ C, long long ldc, int m, const double *__restrict__ P,
                 long long ldp, int k, int strip_tiles, const int *__restrict__ info) {
    using T = SyTile<TM>;
    constexpr int kFr = T::kFr, kFc = T::kFc;  // fragments of a warp: rows, columns
    extern __shared__ __align__(16) double sy_smem[];
    pdl_wait();
    const long long t = blockIdx.x;
    int by, bx;
    if (strip_tiles > 0) {  // only the first strip_tiles column tiles of every row block
        by = (int)(t / strip_tiles);
        bx = (int)(t % strip_tiles);
        if (bx > 2 * by + 1) return;
    } else {  // tile t -> (row block by, column block bx of half its width), bx <= 2 by + 1
        by = (int)((sqrt(4.0 * (double)t + 1.0) - 1.0) * 0.5);
        while ((long long)by * by + by > t) --by;
        while ((long long)(by + 1) * (by + 1) + (by + 1) <= t) ++by;
        bx = (int)(t - (long long)by * by - by);
    }
    const int row0 = by * T::kM, col0 = bx * T::kN;
    if (col0 >= m || row0 >= m) return;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int wr = warp >> 1, wc = warp & 1;
    const int g = lane >> 2, tq = lane & 3;

    double acc[kFr][kFc][2];
#pragma unroll
    for (int i = 0; i < kFr; ++i)
#pragma unroll
        for (int j = 0; j < kFc; ++j) acc[i][j][0] = acc[i][j][1] = 0.0;

    const int nk = (k + SY_TK - 1) / SY_TK;
#pragma unroll
    for (int s = 0; s < SY_STAGES - 1; ++s) {
        if (s < nk) {
            double *st = sy_smem + s * T::kStage;
            syrk_load_tile<T::kM, kAligned16>(st, P, ldp, m, k, row0, s * SY_TK);
            syrk_load_tile<T::kN, kAligned16>(st + T::kM * SY_LD, P, ldp, m, k, col0, s * SY_TK);
        }
        cp_async_commit();
    }
    if (failed(info)) {  // read while the first stages are on their way
        cp_async_wait<0>();
        return;
    }
    for (int kt = 0; kt < nk; ++kt) {
        cp_async_wait<SY_STAGES - 2>();
        __syncthreads();
        const int nxt = kt + SY_STAGES - 1;
        if (nxt < nk) {
            double *st = sy_smem + (nxt % SY_STAGES) * T::kStage;
            syrk_load_tile<T::kM, kAligned16>(st, P, ldp, m, k, row0, nxt * SY_TK);
            syrk_load_tile<T::kN, kAligned16>(st + T::kM * SY_LD, P, ldp, m, k, col0, nxt * SY_TK);
        }
        cp_async_commit();
        const double *As = sy_smem + (kt % SY_STAGES) * T::kStage;
        const double *Bs = As + T::kM * SY_LD;
#pragma unroll
        for (int kk = 0; kk < SY_TK / 4; ++kk) {
            double a[kFr], b[kFc];
#pragma unroll
            for (int i = 0; i < kFr; ++i) a[i] = As[(wr * (T::kM / 2) + i * 8 + g) * SY_LD + kk * 4 + tq];
#pragma unroll
            for (int j = 0; j < kFc; ++j) b[j] = Bs[(wc * (T::kN / 2) + j * 8 + g) * SY_LD + kk * 4 + tq];
#pragma unroll
            for (int i = 0; i < kFr; ++i)
#pragma unroll
                for (int j = 0; j < kFc; ++j) dmma_8x8x4(acc[i][j], a[i], b[j]);
        }
    }
    cp_async_wait<0>();
    __syncthreads();  // every warp is done with the stage buffers
    // Epilogue through shared memory: one coalesced pass loads the C tile (all of
    // it in flight at once; loads to registers waited for memory every few rows),
    // the fragments are subtracted there, one coalesced masked pass stores it
    // (keeps the 64 read-modify-writes per thread from serialising).
    double *Cs = sy_smem;  // T::kM x T::kCld doubles, fits in the stage area
    const int tid = threadIdx.x;
    for (int e = tid; e < T::kM * (T::kN / 2); e += SY_TPB) {
        const int r = e / (T::kN / 2), c = (e % (T::kN / 2)) * 2;
        const int gr = row0 + r, gc = col0 + c;
        const double *src = C + (size_t)gr * ldc + gc;
        const bool in0 = gr < m && gc < m, in1 = gr < m && gc + 1 < m;
        cp_async_8(Cs + r * T::kCld + c, in0 ? src : C, in0 ? 8 : 0);
        cp_async_8(Cs + r * T::kCld + c + 1, in1 ? src + 1 : C, in1 ? 8 : 0);
    }
    cp_async_commit();
    cp_async_wait<0>();
    __syncthreads();
    // fragment (i, j): rows 8 i + g and columns 8 j + 2 tq + {0, 1} of the warp's tile
#pragma unroll
    for (int i = 0; i < kFr; ++i) {
        const int rl = wr * (T::kM / 2) + i * 8 + g;
#pragma unroll
        for (int j = 0; j < kFc; ++j) {
            const int cl = wc * (T::kN / 2) + j * 8 + 2 * tq;
            Cs[rl * T::kCld + cl] -= acc[i][j][0];
            Cs[rl * T::kCld + cl + 1] -= acc[i][j][1];
        }
    }
    __syncthreads();
    for (int e = tid; e < T::kM * (T::kN / 2); e += SY_TPB) {
        const int r = e / (T::kN / 2), c = (e % (T::kN / 2)) * 2;
        const int gr = row0 + r, gc = col0 + c;
        if (gr >= m) continue;
        double *dst = C + (size_t)gr * ldc + gc;
        if (gc < m && gc <= gr) dst[0] = Cs[r * T::kCld + c];
        if (gc + 1 < m && gc + 1 <= gr) dst[1] = Cs[r * T::kCld + c + 1];
    }
    pdl_launch_dependents();
}

// Launch with programmatic stream serialization when `pdl` is set (the kernel
// orders its dependent reads with griddepcontrol.wait).
template <typename... KArgs, typename... Args>
int launch_maybe_pdl(bool pdl, void (*kernel)(KArgs...), dim3 grid, dim3 block, size_t smem,
                     cudaStream_t st, const char *name, Args... args) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = grid;
    cfg.blockDim = block;
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = pdl ? 1 : 0;
    FMLB_TRY(cuda_status(cudaLaunchKernelEx(&cfg, kernel, args...), name));
    return launch_status(name);
}

template <bool kAligned16, int TM>
int launch_syrk_tile(double *C, long long ldc, int m, const double *P, long long ldp, int k,
                     int strip_cols, const int *info, cudaStream_t st, bool pdl) {
    using T = SyTile<TM>;
    static int attr_dev = -1;
    int dev = 0;
    FMLB_TRY(cuda_status(cudaGetDevice(&dev), "syrk: cudaGetDevice"));
    if (attr_dev != dev) {
        FMLB_TRY(cuda_status(cudaFuncSetAttribute(syrk_dmma_kernel<kAligned16, TM>,
                                                  cudaFuncAttributeMaxDynamicSharedMemorySize,
                                                  (int)T::kSmem), "syrk smem attribute"));
        attr_dev = dev;
    }
    const long long Tr = ceil_div(m, T::kM);
    const int strip_tiles = strip_cols > 0 ? ceil_div(std::min(strip_cols, m), T::kN) : 0;
    // full: row block by holds 2 by + 2 column tiles; strip: strip_tiles per row block
    const long long ntiles = strip_tiles ? Tr * strip_tiles : Tr * Tr + Tr;
    return launch_maybe_pdl(pdl, syrk_dmma_kernel<kAligned16, TM>, dim3((unsigned)ntiles),
                            dim3(SY_TPB), T::kSmem, st, "syrk_dmma_kernel", C, ldc, m, P, ldp, k,
                            strip_tiles, info);
}

// 128 x 64 tiles, or 64 x 32 ones while the former would fill their two slots
// per SM less than twice: then the last wave and a tile's own latency count
// (every entry's sum runs in the same order in both).
template <bool kAligned16>
int launch_syrk_impl(double *C, long long ldc, int m, const double *P, long long ldp, int k,
                     int strip_cols, const int *info, cudaStream_t st, bool pdl) {
    const long long Tr = ceil_div(m, 128);
    const long long big = strip_cols > 0 ? Tr * ceil_div(std::min(strip_cols, m), 64) : Tr * Tr + Tr;
    if (big < 4LL * sm_count())
        return launch_syrk_tile<kAligned16, 64>(C, ldc, m, P, ldp, k, strip_cols, info, st, pdl);
    return launch_syrk_tile<kAligned16, 128>(C, ldc, m, P, ldp, k, strip_cols, info, st, pdl);
}

// strip_cols = 0: lower triangle of the m x m block; > 0: only its first
// strip_cols columns (the lower part of that column strip).
int launch_syrk(double *C, long long ldc, int m, const double *P, long long ldp, int k,
                const int *info, cudaStream_t st, int strip_cols = 0, bool pdl = false) {
    if (m <= 0 || k <= 0) return FMLB_OK;
    if (((uintptr_t)P % 16 == 0) && (ldp % 2 == 0))
        return launch_syrk_impl<true>(C, ldc, m, P, ldp, k, strip_cols, info, st, pdl);
    return launch_syrk_impl<false>(C, ldc, m, P, ldp, k, strip_cols, info, st, pdl);
}

// ---- 4. triangular solves with the factor (potrs) ---------------------------
// One launch per direction. A CTA takes one block of 128 unknowns, in the order
// of the substitution by a ticket, and sums the contributions of the blocks
// before it as they appear:
//   forward   y_k = Linv_k (b_k - sum_{j < k} L_kj y_j)
//   backward  x_k = Linv_k^T (y_k - sum_{j > k} L_jk^T x_j)
// The next 128 x 128 block of the factor is loaded into registers before its
// vector block is waited for. A vector block is its own flag: the vector is
// filled with a bit pattern that no result has, and a reader polls each value
// until it is another. A CTA waits only for blocks that CTAs with lower tickets,
// started before it, own, so the first unfinished block can always proceed. All
// sums run in a fixed order (deterministic).
//
// Bound by the chain of n / 128 blocks per direction: one block's value through
// L2, 128 x 128 products with it and with the block inverse (kept in shared
// memory), about 2.4 us, and for large n by reading the factor (n = 32768: 0.87 ms a
// direction, 0.65 for the read); a launch per block and direction took 6.5 us.
constexpr int SV_WARPS = TPB / 32, SV_ROWS = NB / SV_WARPS;  // 8 warps of 16 rows
constexpr size_t kSolveSmem = ((size_t)NB * NB + (size_t)SV_WARPS * NB + 3 * NB) * sizeof(double);
constexpr size_t kSolveCounterBytes = 2 * sizeof(unsigned);  // behind y in the workspace
constexpr unsigned long long kSolveUnset = ~0ull;   // what a byte-wise fill with 0xff leaves

// The value at p once it is set; NaN when the wait takes more than `budget` clock
// cycles (the solution then holds NaN from there on), after which the thread's other
// waits don't wait any more.
__device__ __forceinline__ double solve_wait(const double *p, long long &budget) {
    const long long t0 = clock64();
    for (;;) {
        unsigned long long u;
        asm volatile("ld.relaxed.gpu.global.u64 %0, [%1];" : "=l"(u) : "l"(p) : "memory");
        if (u != kSolveUnset) return __longlong_as_double((long long)u);
        if (clock64() - t0 > budget) {
            budget = -1;
            return __longlong_as_double(0x7ff8000000000000LL);
        }
    }
}
__device__ __forceinline__ void solve_publish(double *p, double v) {
    unsigned long long u = (unsigned long long)__double_as_longlong(v);
    if (u == kSolveUnset) u = 0x7ff8000000000000ull;  // a NaN like any other
    asm volatile("st.relaxed.gpu.global.u64 [%0], %1;" ::"l"(p), "l"(u) : "memory");
}

// This CTA's place in the order (the counter starts at 0xffffffff). Past the last
// block, when solves that share a workspace overlap: the CTA has nothing to do.
__device__ __forceinline__ unsigned solve_ticket(unsigned *counter) {
    __shared__ unsigned place;
    if (threadIdx.x == 0) place = atomicAdd(counter, 1u) + 1u;
    __syncthreads();
    return place;
}

// The block inverse (zeros above the diagonal) into shared memory, asynchronously.
__device__ __forceinline__ void solve_load_inverse(double *Li, const double *__restrict__ Linv) {
    for (int t = threadIdx.x; t < NB * NB; t += TPB) cp_async_8(Li + t, Linv + t, 8);
    cp_async_commit();
}

// Rows warp * 16 .. + 15 of a 128 x 128 block, columns lane + 32 i: rows past
// `rows` and columns past `cols` as zeros.
__device__ __forceinline__ void solve_load_rows(double (&lv)[SV_ROWS][NB / 32],
                                                const double *__restrict__ block, long long lda,
                                                int rows, int cols) {
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
#pragma unroll
    for (int r = 0; r < SV_ROWS; ++r)
#pragma unroll
        for (int i = 0; i < NB / 32; ++i) {
            const int row = warp * SV_ROWS + r, c = lane + 32 * i;
            lv[r][i] = row < rows && c < cols ? block[(size_t)row * lda + c] : 0.0;
        }
}

// Sums of a[0 .. 15] over the warp's lanes: lane l returns that of a[l / 2].
__device__ __forceinline__ double warp_sums16(double (&a)[SV_ROWS]) {
    const int lane = threadIdx.x & 31;
    static_assert(SV_ROWS == 16, "four halvings");
#pragma unroll
    for (int m = 8; m >= 1; m >>= 1) {
        const bool up = lane & (2 * m);
#pragma unroll
        for (int q = 0; q < m; ++q) {
            const double give = up ? a[q] : a[q + m], keep = up ? a[q + m] : a[q];
            a[q] = keep + __shfl_xor_sync(0xffffffffu, give, 2 * m);
        }
    }
    return a[0] + __shfl_xor_sync(0xffffffffu, a[0], 1);
}

__global__ void __launch_bounds__(TPB, 1)
solve_forward_kernel(const double *__restrict__ L, long long lda, int n,
                     const double *__restrict__ Linv, const double *__restrict__ b,
                     double *y, unsigned *counter, long long budget, int withhold) {
    extern __shared__ __align__(16) double sv_smem[];
    double *Li = sv_smem, *v = Li + NB * NB, *yb = v + NB;  // yb: two blocks
    const unsigned place = solve_ticket(counter);
    if (place >= (unsigned)(n + NB - 1) / NB) return;
    const int k = (int)place, k0 = k * NB, kn = min(NB, n - k0);
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    solve_load_inverse(Li, Linv + (size_t)k * NB * NB);
    const double *rows = L + (size_t)k0 * lda;
    double lv[SV_ROWS][NB / 32], acc[SV_ROWS];
#pragma unroll
    for (int r = 0; r < SV_ROWS; ++r) acc[r] = 0.0;
    if (k > 0) solve_load_rows(lv, rows, lda, kn, NB);
    for (int j = 0; j < k; ++j) {
        double *yj = yb + (j & 1) * NB;
        if (tid < NB) yj[tid] = solve_wait(y + j * NB + tid, budget);
        __syncthreads();
#pragma unroll
        for (int i = 0; i < NB / 32; ++i) {
            const double yv = yj[lane + 32 * i];
#pragma unroll
            for (int r = 0; r < SV_ROWS; ++r) acc[r] = fma(lv[r][i], yv, acc[r]);
        }
        if (j + 1 < k) solve_load_rows(lv, rows + (j + 1) * NB, lda, kn, NB);
    }
    const int row = warp * SV_ROWS + (lane >> 1);
    const double bk = row < kn ? b[k0 + row] : 0.0;
    double s = warp_sums16(acc);
    if ((lane & 1) == 0) v[row] = bk - s;
    cp_async_wait<0>();
    __syncthreads();
#pragma unroll
    for (int r = 0; r < SV_ROWS; ++r) {
        double p = 0.0;
#pragma unroll
        for (int i = 0; i < NB / 32; ++i)
            p = fma(Li[(warp * SV_ROWS + r) * NB + lane + 32 * i], v[lane + 32 * i], p);
        acc[r] = p;
    }
    s = warp_sums16(acc);
    if ((lane & 1) == 0 && row < kn && !(withhold && k == 0)) solve_publish(y + k0 + row, s);
}

// Columns of the warps' partial sums p[i] (columns lane + 32 i), added in warp
// order: thread c < 128 returns column c's.
__device__ __forceinline__ double solve_column_sums(double *part, const double (&p)[NB / 32]) {
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
#pragma unroll
    for (int i = 0; i < NB / 32; ++i) part[warp * NB + lane + 32 * i] = p[i];
    __syncthreads();
    double s = 0.0;
    if (tid < NB)
#pragma unroll
        for (int w = 0; w < SV_WARPS; ++w) s += part[w * NB + tid];
    return s;
}

__global__ void __launch_bounds__(TPB, 1)
solve_backward_kernel(const double *__restrict__ L, long long lda, int n,
                      const double *__restrict__ Linv, const double *__restrict__ y, double *x,
                      unsigned *counter, long long budget, int withhold) {
    extern __shared__ __align__(16) double sv_smem[];
    double *Li = sv_smem, *v = Li + NB * NB, *xb = v + NB, *part = xb + 2 * NB;
    const int nblk = (n + NB - 1) / NB;
    const unsigned place = solve_ticket(counter);
    if (place >= (unsigned)nblk) return;
    const int k = nblk - 1 - (int)place, k0 = k * NB, kn = min(NB, n - k0);
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    solve_load_inverse(Li, Linv + (size_t)k * NB * NB);
    double lv[SV_ROWS][NB / 32], acc[2][NB / 32];
#pragma unroll
    for (int i = 0; i < NB / 32; ++i) acc[0][i] = acc[1][i] = 0.0;
    if (k < nblk - 1)
        solve_load_rows(lv, L + (size_t)(nblk - 1) * NB * lda + k0, lda, n - (nblk - 1) * NB, NB);
    for (int j = nblk - 1; j > k; --j) {
        double *xj = xb + (j & 1) * NB;
        if (tid < NB) xj[tid] = j * NB + tid < n ? solve_wait(x + j * NB + tid, budget) : 0.0;
        __syncthreads();
#pragma unroll
        for (int r = 0; r < SV_ROWS; ++r) {
            const double xv = xj[warp * SV_ROWS + r];
#pragma unroll
            for (int i = 0; i < NB / 32; ++i) acc[r & 1][i] = fma(lv[r][i], xv, acc[r & 1][i]);
        }
        if (j - 1 > k) solve_load_rows(lv, L + (size_t)(j - 1) * NB * lda + k0, lda, NB, NB);
    }
    double p[NB / 32];
#pragma unroll
    for (int i = 0; i < NB / 32; ++i) p[i] = acc[0][i] + acc[1][i];
    double s = solve_column_sums(part, p);
    if (tid < NB) v[tid] = tid < kn ? y[k0 + tid] - s : 0.0;
    cp_async_wait<0>();
    __syncthreads();
#pragma unroll
    for (int i = 0; i < NB / 32; ++i) acc[0][i] = acc[1][i] = 0.0;
#pragma unroll
    for (int r = 0; r < SV_ROWS; ++r) {
        const double vr = v[warp * SV_ROWS + r];
#pragma unroll
        for (int i = 0; i < NB / 32; ++i)
            acc[r & 1][i] = fma(Li[(warp * SV_ROWS + r) * NB + lane + 32 * i], vr, acc[r & 1][i]);
    }
#pragma unroll
    for (int i = 0; i < NB / 32; ++i) p[i] = acc[0][i] + acc[1][i];
    s = solve_column_sums(part, p);
    if (tid < kn && !(withhold && k == nblk - 1)) solve_publish(x + k0 + tid, s);
}

// ---- 5. inverse from the factor (potri) ------------------------------------
// inv(A) = L^-T L^-1 = V V^T with V = L^-T (upper triangular). V solves
// V L^T = I column block by column block, right-looking:
//   V[:, i] = U[:, i] Linv_ii^T                      (rows_trsm_kernel)
//   U[:, j] -= V[:, i] L[j, i]^T for blocks j > i    (gemm_nt_dmma_kernel)
// with U = I initially (only rows above block i+1 are non-zero). Then the
// lower triangle of V V^T (gemm_nt_dmma_kernel, triangle mode, k from the
// tile's first row on since V is upper triangular). 2n^3/3 flops, as LAPACK
// dpotri; both products on the FP64 tensor cores with the trailing update's
// tiles (128 x 64, DMMA m8n8k4, 3-stage cp.async).
//
// kTri = false: C (M x N) -= A B^T, A (M x K), B (N x K), all row-major.
// kTri = true:  C (M x M, triangle c <= r) = A A^T with A upper triangular
//               (B = A, the k-loop of row block r0 starts at r0).
template <bool kAligned16, bool kTri>
__global__ void __launch_bounds__(SY_TPB, 2)
gemm_nt_dmma_kernel(double *__restrict__ C, long long ldc, int M, int N,
                    const double *__restrict__ A, long long lda, const double *__restrict__ B,
                    long long ldb, int K, int tiles_n, const int *__restrict__ info) {
    extern __shared__ __align__(16) double sy_smem[];
    if (failed(info)) return;
    const long long t = blockIdx.x;
    int by, bx;
    if (kTri) {  // tile t -> (by, bx <= 2 by + 1), as the trailing update
        by = (int)((sqrt(4.0 * (double)t + 1.0) - 1.0) * 0.5);
        while ((long long)by * by + by > t) --by;
        while ((long long)(by + 1) * (by + 1) + (by + 1) <= t) ++by;
        bx = (int)(t - (long long)by * by - by);
    } else {
        by = (int)(t / tiles_n);
        bx = (int)(t % tiles_n);
    }
    const int row0 = by * SY_TM, col0 = bx * SY_TN;
    if (row0 >= M || col0 >= N) return;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int wr = warp >> 1, wc = warp & 1;
    const int g = lane >> 2, tq = lane & 3;

    double acc[8][4][2];
#pragma unroll
    for (int i = 0; i < 8; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) acc[i][j][0] = acc[i][j][1] = 0.0;

    const int kt0 = kTri ? row0 / SY_TK : 0;  // row0 is a multiple of SY_TK
    const int nk = (K + SY_TK - 1) / SY_TK;
#pragma unroll
    for (int s = 0; s < SY_STAGES - 1; ++s) {
        if (kt0 + s < nk) {
            double *st = sy_smem + s * SY_STAGE_DOUBLES;
            syrk_load_tile<SY_TM, kAligned16>(st, A, lda, M, K, row0, (kt0 + s) * SY_TK);
            syrk_load_tile<SY_TN, kAligned16>(st + SY_TM * SY_LD, B, ldb, N, K, col0,
                                              (kt0 + s) * SY_TK);
        }
        cp_async_commit();
    }
    for (int kt = kt0; kt < nk; ++kt) {
        cp_async_wait<SY_STAGES - 2>();
        __syncthreads();
        const int nxt = kt + SY_STAGES - 1;
        if (nxt < nk) {
            double *st = sy_smem + ((nxt - kt0) % SY_STAGES) * SY_STAGE_DOUBLES;
            syrk_load_tile<SY_TM, kAligned16>(st, A, lda, M, K, row0, nxt * SY_TK);
            syrk_load_tile<SY_TN, kAligned16>(st + SY_TM * SY_LD, B, ldb, N, K, col0,
                                              nxt * SY_TK);
        }
        cp_async_commit();
        const double *As = sy_smem + ((kt - kt0) % SY_STAGES) * SY_STAGE_DOUBLES;
        const double *Bs = As + SY_TM * SY_LD;
#pragma unroll
        for (int kk = 0; kk < SY_TK / 4; ++kk) {
            double a[8], b[4];
#pragma unroll
            for (int i = 0; i < 8; ++i) a[i] = As[(wr * 64 + i * 8 + g) * SY_LD + kk * 4 + tq];
#pragma unroll
            for (int j = 0; j < 4; ++j) b[j] = Bs[(wc * 32 + j * 8 + g) * SY_LD + kk * 4 + tq];
#pragma unroll
            for (int i = 0; i < 8; ++i)
#pragma unroll
                for (int j = 0; j < 4; ++j) dmma_8x8x4(acc[i][j], a[i], b[j]);
        }
    }
    cp_async_wait<0>();
    __syncthreads();
    double *Cs = sy_smem;  // SY_TM x SY_CLD
    const int tid = threadIdx.x;
    for (int e = tid; e < SY_TM * (SY_TN / 2); e += SY_TPB) {
        const int r = e / (SY_TN / 2), c = (e % (SY_TN / 2)) * 2;
        const int gr = row0 + r, gc = col0 + c;
        double v0 = 0.0, v1 = 0.0;
        if (!kTri && gr < M) {
            const double *src = C + (size_t)gr * ldc + gc;
            if (gc < N) v0 = src[0];
            if (gc + 1 < N) v1 = src[1];
        }
        Cs[r * SY_CLD + c] = v0;
        Cs[r * SY_CLD + c + 1] = v1;
    }
    __syncthreads();
#pragma unroll
    for (int i = 0; i < 8; ++i) {
        const int rl = wr * 64 + i * 8 + g;
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const int cl = wc * 32 + j * 8 + 2 * tq;
            if (kTri) {
                Cs[rl * SY_CLD + cl] += acc[i][j][0];
                Cs[rl * SY_CLD + cl + 1] += acc[i][j][1];
            } else {
                Cs[rl * SY_CLD + cl] -= acc[i][j][0];
                Cs[rl * SY_CLD + cl + 1] -= acc[i][j][1];
            }
        }
    }
    __syncthreads();
    for (int e = tid; e < SY_TM * (SY_TN / 2); e += SY_TPB) {
        const int r = e / (SY_TN / 2), c = (e % (SY_TN / 2)) * 2;
        const int gr = row0 + r, gc = col0 + c;
        if (gr >= M) continue;
        double *dst = C + (size_t)gr * ldc + gc;
        if (gc < N && (!kTri || gc <= gr)) dst[0] = Cs[r * SY_CLD + c];
        if (gc + 1 < N && (!kTri || gc + 1 <= gr)) dst[1] = Cs[r * SY_CLD + c + 1];
    }
}

template <bool kTri>
int launch_gemm_nt(double *C, long long ldc, int M, int N, const double *A, long long lda,
                   const double *B, long long ldb, int K, const int *info, cudaStream_t st) {
    if (M <= 0 || N <= 0 || K <= 0) return FMLB_OK;
    const bool al = (uintptr_t)A % 16 == 0 && lda % 2 == 0 && (uintptr_t)B % 16 == 0 &&
                    ldb % 2 == 0;
    const long long Tr = ceil_div(M, SY_TM);
    const int tiles_n = ceil_div(N, SY_TN);
    const long long ntiles = kTri ? Tr * Tr + Tr : Tr * tiles_n;
    if (al) {
        FMLB_TRY(cuda_status(cudaFuncSetAttribute(gemm_nt_dmma_kernel<true, kTri>,
                                                  cudaFuncAttributeMaxDynamicSharedMemorySize,
                                                  (int)kSyrkSmem), "gemm smem attribute"));
        gemm_nt_dmma_kernel<true, kTri><<<(unsigned)ntiles, SY_TPB, kSyrkSmem, st>>>(
            C, ldc, M, N, A, lda, B, ldb, K, tiles_n, info);
    } else {
        FMLB_TRY(cuda_status(cudaFuncSetAttribute(gemm_nt_dmma_kernel<false, kTri>,
                                                  cudaFuncAttributeMaxDynamicSharedMemorySize,
                                                  (int)kSyrkSmem), "gemm smem attribute"));
        gemm_nt_dmma_kernel<false, kTri><<<(unsigned)ntiles, SY_TPB, kSyrkSmem, st>>>(
            C, ldc, M, N, A, lda, B, ldb, K, tiles_n, info);
    }
    return launch_status("gemm_nt_dmma_kernel");
}

// V = I on the leading (n, n) block of a row-major buffer with stride ldv
__global__ void identity_kernel(double *__restrict__ V, long long ldv, int n) {
    const int r = blockIdx.y, c = blockIdx.x * blockDim.x + threadIdx.x;
    if (r < n && c < n) V[(size_t)r * ldv + c] = (r == c) ? 1.0 : 0.0;
}

int set_smem_attrs() {
    static int attr_dev = -1;
    int dev = 0;
    FMLB_TRY(cuda_status(cudaGetDevice(&dev), "potrf: cudaGetDevice"));
    if (attr_dev == dev) return FMLB_OK;
    FMLB_TRY(cuda_status(cudaFuncSetAttribute(potf2_block_kernel,
                                              cudaFuncAttributeMaxDynamicSharedMemorySize,
                                              (int)kPotf2Smem), "potf2 smem attribute"));
    FMLB_TRY(cuda_status(cudaFuncSetAttribute(panel_trsm_kernel,
                                              cudaFuncAttributeMaxDynamicSharedMemorySize,
                                              (int)kTrsmSmem), "trsm smem attribute"));
    FMLB_TRY(cuda_status(cudaFuncSetAttribute(rows_trsm_kernel,
                                              cudaFuncAttributeMaxDynamicSharedMemorySize,
                                              (int)kRowsTrsmSmem), "rows trsm smem attribute"));
    FMLB_TRY(cuda_status(cudaFuncSetAttribute(block_inverse_kernel,
                                              cudaFuncAttributeMaxDynamicSharedMemorySize,
                                              (int)kBlockInvSmem), "block inverse smem attribute"));
    FMLB_TRY(cuda_status(cudaFuncSetAttribute(solve_forward_kernel,
                                              cudaFuncAttributeMaxDynamicSharedMemorySize,
                                              (int)kSolveSmem), "solve smem attribute"));
    FMLB_TRY(cuda_status(cudaFuncSetAttribute(solve_backward_kernel,
                                              cudaFuncAttributeMaxDynamicSharedMemorySize,
                                              (int)kSolveSmem), "solve smem attribute"));
    attr_dev = dev;
    return FMLB_OK;
}

}  // namespace
}  // namespace fmlb

extern "C" size_t fmlb_potrf_workspace_bytes(int n) {
    if (n <= 0) return 256;
    const size_t nblk = (size_t)(n + fmlb::NB - 1) / fmlb::NB;
    return nblk * fmlb::NB * fmlb::NB * sizeof(double) +
           ((size_t)n * sizeof(double) + fmlb::kSolveCounterBytes + 255) / 256 * 256;
}

// Per host thread, device and caller stream: the high-priority stream that
// runs the panel chain (strip update, diagonal block, panel solve) of the
// lookahead, and two events to order it against the caller's stream.
// Factorisations issued on different caller streams get different panel
// streams, so they can overlap: one's narrow final steps run under another's
// bulk updates. Past kPerCaller caller streams a thread shares one entry per
// device; its panel stream then serialises those callers' panel chains, which
// is slower but still ordered correctly, since every wait names the event
// recorded by the same call. The streams and events live for the life of the
// host thread and do not survive cudaDeviceReset: a process that resets a
// device must not factor on it again from the same thread.
struct Lookahead {
    cudaStream_t panel = nullptr;
    cudaEvent_t main_done = nullptr, panel_done = nullptr;
};

static int lookahead_for(cudaStream_t caller, Lookahead **out) {
    using namespace fmlb;
    constexpr int kPerCaller = 16;
    struct Entry {
        int dev = -1;
        cudaStream_t caller = nullptr;
        Lookahead la;
    };
    static thread_local Entry by_caller[kPerCaller];
    static thread_local Lookahead shared_per_dev[64];
    int dev = 0;
    FMLB_TRY(cuda_status(cudaGetDevice(&dev), "fmlb_potrf_f64: cudaGetDevice"));
    FMLB_REQUIRE(dev >= 0 && dev < 64, "fmlb_potrf_f64: device %d out of range", dev);
    Lookahead *lp = nullptr;
    for (int i = 0; i < kPerCaller && !lp; ++i)
        if (by_caller[i].dev == dev && by_caller[i].caller == caller) lp = &by_caller[i].la;
    for (int i = 0; i < kPerCaller && !lp; ++i)
        if (by_caller[i].dev < 0) {
            by_caller[i].dev = dev;
            by_caller[i].caller = caller;
            lp = &by_caller[i].la;
        }
    if (!lp) lp = &shared_per_dev[dev];
    Lookahead &L = *lp;
    if (!L.panel) {
        int lo = 0, hi = 0;
        FMLB_TRY(cuda_status(cudaDeviceGetStreamPriorityRange(&lo, &hi), "stream priorities"));
        FMLB_TRY(cuda_status(cudaStreamCreateWithPriority(&L.panel, cudaStreamNonBlocking, hi),
                             "fmlb_potrf_f64: panel stream"));
        FMLB_TRY(cuda_status(cudaEventCreateWithFlags(&L.main_done, cudaEventDisableTiming),
                             "fmlb_potrf_f64: event"));
        FMLB_TRY(cuda_status(cudaEventCreateWithFlags(&L.panel_done, cudaEventDisableTiming),
                             "fmlb_potrf_f64: event"));
    }
    *out = &L;
    return FMLB_OK;
}

static int panel_factor(double *A, long long lda, int n, int k0, double *Li, int *info,
                        cudaStream_t st, bool after_kernel) {
    using namespace fmlb;
    const int kn = std::min(NB, n - k0);
    // the chain of one outer panel: each kernel follows the previous one of
    // the stream with a programmatic dependency; the first block of an outer
    // panel is launched normally, as what precedes it may be a memset or an
    // event wait rather than a kernel of the chain
    FMLB_TRY(launch_maybe_pdl(after_kernel, potf2_block_kernel, dim3(1), dim3(TPB), kPotf2Smem, st,
                              "potf2_block_kernel", A, lda, k0, kn, Li, info));
    const int rest = n - k0 - kn;
    if (rest > 0)
        FMLB_TRY(launch_maybe_pdl(
            true, panel_trsm_kernel, dim3(std::min(ceil_div(rest, TRSM_ROWS), sm_count())),
            dim3(TPB), kTrsmSmem, st, "panel_trsm_kernel", A, lda, n, k0, (const double *)Li,
            (const int *)info));
    return FMLB_OK;
}

// Factor the outer panel of columns [K0, K0 + width) on stream st: per inner
// panel of NB columns, the diagonal block and the panel solve (all rows below),
// then an update inside the outer panel. The updates are those of recursive
// halving: after j inner panels, the last s = lowest set bit of j of them
// update the next s, so half of the work runs with k = width / 2 and a quarter
// with k = width / 4 (28 and 24 TFLOP/s) instead of all of it with k = NB (17).
static int factor_outer_panel(double *A, long long lda, int n, int K0, int width, double *Linv,
                              int *info, cudaStream_t st) {
    using namespace fmlb;
    const int end = std::min(K0 + width, n);
    for (int k0 = K0; k0 < end; k0 += NB) {
        FMLB_TRY(panel_factor(A, lda, n, k0, Linv + (size_t)(k0 / NB) * NB * NB, info, st,
                              k0 > K0));
        const size_t b = (size_t)(k0 + NB);
        const int rem = end - (int)b;
        if (rem > 0) {
            const int j = (int)(b - K0) / NB, s = (j & -j) * NB;
            FMLB_TRY(launch_syrk(A + b * lda + b, lda, n - (int)b, A + b * lda + b - s, lda, s, info,
                                 st, std::min(s, rem), true));
        }
    }
    return FMLB_OK;
}

// Outer panel width: wide panels give the trailing update a long k-loop
// (k = 512: ~28 TFLOP/s against ~17 at k = 128 on B200) and fewer steps.
// Measured at n = 32768 on B200: 455 ms (512), 436 ms (768), 429 ms (1024).
static int outer_width(int n) {
    return n >= 16384 ? 8 * fmlb::NB : n >= 8192 ? 4 * fmlb::NB : 2 * fmlb::NB;
}

// Two-level blocked factorisation with a lookahead of depth one. For outer
// panel K (factored), with outer block K+1 the next:
//   panel stream:  strip update of outer block K+1 by panel K (k = width),
//                  then the factorisation of outer panel K+1;
//   caller stream: update of the trailing matrix past block K+1 by panel K.
// The two regions are disjoint, so the panel chain runs under the bulk update.
// With `oz` set, the strip and bulk updates run on the int8 tensor cores
// (ozaki_f64.cu): panel K's rows below it are split into digit planes once,
// on the caller stream, before either update reads them; the next split waits
// for the panel stream, so the planes are never overwritten while read.
static int potrf_blocked(double *A, long long lda, int n, void *work, int *info,
                         cudaStream_t st, const fmlb::OzakiSlices *oz) {
    using namespace fmlb;
    FMLB_TRY(set_smem_attrs());
    Lookahead *la = nullptr;
    FMLB_TRY(lookahead_for(st, &la));
    double *Linv = static_cast<double *>(work);
    const int W = outer_width(n);
    const int nob = ceil_div(n, W);
    FMLB_TRY(factor_outer_panel(A, lda, n, 0, W, Linv, info, st));
    bool panel_used = false;
    for (int K = 0; K + 1 < nob; ++K) {
        const int K0 = K * W;
        const size_t base = (size_t)(K0 + W);  // first row / column of outer block K+1
        const int rest = n - (int)base;
        if (panel_used)  // outer panel K was factored on the panel stream
            FMLB_TRY(cuda_status(cudaStreamWaitEvent(st, la->panel_done, 0), "wait panel"));
        if (oz)  // digit planes of panel K, rows [base, n)
            FMLB_TRY(ozaki_split(A + base * lda + K0, lda, rest, W, *oz, info, st));
        FMLB_TRY(cuda_status(cudaEventRecord(la->main_done, st), "record main"));
        FMLB_TRY(cuda_status(cudaStreamWaitEvent(la->panel, la->main_done, 0), "wait main"));
        if (oz)
            FMLB_TRY(ozaki_syrk(A + base * lda + base, lda, rest, *oz, 0, W, info, la->panel));
        else
            FMLB_TRY(launch_syrk(A + base * lda + base, lda, rest, A + base * lda + K0, lda, W,
                                 info, la->panel, W));
        FMLB_TRY(factor_outer_panel(A, lda, n, (int)base, W, Linv, info, la->panel));
        FMLB_TRY(cuda_status(cudaEventRecord(la->panel_done, la->panel), "record panel"));
        panel_used = true;
        const int rest2 = rest - W;
        if (rest2 > 0) {
            const size_t b2 = base + W;
            if (oz)
                FMLB_TRY(ozaki_syrk(A + b2 * lda + b2, lda, rest2, *oz, W, 0, info, st));
            else
                FMLB_TRY(launch_syrk(A + b2 * lda + b2, lda, rest2, A + b2 * lda + K0, lda, W,
                                     info, st));
        }
    }
    if (panel_used)
        FMLB_TRY(cuda_status(cudaStreamWaitEvent(st, la->panel_done, 0), "join panel stream"));
    block_inverse_kernel<<<ceil_div(n, NB), TPB, kBlockInvSmem, st>>>(A, lda, n, Linv, info);
    return launch_status("block_inverse_kernel");
}

extern "C" int fmlb_potrf_f64(double *A, long long lda, int n, void *work, int *info,
                              void *stream) {
    using namespace fmlb;
    cudaStream_t st = FMLB_STREAM(stream);
    FMLB_REQUIRE(n >= 0 && lda >= n, "fmlb_potrf_f64: bad n=%d / lda=%lld", n, lda);
    FMLB_REQUIRE(info, "fmlb_potrf_f64: info pointer is null");
    FMLB_TRY(cuda_status(cudaMemsetAsync(info, 0, sizeof(int), st), "fmlb_potrf_f64: clear info"));
    if (n == 0) return FMLB_OK;
    FMLB_REQUIRE(A && work, "fmlb_potrf_f64: null pointer");
    return potrf_blocked(A, lda, n, work, info, st, nullptr);
}

extern "C" size_t fmlb_potrf_ozaki_workspace_bytes(int n, int nslices) {
    if (n <= 0 || nslices <= 0) return 256;
    const int W = outer_width(n);
    // a multiple of 256, so that workspaces laid side by side stay aligned (the
    // digit data of an odd n ends on 4 bytes, and a second workspace right behind
    // it held its doubles misaligned)
    return ((fmlb_potrf_workspace_bytes(n) + 255) / 256 * 256 +
            fmlb::ozaki_slice_bytes(n, W, nslices) + 255) / 256 * 256;
}

extern "C" int fmlb_potrf_ozaki_f64(double *A, long long lda, int n, int nslices, void *work,
                                    size_t ws_bytes, int *info, void *stream) {
    using namespace fmlb;
    cudaStream_t st = FMLB_STREAM(stream);
    FMLB_REQUIRE(n >= 0 && lda >= n, "fmlb_potrf_ozaki_f64: bad n=%d / lda=%lld", n, lda);
    FMLB_REQUIRE(nslices >= 1 && nslices <= OZAKI_MAX_SLICES,
                 "fmlb_potrf_ozaki_f64: nslices must be 1..%d", OZAKI_MAX_SLICES);
    FMLB_REQUIRE(info, "fmlb_potrf_ozaki_f64: info pointer is null");
    FMLB_TRY(cuda_status(cudaMemsetAsync(info, 0, sizeof(int), st),
                         "fmlb_potrf_ozaki_f64: clear info"));
    if (n == 0) return FMLB_OK;
    FMLB_REQUIRE(A && work, "fmlb_potrf_ozaki_f64: null pointer");
    const size_t need = fmlb_potrf_ozaki_workspace_bytes(n, nslices);
    if (ws_bytes < need) {
        set_error("fmlb_potrf_ozaki_f64: workspace %zu < %zu bytes", ws_bytes, need);
        return FMLB_ENOMEM;
    }
    OzakiSlices oz;
    const size_t off = (fmlb_potrf_workspace_bytes(n) + 255) / 256 * 256;
    FMLB_TRY(ozaki_bind(static_cast<char *>(work) + off, n, outer_width(n), nslices, oz));
    return potrf_blocked(A, lda, n, work, info, st, &oz);
}

extern "C" int fmlb_potrs_f64(const double *L, long long lda, int n, const void *work, double *x,
                              void *stream) {
    using namespace fmlb;
    cudaStream_t st = FMLB_STREAM(stream);
    FMLB_REQUIRE(n >= 0 && lda >= n, "fmlb_potrs_f64: bad n=%d / lda=%lld", n, lda);
    if (n == 0) return FMLB_OK;
    FMLB_REQUIRE(L && work && x, "fmlb_potrs_f64: null pointer");
    FMLB_TRY(set_smem_attrs());
    const double *Linv = static_cast<const double *>(work);
    const size_t nblk = (size_t)(n + NB - 1) / NB;
    // y and the two counters live after the inverted blocks in the workspace
    // (written by potrs only)
    double *y = const_cast<double *>(Linv + nblk * NB * NB);
    unsigned *counters = reinterpret_cast<unsigned *>(y + n);
    FMLB_TRY(cuda_status(cudaMemsetAsync(y, 0xff, (size_t)n * sizeof(double) + kSolveCounterBytes,
                                         st), "fmlb_potrs_f64: fill"));
    const tc::TestHooks hooks = tc::test_hooks();
    const unsigned grid = (unsigned)nblk + (hooks.extra_block ? 1 : 0);
    solve_forward_kernel<<<grid, TPB, kSolveSmem, st>>>(L, lda, n, Linv, x, y, counters,
                                                        hooks.wait_budget, hooks.withhold);
    FMLB_TRY(launch_status("solve_forward_kernel"));
    FMLB_TRY(cuda_status(cudaMemsetAsync(x, 0xff, (size_t)n * sizeof(double), st),
                         "fmlb_potrs_f64: fill"));
    solve_backward_kernel<<<grid, TPB, kSolveSmem, st>>>(L, lda, n, Linv, y, x, counters + 1,
                                                         hooks.wait_budget, hooks.withhold);
    return launch_status("solve_backward_kernel");
}

extern "C" int fmlb_syrk_lower_f64(double *C, long long ldc, int m, const double *P,
                                   long long ldp, int k, int strip_cols, const int *info,
                                   void *stream) {
    using namespace fmlb;
    FMLB_REQUIRE(m >= 0 && k >= 0 && ldc >= m && ldp >= k && strip_cols >= 0,
                 "fmlb_syrk_lower_f64: bad sizes");
    if (m == 0 || k == 0) return FMLB_OK;
    FMLB_REQUIRE(C && P, "fmlb_syrk_lower_f64: null pointer");
    return launch_syrk(C, ldc, m, P, ldp, k, info, FMLB_STREAM(stream), strip_cols);
}

extern "C" int fmlb_potri_f64(double *A, long long lda, int n, const void *work, double *V,
                              long long ldv, const int *info, void *stream) {
    using namespace fmlb;
    cudaStream_t st = FMLB_STREAM(stream);
    FMLB_REQUIRE(n >= 0 && lda >= n && ldv >= n, "fmlb_potri_f64: bad n=%d / lda / ldv", n);
    if (n == 0) return FMLB_OK;
    FMLB_REQUIRE(A && work && V, "fmlb_potri_f64: null pointer");
    FMLB_REQUIRE(n <= 65535, "fmlb_potri_f64: n=%d above 65535", n);
    FMLB_TRY(set_smem_attrs());
    const double *Linv = static_cast<const double *>(work);
    identity_kernel<<<dim3(ceil_div(n, 256), n), 256, 0, st>>>(V, ldv, n);
    FMLB_TRY(launch_status("identity_kernel"));
    for (int k0 = 0, kb = 0; k0 < n; k0 += NB, ++kb) {
        const int kn = std::min(NB, n - k0), R = k0 + kn;
        rows_trsm_kernel<<<ceil_div(R, RTRSM_ROWS), TPB, kRowsTrsmSmem, st>>>(
            V, ldv, R, k0, kn, Linv + (size_t)kb * NB * NB, info);
        FMLB_TRY(launch_status("rows_trsm_kernel"));
        if (R < n)
            FMLB_TRY(launch_gemm_nt<false>(V + R, ldv, R, n - R, V + k0, ldv,
                                           A + (size_t)R * lda + k0, lda, kn, info, st));
    }
    return launch_gemm_nt<true>(A, lda, n, n, V, ldv, V, ldv, n, info, st);
}
