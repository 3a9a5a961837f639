// FP64 distance tile shared by the kernel matrices, the fused prediction and
// the atomic vector kernels.
//
// A CTA of 128 threads holds a (16 RI) x 64 tile of row pairs, 4 RI rows x 64
// columns per warp and RI x 8 pairs per thread in registers. Features are
// staged 8 (or 16) at a time in shared memory, transposed, by asynchronous copies three
// chunks ahead. Features are added in ascending order by one thread per pair,
// so a pair's distance does not depend on the tile that it falls in.
//
// Bound by FP64 issue: two instructions (three without contraction) per pair
// and feature. A 64-bit shared load takes two wavefronts whatever is broadcast,
// so 4 x 8 pairs per thread need 24 of them per 32 cycles of FP64 work; 4 x 4
// pairs need as many as there are cycles. The copies go past the registers,
// which leaves room for 16 warps per SM (a warp cannot issue FP64 instructions
// back to back). Gaussian, 8191 x 8191, d = 435, symmetric, 3 sigmas: 2.22 ms
// (71 % of the FP64 issue rate); 2.41 ms with 64 x 64 tiles of 4 x 4 pairs and a
// single buffer, 2.38 with 4 x 4 pairs and these copies.
#pragma once

#include <cuda_runtime.h>

namespace fmlb {
namespace dist {

constexpr int DT_TPB = 128, DT_N = 64, DT_BUFS = 4;
constexpr int DT_P = DT_N + 2;  // row pitch: the transposing copies spread

// Features of a chunk, row pitch of A's part of it, doubles of the stage. Where the
// tiles are 16 rows high few CTAs run, and the memory's latency per chunk is what
// they take: 16 features, in a stage that would leave no room for four CTAs.
template <int RI>
__host__ __device__ constexpr int chunk() { return RI == 1 ? 16 : 8; }
template <int RI>
__host__ __device__ constexpr int pitch_a() { return RI == 1 ? 18 : DT_P; }
template <int RI>
__host__ __device__ constexpr int stage_doubles() {
    return DT_BUFS * chunk<RI>() * (pitch_a<RI>() + DT_P);
}

enum Op { kSquare = 0, kAbs = 1, kSquareUnfused = 2 };

template <Op kOp>
__device__ __forceinline__ double add_term(double acc, double a, double b) {
    const double e = __dsub_rn(a, b);
    if (kOp == kSquare) return fma(e, e, acc);
    return __dadd_rn(acc, kOp == kAbs ? fabs(e) : __dmul_rn(e, e));
}

__device__ __forceinline__ void copy8_async(double *dst, const double *src, bool valid) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;\n" ::"r"(
                     (unsigned)__cvta_generic_to_shared(dst)),
                 "l"(src), "r"(valid ? 8 : 0)
                 : "memory");
}

// First row and column of this thread's pairs: acc[i][j] belongs to row
// first_row<RI>() + 4 i and column first_col() + 8 j of the tile.
template <int RI>
__device__ __forceinline__ int first_row() {
    return (threadIdx.x >> 5) * 4 * RI + ((threadIdx.x & 31) >> 3);
}
__device__ __forceinline__ int first_col() {
    return threadIdx.x & 7;
}

// Distance sums of the tile's first nr rows and nc columns; the rest is left
// undefined. row_a(r) / row_b(c) give the row's features, d of them.
// Synchronises before the stage is first written; the caller synchronises
// before the stage is used otherwise.
template <Op kOp, int RI, typename RowA, typename RowB>
__device__ __forceinline__ void dist_tile(double (&acc)[RI][8], double *stage, RowA row_a,
                                          RowB row_b, int nr, int nc, int d) {
    constexpr int kRows = 16 * RI, kK = chunk<RI>(), kPA = pitch_a<RI>();
    constexpr int kPass = DT_TPB / kK, kChunk = kK * (kPA + DT_P);
    const int tid = threadIdx.x;
    const int r0 = first_row<RI>(), c0 = first_col();
    // loader: the chunk's features of kPass rows a pass
    const int lk = tid & (kK - 1), lr = tid / kK;
    const double *pa[kRows / kPass], *pb[DT_N / kPass];
#pragma unroll
    for (int q = 0; q < kRows / kPass; ++q)
        pa[q] = lr + kPass * q < nr ? row_a(lr + kPass * q) : nullptr;
#pragma unroll
    for (int q = 0; q < DT_N / kPass; ++q)
        pb[q] = lr + kPass * q < nc ? row_b(lr + kPass * q) : nullptr;
    const double *any = row_b(0);  // a valid address for the zero-filled copies
    const int nk = (d + kK - 1) / kK;
    auto copy = [&](int chunk) {
        if (chunk < nk) {
            double *As = stage + (chunk % DT_BUFS) * kChunk, *Bs = As + kK * kPA;
            const int f = chunk * kK + lk;
#pragma unroll
            for (int q = 0; q < kRows / kPass; ++q) {
                const bool ok = pa[q] && f < d;
                copy8_async(As + lk * kPA + lr + kPass * q, ok ? pa[q] + f : any, ok);
            }
#pragma unroll
            for (int q = 0; q < DT_N / kPass; ++q) {
                const bool ok = pb[q] && f < d;
                copy8_async(Bs + lk * DT_P + lr + kPass * q, ok ? pb[q] + f : any, ok);
            }
        }
        asm volatile("cp.async.commit_group;\n" ::: "memory");
    };
#pragma unroll
    for (int i = 0; i < RI; ++i)
#pragma unroll
        for (int j = 0; j < 8; ++j) acc[i][j] = 0.0;
    // columns of 8 that this warp has work in (the same for its 32 lanes)
    const int jn = (tid >> 5) * 4 * RI < nr ? (nc + 7) / 8 : 0;
    __syncthreads();  // the stage is free
#pragma unroll
    for (int c = 0; c < DT_BUFS - 1; ++c) copy(c);
    for (int c = 0; c < nk; ++c) {
        asm volatile("cp.async.wait_group %0;\n" ::"n"(DT_BUFS - 2) : "memory");
        __syncthreads();  // chunk c has landed, and chunk c - 1 is no longer read
        copy(c + DT_BUFS - 1);
        const double *As = stage + (c % DT_BUFS) * kChunk + r0;
        const double *Bs = stage + (c % DT_BUFS) * kChunk + kK * kPA + c0;
        if (jn >= 8) {
#pragma unroll
            for (int kk = 0; kk < kK; ++kk) {
                double a[RI], b[8];
#pragma unroll
                for (int i = 0; i < RI; ++i) a[i] = As[kk * kPA + 4 * i];
#pragma unroll
                for (int j = 0; j < 8; ++j) b[j] = Bs[kk * DT_P + 8 * j];
#pragma unroll
                for (int i = 0; i < RI; ++i)
#pragma unroll
                    for (int j = 0; j < 8; ++j) acc[i][j] = add_term<kOp>(acc[i][j], a[i], b[j]);
            }
        } else if (jn > 0) {
#pragma unroll 2
            for (int kk = 0; kk < kK; ++kk) {
                double a[RI];
#pragma unroll
                for (int i = 0; i < RI; ++i) a[i] = As[kk * kPA + 4 * i];
#pragma unroll
                for (int j = 0; j < 7; ++j) {
                    if (j < jn) {
                        const double b = Bs[kk * DT_P + 8 * j];
#pragma unroll
                        for (int i = 0; i < RI; ++i)
                            acc[i][j] = add_term<kOp>(acc[i][j], a[i], b);
                    }
                }
            }
        }
    }
}

}  // namespace dist
}  // namespace fmlb
