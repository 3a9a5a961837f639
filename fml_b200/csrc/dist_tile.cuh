// FP64 distance tile shared by the kernel matrices, the fused prediction and
// the atomic vector kernels.
//
// A CTA of 128 threads holds a tile of row pairs, 64 columns wide, RI x CJ pairs per
// thread in registers. Features are staged 8 (or 16) at a time in shared memory,
// transposed, by asynchronous copies three chunks ahead. Features are added in
// ascending order by one thread per pair, so a pair's distance does not depend on
// the tile that it falls in.
//
// Bound by FP64 issue: two instructions (three without contraction) per pair
// and feature. A 64-bit shared load takes two wavefronts whatever is broadcast,
// so 4 x 8 pairs per thread need 24 of them per 32 cycles of FP64 work; 4 x 4
// pairs need as many as there are cycles, 2 x 8 pairs 20 per 16. The copies go past
// the registers, which leaves room for 16 warps per SM (a warp cannot issue FP64
// instructions back to back); they are issued behind a chunk's arithmetic, since
// between the barrier and the chunk's first loads every warp waited for their
// address arithmetic. Gaussian, 8191 x 8191, d = 435, symmetric, 3 sigmas: 2.16 ms
// (73 % of the FP64 issue rate); 2.41 ms with 64 x 64 tiles of 4 x 4 pairs, 256 threads
// and a single buffer, 2.38 with 4 x 4 pairs and these copies.
#pragma once

#include <cuda_runtime.h>

namespace fmlb {
namespace dist {

constexpr int DT_TPB = 128, DT_N = 64, DT_BUFS = 4;
constexpr int DT_P = DT_N + 2;  // row pitch: the transposing copies spread

// A warp holds 4 RI rows x 8 CJ columns; the warps lie side by side over the 64
// columns, then below one another.
template <int CJ>
__host__ __device__ constexpr int warps_across() { return DT_N / (8 * CJ); }
template <int RI, int CJ>
__host__ __device__ constexpr int tile_rows() {
    return 4 * RI * (DT_TPB / 32) / warps_across<CJ>();
}

// Features of a chunk, row pitch of A's part of it, doubles of the stage. Where the
// tiles are 16 rows high few CTAs run, and the memory's latency per chunk is what
// they take: 16 features, in a stage of 42 KB that leaves room for five CTAs per SM.
template <int RI>
__host__ __device__ constexpr int chunk() { return RI == 1 ? 16 : 8; }
template <int RI, int CJ>
__host__ __device__ constexpr int pitch_a() { return tile_rows<RI, CJ>() + 2; }
template <int RI, int CJ>
__host__ __device__ constexpr int stage_doubles() {
    return DT_BUFS * chunk<RI>() * (pitch_a<RI, CJ>() + DT_P);
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
// first_row<RI, CJ>() + 4 i and column first_col<CJ>() + 8 j of the tile.
template <int RI, int CJ>
__device__ __forceinline__ int first_row() {
    return (threadIdx.x >> 5) / warps_across<CJ>() * 4 * RI + ((threadIdx.x & 31) >> 3);
}
template <int CJ>
__device__ __forceinline__ int first_col() {
    return (threadIdx.x >> 5) % warps_across<CJ>() * 8 * CJ + (threadIdx.x & 7);
}

// A chunk's features for the thread's first N columns (8 apart).
template <Op kOp, int N, int RI, int CJ>
__device__ __forceinline__ void add_chunk(double (&acc)[RI][CJ], const double *As,
                                          const double *Bs) {
#pragma unroll
    for (int kk = 0; kk < chunk<RI>(); ++kk) {
        double a[RI], b[N];
#pragma unroll
        for (int i = 0; i < RI; ++i) a[i] = As[kk * pitch_a<RI, CJ>() + 4 * i];
#pragma unroll
        for (int j = 0; j < N; ++j) b[j] = Bs[kk * DT_P + 8 * j];
#pragma unroll
        for (int i = 0; i < RI; ++i)
#pragma unroll
            for (int j = 0; j < N; ++j) acc[i][j] = add_term<kOp>(acc[i][j], a[i], b[j]);
    }
}

// Distance sums of the tile's first nr rows and nc columns (at least one each); the
// rest is left undefined. row_a(r) / row_b(c) give the row's features, d of them.
// kNarrow: tiles with few columns are common, so a warp works on the columns there
// are, two steps of 8 at a time (with a loop over them and a test in it one such tile
// held up a whole call: 1700 rows symmetric, 36 in the last tile, 109 us, 1787 rows 84);
// the code of the other widths costs the full one 1 %.
// Synchronises before the stage is first written; the caller synchronises
// before the stage is used otherwise.
template <Op kOp, bool kNarrow, int RI, int CJ, typename RowA, typename RowB>
__device__ __forceinline__ void dist_tile(double (&acc)[RI][CJ], double *stage, RowA row_a,
                                          RowB row_b, int nr, int nc, int d) {
    constexpr int kRows = tile_rows<RI, CJ>(), kK = chunk<RI>(), kPA = pitch_a<RI, CJ>();
    constexpr int kPass = DT_TPB / kK, kChunk = kK * (kPA + DT_P);
    // 4 x 4 pairs: rows and columns past the tile's repeat its last, which saves the
    // test of every copy (4 % of such a tile, but registers that 4 x 8 pairs lack)
    constexpr bool kRepeat = CJ < 8;
    const int tid = threadIdx.x;
    const int r0 = first_row<RI, CJ>(), c0 = first_col<CJ>();
    // loader: the chunk's features of kPass rows a pass
    const int lk = tid & (kK - 1), lr = tid / kK;
    const double *pa[kRows / kPass], *pb[DT_N / kPass];
#pragma unroll
    for (int q = 0; q < kRows / kPass; ++q) {
        const int r = lr + kPass * q;
        pa[q] = kRepeat ? row_a(min(r, nr - 1)) : r < nr ? row_a(r) : nullptr;
    }
#pragma unroll
    for (int q = 0; q < DT_N / kPass; ++q) {
        const int c = lr + kPass * q;
        pb[q] = kRepeat ? row_b(min(c, nc - 1)) : c < nc ? row_b(c) : nullptr;
    }
    const double *any = row_b(0);  // a valid address for the zero-filled copies
    const int nk = (d + kK - 1) / kK;
    auto copy = [&](int chunk) {
        if (chunk < nk) {
            double *As = stage + (chunk % DT_BUFS) * kChunk, *Bs = As + kK * kPA;
            const int k = chunk * kK + lk, f = kRepeat ? (k < d ? k : 0) : k;
#pragma unroll
            for (int q = 0; q < kRows / kPass; ++q) {
                const bool ok = k < d && (kRepeat || pa[q]);
                copy8_async(As + lk * kPA + lr + kPass * q, kRepeat || ok ? pa[q] + f : any, ok);
            }
#pragma unroll
            for (int q = 0; q < DT_N / kPass; ++q) {
                const bool ok = k < d && (kRepeat || pb[q]);
                copy8_async(Bs + lk * DT_P + lr + kPass * q, kRepeat || ok ? pb[q] + f : any, ok);
            }
        }
        asm volatile("cp.async.commit_group;\n" ::: "memory");
    };
#pragma unroll
    for (int i = 0; i < RI; ++i)
#pragma unroll
        for (int j = 0; j < CJ; ++j) acc[i][j] = 0.0;
    // steps of 8 columns that this warp has work in (the same for its 32 lanes)
    const int left = nc - (c0 & ~7);
    const int jn = (r0 & ~3) < nr && left > 0 ? (left + 7) / 8 : 0;
    __syncthreads();  // the stage is free
#pragma unroll
    for (int c = 0; c < DT_BUFS - 1; ++c) copy(c);
    for (int c = 0; c < nk; ++c) {
        asm volatile("cp.async.wait_group %0;\n" ::"n"(DT_BUFS - 2) : "memory");
        __syncthreads();  // chunk c has landed, and chunk c - 1 is no longer read
        const double *As = stage + (c % DT_BUFS) * kChunk + r0;
        const double *Bs = stage + (c % DT_BUFS) * kChunk + kK * kPA + c0;
        if (!kNarrow) {
            if (jn > 0) add_chunk<kOp, CJ>(acc, As, Bs);
        } else if (jn > 6) {
            add_chunk<kOp, 8>(acc, As, Bs);
        } else if (jn > 4) {
            add_chunk<kOp, 6>(acc, As, Bs);
        } else if (jn > 2) {
            add_chunk<kOp, 4>(acc, As, Bs);
        } else if (jn > 0) {
            add_chunk<kOp, 2>(acc, As, Bs);
        }
        copy(c + DT_BUFS - 1);
    }
}

}  // namespace dist
}  // namespace fmlb
