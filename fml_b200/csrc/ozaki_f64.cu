// FP64 trailing update C -= P P^T of the Cholesky factorisation on the int8
// tensor cores: the Ozaki splitting scheme (K. Ozaki, T. Ogita, S. Oishi,
// S. M. Rump, "Error-free transformations of matrix multiplication by using
// fast routines of matrix multiplication and its applications", Numer.
// Algorithms 59, 2012; int8 form: H. Ootomo, K. Ozaki, R. Yokota, "DGEMM on
// integer matrix multiplication unit", IJHPCA 2024), written for tcgen05.
//
// Splitting. Each row r of P (k columns) gets the exponent e_r with
// max_c |P[r, c]| < 2^e_r, so x = P[r, c] 2^-(e_r + 1) lies in (-1/2, 1/2),
// and s base-256 digits by repeated flooring, all exact in FP64:
//     d_1 = floor(256 x) in [-128, 127];  u_t = floor(256 rem_{t-1}) in [0, 255]
// (a remainder 1 - |tiny| that rounds to 1.0 after a leading -1 is carried
// back into the digit, so every remainder stays in [0, 1))
// stored as signed bytes with a zero point: v_t = u_t - 128 in [-128, 127], so
//     x = xt + c + rho,   xt = d_1 / 256 + sum_{t>1} v_t 256^-t,
//     c = 128 sum_{t=2..s} 256^-t,   0 <= rho < 256^-s.
// With c' = c + 256^-s / 2 the error x - (xt + c') is zero-mean, and so are
// the dropped digit products below (v_t is centred), which keeps the errors
// of the k-term sums from adding up coherently. Then, summing over k,
//     x_r . x_c ~ xt_r . xt_c + c' (S_r + S_c) + k c'^2,   S_r = sum_k xt_r,k,
// and the product of two rows keeps the digit pairs (t, u) with t + u <= s + 1,
// grouped by diagonal q = t + u - 1:
//     xt_r . xt_c ~ 256^-(s + 1) sum_{q=1..s} D_q 256^(s - q),
//     D_q = sum_{t + u = q + 1} dig_t[r, :] . dig_u[c, :]       (exact in int32)
// s (s + 1) / 2 signed int8 products in all, every D_q accumulated exactly in
// its own TMEM accumulator and combined once, in FP64, by the epilogue
// (Horner in 256), which adds the zero-point terms and scales by
// 2^(e_r + e_c + 2). |dig| <= 128 bounds |D_q| by (q + 1) 2^14 k < 2^31 for
// k <= 8192. Six planes carry the accuracy of seven truncated 7-bit ones
// (21 products instead of 28); the error of one entry stays below
// k (s + 3) 2^(e_r + e_c + 2 - 8 s).
//
// Kernel (one CTA per SM at a time, four tiles per CTA, 384 threads), output
// tile 128 x 128, diagonals in passes of at most four (512 TMEM columns):
//   warp 0       TMA producer: per stage of 64 k values, the pass's digit planes
//                of the 128 A rows and 128 B rows (one 3-D box each, 64-byte
//                swizzle) into a ring as deep as shared memory allows (2 stages
//                at s = 6; 64-byte box rows move 1.6 times what 32-byte ones do);
//   warp 1       allocates the 512 TMEM columns and issues tcgen05.mma kind::i8
//                (M 128, N 128, K 32), the stage's MMAs fully unrolled;
//   warps 4..11  epilogue (registers moved there from the first warpgroup).
// C goes through registers and a small stage per warp: a whole tile of it in
// shared memory left room for 32-byte k steps only.
// m = 16384, k = 1024, s = 6: 3.13 ms = 88 FP64-equivalent TFLOP/s (4.71 ms before
// the wider stages, the unrolled issue and the separate drain). Shared memory is
// what bounds it now: the MMAs read 8 KB per 64 cycles of work, and their operands'
// copies and the epilogue pass through it as well.
// Every mbarrier wait is bounded; a wait that runs out stores FMLB_ETIMEDOUT
// in *info, and every kernel that reads info returns at once.
#include <math.h>
#include <stdint.h>

#include <algorithm>
#include <cstring>

#include "common.cuh"
#include "ozaki.cuh"
#include "tc_common.cuh"

namespace fmlb {
namespace {

constexpr int OZ_BM = 128, OZ_BN = 128;
// Diagonals (int32 accumulators of 128 columns) per pass: what the 512 TMEM columns hold.
constexpr int OZ_PASS_Q = 4;
constexpr int OZ_MAX_PASSES = (8 + OZ_PASS_Q - 1) / OZ_PASS_Q;
constexpr int OZ_KB = 64;          // int8 k values (bytes) per stage: two MMA K steps
constexpr int OZ_MMA_K = 32;       // k values of one MMA
constexpr int OZ_MAX_STAGES = 8;  // the ring depth is set per launch from shared memory
constexpr int OZ_THREADS = 384;    // 3 warpgroups: producer and MMA issuer, two of epilogue
// Registers a thread. The block starts with 168 each (65536 / 384, as the
// compiler grants them); the first warpgroup gives back what the epilogue takes,
// which keeps 64 drained columns in registers. The host checks the start, and runs
// the form that moves none where the compiler granted another number.
constexpr int OZ_REGS = 168, OZ_REGS_LOAD = 40, OZ_REGS_EPI = 232;
static_assert(OZ_REGS_LOAD + 2 * OZ_REGS_EPI <= 3 * OZ_REGS, "the registers of the block");
constexpr int OZ_EPI_WARPS = 8;
constexpr int OZ_TMEM_COLS = 512;
constexpr int OZ_A_PLANE = OZ_BM * OZ_KB;   // 8192 bytes per A digit plane per stage
constexpr int OZ_B_PLANE = OZ_BN * OZ_KB;   // 8192
constexpr int OZ_CHUNK = 8;        // columns of C that pass through shared memory at a time
// doubles of an epilogue warp: a 32 x 8 chunk of the update, the data of its 64
// columns and 32 rows
constexpr int OZ_WARP_STAGE = 32 * OZ_CHUNK + 2 * 64 + 2 * 32;
constexpr int OZ_CSTAGE_BYTES = OZ_EPI_WARPS * OZ_WARP_STAGE * (int)sizeof(double);  // 28 KB
constexpr int OZ_ALIGN = 1024;
constexpr int OZ_NONFINITE = 0x7fffffff;    // exponent marking a row with Inf / NaN

constexpr long long kOzDefaultBudget = 4000000000LL;  // clock cycles (~2 s)
constexpr int OZ_SMEM_LIMIT = 232448 - 64;  // opt-in shared memory per CTA, less static
constexpr int OZ_BAR_BYTES = (2 * OZ_MAX_STAGES + 3) * 8 + 8;

struct OzParams {
    int m;             // rows (= columns) of C
    int p_row0;        // slice row of C's row 0 (and column 0)
    int nkb;           // stages of OZ_KB k values
    int strip_cols;    // > 0: only the first strip_cols columns
    int strip_tiles;   // column tiles per row block in strip mode
    long long ntiles;
    long long ldc;
    double zp_c;       // c' (zero point of the digit planes)
    double zp_kc2;     // kp c'^2
    int skip_loads;    // test hook: the producer issues no copies
    int stages;        // depth of the operand ring
};

// Tensor maps of the digit planes, one per pass (boxes of that pass's planes).
struct OzMaps {
    CUtensorMap m[OZ_MAX_PASSES];
};

// Instruction descriptor, kind::i8: signed A and B, int32 accumulator, both
// K-major, M = 128, N = 128.
constexpr uint32_t kIdescI8 = (2u << 4) | (1u << 7) | (1u << 10) |
                              ((uint32_t)(OZ_BN >> 3) << 17) | ((uint32_t)(OZ_BM >> 4) << 24);

__device__ __forceinline__ void mma_i8(uint32_t tmem_d, uint64_t adesc, uint64_t bdesc,
                                       uint32_t accumulate) {
    asm volatile(
        "{\n .reg .pred p;\n setp.ne.b32 p, %4, 0;\n"
        " tcgen05.mma.cta_group::1.kind::i8 [%0], %1, %2, %3, p;\n}\n" ::"r"(tmem_d),
        "l"(adesc), "l"(bdesc), "r"(kIdescI8), "r"(accumulate));
}

// Tile t -> (row0, col0) of the lower triangle of 128 x 128 tiles (row block
// `by` holds column tiles 0 .. by), or of the first strip_tiles column tiles
// of every row block. Tiles run in bands of OZ_BAND row blocks and, inside a
// band, in groups of OZ_BAND column tiles (a 1024 x 1024 block of C), so the
// ~148 tiles in flight at a time share their digit planes through L2. Band
// b holds b + 1 groups below and on the diagonal. The enumeration covers a
// superset of C; false for tiles outside C.
constexpr int OZ_BAND = 8;
constexpr int OZ_GROUP = OZ_BAND * OZ_BAND;  // tiles of a band x group block
__device__ __forceinline__ bool oz_tile(long long t, const OzParams &p, int &row0, int &col0) {
    int by, bx;
    if (p.strip_tiles > 0) {
        const int band = (int)(t / (OZ_BAND * p.strip_tiles));
        const int w = (int)(t % (OZ_BAND * p.strip_tiles));
        by = band * OZ_BAND + w / p.strip_tiles;
        bx = w % p.strip_tiles;
    } else {
        // bands before band b: OZ_GROUP b (b + 1) / 2 tiles
        int b = (int)((sqrt(8.0 * (double)t / OZ_GROUP + 1.0) - 1.0) * 0.5);
        while ((long long)OZ_GROUP * b * (b + 1) / 2 > t) --b;
        while ((long long)OZ_GROUP * (b + 1) * (b + 2) / 2 <= t) ++b;
        const int u = (int)(t - (long long)OZ_GROUP * b * (b + 1) / 2);
        const int g = u / OZ_GROUP, w = u % OZ_GROUP;
        by = b * OZ_BAND + w / OZ_BAND;
        bx = g * OZ_BAND + w % OZ_BAND;
    }
    if (bx > by) return false;
    row0 = by * OZ_BM;
    col0 = bx * OZ_BN;
    return row0 < p.m && col0 < p.m;
}

__device__ __forceinline__ void oz_fail(int *info) { atomicCAS(info, 0, FMLB_ETIMEDOUT); }

// 2^(e + 1) for a row or column exponent in [-500, 500] (the scaled product
// core * 2^(e_r+1) * 2^(e_c+1) then equals ldexp(core, e_r + e_c + 2)), else 0.
__device__ __forceinline__ double oz_pow2_factor(int e) {
    return (e >= -500 && e <= 500) ? __longlong_as_double((long long)(e + 1 + 1023) << 52) : 0.0;
}

// The scaling for a non-finite row or column, or an exponent outside +-500.
__device__ __forceinline__ double oz_scale_far(double core, int er, int ec) {
    return (er == OZ_NONFINITE || ec == OZ_NONFINITE) ? __longlong_as_double(0x7ff8000000000000LL)
                                                      : ldexp(core, er + ec + 2);
}

// First tile t' >= t of this CTA's sequence (stride gridDim.x) inside C, or ntiles.
__device__ __forceinline__ long long oz_next_tile(long long t, const OzParams &p, int &row0,
                                                  int &col0) {
    for (; t < p.ntiles; t += gridDim.x)
        if (oz_tile(t, p, row0, col0)) return t;
    return p.ntiles;
}

// Exact int32 -> double: the value's bits beside the exponent of 2^52, then one
// addition (the conversion instruction runs at a quarter of the FP64 rate).
__device__ __forceinline__ double oz_double(uint32_t v) {
    return __dadd_rn(__hiloint2double(0x43300000, (int)(v ^ 0x80000000u)),
                     -4503601774854144.0);  // -(2^52 + 2^31)
}

// Double (row, c) of an epilogue warp's 32 x 8 stage: pairs of columns are
// permuted by the row, so that rows written by one lane each (16 bytes at a
// time) and rows read by 8 lanes each both spread over the banks.
__device__ __forceinline__ int oz_stage_at(int row, int c) {
    return row * OZ_CHUNK + (((c >> 1) ^ ((row >> 1) & 3)) << 1) + (c & 1);
}

// Passes over the diagonals: [0, Q), [Q, 2Q), .. [.., NS). A pass that ends
// before diagonal q1 reads the digit planes 0 .. q1-1.
constexpr int oz_passes(int ns) { return (ns + OZ_PASS_Q - 1) / OZ_PASS_Q; }
__host__ __device__ constexpr int oz_pass_end(int ns, int ps) {
    return (ps + 1) * OZ_PASS_Q < ns ? (ps + 1) * OZ_PASS_Q : ns;
}

// The MMAs of one stage of pass PS, all of them unrolled: one thread issues
// them, and with the loops and their index arithmetic an MMA took 148 cycles,
// 84 unrolled.
template <int NS, int PS>
__device__ __forceinline__ void oz_issue(uint32_t tmem, uint64_t da, uint64_t db, uint32_t first) {
    constexpr int q0 = PS * OZ_PASS_Q, q1 = oz_pass_end(NS, PS);
#pragma unroll
    for (int h = 0; h < OZ_KB / OZ_MMA_K; ++h) {
#pragma unroll
        for (int q = q0; q < q1; ++q) {
#pragma unroll
            for (int a = 0; a <= q; ++a)  // offsets in 16-byte units of the descriptor address
                mma_i8(tmem + (uint32_t)((q - q0) * OZ_BN),
                       da + (uint64_t)((a * OZ_A_PLANE + h * OZ_MMA_K) >> 4),
                       db + (uint64_t)(((q - a) * OZ_B_PLANE + h * OZ_MMA_K) >> 4),
                       h == 0 && a == 0 ? first : 1u);
        }
    }
}

template <int NS, bool kMoveRegs>
__global__ void __launch_bounds__(OZ_THREADS, 1)
ozaki_syrk_kernel(const __grid_constant__ OzMaps maps,
                  const int *__restrict__ exps, const double *__restrict__ rsum, OzParams p,
                  double *__restrict__ C, int *__restrict__ info, long long budget) {
    extern __shared__ uint8_t oz_smem_raw[];
    uint8_t *smem = reinterpret_cast<uint8_t *>(
        (reinterpret_cast<uintptr_t>(oz_smem_raw) + OZ_ALIGN - 1) & ~(uintptr_t)(OZ_ALIGN - 1));
    constexpr int stage_bytes = NS * (OZ_A_PLANE + OZ_B_PLANE);  // B planes after NS A planes
    constexpr int npass = oz_passes(NS);
    const int nst = p.stages;
    double *cstage = reinterpret_cast<double *>(smem + nst * stage_bytes);
    uint64_t *bars = reinterpret_cast<uint64_t *>(smem + nst * stage_bytes + OZ_CSTAGE_BYTES);
    uint64_t *full = bars, *empty = bars + OZ_MAX_STAGES;
    uint64_t *tmem_full = bars + 2 * OZ_MAX_STAGES, *tmem_empty = tmem_full + 1,
             *mma_done = tmem_empty + 1;
    uint32_t *tmem_slot = reinterpret_cast<uint32_t *>(mma_done + 1);
    __shared__ int abort_cta;

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    if (threadIdx.x == 0) {
        abort_cta = *(volatile const int *)info != 0;
        for (int s = 0; s < nst; ++s) {
            tc::mbar_init(&full[s], 1);
            tc::mbar_init(&empty[s], 1);
        }
        tc::mbar_init(tmem_full, 1);
        tc::mbar_init(tmem_empty, OZ_EPI_WARPS);
        tc::mbar_init(mma_done, 1);
        tc::mbar_fence_init();
    }
    __syncthreads();
    if (abort_cta) return;  // a failed factorisation: the whole CTA leaves together
    if (warp == 1) tc::tmem_alloc(tmem_slot, OZ_TMEM_COLS);
    tc::fence_before_sync();
    __syncthreads();
    tc::fence_after_sync();
    const uint32_t tmem_base = *tmem_slot;

    // each warpgroup sets its registers inside its own branch: where the two meet
    // the compiler can count on the smaller number only
    if (kMoveRegs && warp < 4)
        asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;\n" ::"n"(OZ_REGS_LOAD));
    if (warp == 0) {
        // ------------------------------------------------------------ producer
        if (lane == 0) {
            long long issued = 0;
            bool ok = true;
            for (long long t = blockIdx.x; t < p.ntiles && ok; t += gridDim.x) {
                int row0, col0;
                if (!oz_tile(t, p, row0, col0)) continue;
                for (int ps = 0; ps < npass && ok; ++ps) {
                    const int q1 = oz_pass_end(NS, ps);
                    const CUtensorMap *map = &maps.m[ps];  // boxes of q1 planes
                    for (int kb = 0; kb < p.nkb && !p.skip_loads; ++kb, ++issued) {
                        const int st = (int)(issued % nst);
                        const uint32_t ph = (uint32_t)((issued / nst) & 1);
                        if (!tc::mbar_wait(&empty[st], ph ^ 1, budget)) {
                            oz_fail(info);
                            ok = false;
                            break;
                        }
                        uint8_t *sa = smem + st * stage_bytes;
                        uint8_t *sb = sa + NS * OZ_A_PLANE;
                        tc::mbar_arrive_expect_tx(&full[st], (uint32_t)(q1 * (OZ_A_PLANE + OZ_B_PLANE)));
                        tc::tma_load_3d(sa, map, &full[st], kb * OZ_KB, p.p_row0 + row0, 0);
                        tc::tma_load_3d(sb, map, &full[st], kb * OZ_KB, p.p_row0 + col0, 0);
                    }
                }
            }
            // every copy this thread issued has landed before the CTA winds down
            for (long long l = std::max(0LL, issued - (long long)nst); l < issued; ++l)
                if (!tc::mbar_wait(&full[l % nst], (uint32_t)((l / nst) & 1), budget))
                    oz_fail(info);
        }
    } else if (warp == 1) {
        // ------------------------------------------------------------- MMA issuer
        if (lane == 0) {
            long long consumed = 0;
            int lp = 0;  // passes issued
            bool ok = true;
            for (long long t = blockIdx.x; t < p.ntiles && ok; t += gridDim.x) {
                int row0, col0;
                if (!oz_tile(t, p, row0, col0)) continue;
                for (int ps = 0; ps < npass; ++ps, ++lp) {
                    if (!tc::mbar_wait(tmem_empty, (uint32_t)((lp & 1) ^ 1), budget)) {
                        oz_fail(info);
                        ok = false;
                        break;
                    }
                    tc::fence_after_sync();
                    for (int kb = 0; kb < p.nkb; ++kb, ++consumed) {
                        const int st = (int)(consumed % nst);
                        const uint32_t ph = (uint32_t)((consumed / nst) & 1);
                        if (!tc::mbar_wait(&full[st], ph, budget)) {
                            oz_fail(info);
                            ok = false;
                            break;
                        }
                        tc::fence_after_sync();
                        const uint8_t *sa = smem + st * stage_bytes;
                        const uint8_t *sb = sa + NS * OZ_A_PLANE;
                        const uint64_t da = tc::smem_desc_kmajor(sa, OZ_KB);
                        const uint64_t db = tc::smem_desc_kmajor(sb, OZ_KB);
                        if (ps == 0) oz_issue<NS, 0>(tmem_base, da, db, kb > 0);
                        else oz_issue<NS, npass - 1>(tmem_base, da, db, kb > 0);
                        tc::mma_commit(&empty[st]);  // frees the stage once these MMAs finish
                    }
                    if (!ok) break;
                    tc::mma_commit(tmem_full);
                }
            }
            // every MMA issued has finished before TMEM is released
            tc::mma_commit(mma_done);
            if (!tc::mbar_wait(mma_done, 0, budget)) oz_fail(info);
        }
    } else if (warp >= 4) {
        if (kMoveRegs) asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;\n" ::"n"(OZ_REGS_EPI));
        // --------------------------------------------------------------- epilogue
        // Two warps per TMEM lane quarter, 64 columns each. The tensor cores wait
        // from a pass's last MMA until its accumulators are drained, so that comes
        // first and alone: into FP64 (Horner in 256), a row and 64 columns per
        // lane in registers, the next 8 columns' loads in flight while 8 are
        // converted. The rest runs beside the next pass's MMAs: 8 columns at a
        // time go through the warp's stage to the lanes that hold those entries of
        // C in 64-byte row segments, which scale, subtract and store them. An entry
        // of C belongs to the same lane in every pass; C's lines are brought into
        // L2 while the tile's first pass runs.
        // Cycles of a tile (6 planes, k = 1024): 96k, of which the MMAs wait 8k for
        // the drain and 9k for operands; 136k with the drain, the scaling and C's
        // update in one loop, 33k of them waiting for it.
        const int qw = warp & 3;
        const int half = (warp - 4) >> 2;
        double *stage = cstage + (warp - 4) * OZ_WARP_STAGE;
        double *colf = stage + 32 * OZ_CHUNK, *colsum = colf + 64;
        double *rowf = colsum + 64, *rowsum = rowf + 32;
        const int sr0 = lane >> 3, sc0 = lane & 7;
        int lp = 0;
        bool ok = true;
        int row0 = 0, col0 = 0;
        for (long long t = oz_next_tile(blockIdx.x, p, row0, col0); t < p.ntiles && ok;
             t = oz_next_tile(t + gridDim.x, p, row0, col0)) {
            const int wrow = row0 + qw * 32, wcol = col0 + half * 64;  // the warp's part of C
            double *cbase = C + (size_t)(wrow + sr0) * p.ldc + wcol + sc0;
            // entry i of chunk ch: row 4 i + sr0, column 8 ch + sc0
            auto inside = [&](int i, int ch) {
                const int gr = wrow + 4 * i + sr0, gc = wcol + OZ_CHUNK * ch + sc0;
                return gr < p.m && gc <= gr && (p.strip_cols == 0 || gc < p.strip_cols);
            };
            {   // the 512-byte row segment of each lane's row
                const int gr = wrow + lane;
                if (gr < p.m && wcol <= gr)
                    for (int c = 0; c < 64; c += 16)
                        asm volatile("prefetch.global.L2 [%0];" ::"l"(
                            C + (size_t)gr * p.ldc + min(wcol + c, p.m - 1)));
            }
            // data of the warp's 64 columns and 32 rows: 2^(e + 1) (0 where the
            // exact scaling needs ldexp) and the digit sums S
            bool plain = true;
            for (int c = lane; c < 96; c += 32) {
                const int g = c < 64 ? wcol + c : wrow + c - 64;
                const double f = oz_pow2_factor(g < p.m ? exps[p.p_row0 + g] : 0);
                plain = plain && f != 0.0;
                (c < 64 ? colf + c : rowf + c - 64)[0] = f;
                (c < 64 ? colsum + c : rowsum + c - 64)[0] = g < p.m ? rsum[p.p_row0 + g] : 0.0;
            }
            plain = __all_sync(0xffffffffu, plain);
            for (int ps = 0; ps < npass; ++ps, ++lp) {
                const int q1 = oz_pass_end(NS, ps), nq = q1 - ps * OZ_PASS_Q;
                const bool last = ps == npass - 1;
                // Horner over diagonals q0 .. q1-1 carries 256^(q1-1-q): scale by 256^-(q1+1)
                const double pbias = __longlong_as_double((long long)(1023 - 8 * (q1 + 1)) << 52);
                if (!tc::mbar_wait(tmem_full, (uint32_t)(lp & 1), budget)) {
                    oz_fail(info);
                    ok = false;
                    break;
                }
                tc::fence_after_sync();
                const uint32_t tbase = tmem_base + ((uint32_t)(qw * 32) << 16) +
                                       (uint32_t)(half * 64);
                double acc[64];
                {
                    uint32_t v[OZ_PASS_Q][OZ_CHUNK];
                    auto load = [&](int cb) {
#pragma unroll
                        for (int q = 0; q < OZ_PASS_Q; ++q)
                            if (q < nq) tc::tmem_ld8_async(tbase + (uint32_t)(q * OZ_BN + cb), v[q]);
                    };
                    load(0);
#pragma unroll
                    for (int cb = 0; cb < 64; cb += OZ_CHUNK) {
                        tc::tmem_ld_wait();
#pragma unroll
                        for (int q = 0; q < OZ_PASS_Q; ++q) {
                            if (q < nq) {
#pragma unroll
                                for (int j = 0; j < OZ_CHUNK; ++j) {
                                    const double x = oz_double(tc::after_ld_wait(v[q][j]));
                                    acc[cb + j] = q ? fma(acc[cb + j], 256.0, x) : x;
                                }
                            }
                        }
                        if (cb + OZ_CHUNK < 64) load(cb + OZ_CHUNK);
                    }
                }
                tc::fence_before_sync();
                __syncwarp();
                if (lane == 0) tc::mbar_arrive(tmem_empty);  // the accumulators are free
#pragma unroll
                for (int ch = 0; ch < 64 / OZ_CHUNK; ++ch) {
                    const int cb = ch * OZ_CHUNK;
#pragma unroll
                    for (int c = 0; c < OZ_CHUNK; c += 2)
                        *reinterpret_cast<double2 *>(&stage[oz_stage_at(lane, c)]) =
                            make_double2(acc[cb + c], acc[cb + c + 1]);
                    __syncwarp();
                    // last pass: (acc 256^-(s+1) + c' (S_r + S_c) + k c'^2) 2^(e_r + e_c + 2),
                    // earlier passes: acc 256^-(q1+1) 2^(e_r + e_c + 2); fixed order, no
                    // contraction. Both power-of-two scalings are exact multiplications
                    // (core * 2^(e_r+1) is normal), so the result is ldexp's, rounded once.
                    auto core_of = [&](int r) {
                        const double core = __dmul_rn(stage[oz_stage_at(r, sc0)], pbias);
                        return last ? __dadd_rn(__dadd_rn(core, __dmul_rn(p.zp_c,
                                                                          __dadd_rn(rowsum[r],
                                                                                    colsum[cb + sc0]))),
                                                p.zp_kc2)
                                    : core;
                    };
                    double *cc = cbase + cb;
                    if (plain) {
                        const double f = colf[cb + sc0];
                        double cv[8];
#pragma unroll
                        for (int i = 0; i < 8; ++i)
                            cv[i] = inside(i, ch) ? cc[(size_t)(4 * i) * p.ldc] : 0.0;
#pragma unroll
                        for (int i = 0; i < 8; ++i) {
                            const int r = 4 * i + sr0;
                            const double v = __dmul_rn(__dmul_rn(core_of(r), rowf[r]), f);
                            if (inside(i, ch)) cc[(size_t)(4 * i) * p.ldc] = __dsub_rn(cv[i], v);
                        }
                    } else {  // a non-finite row or column, or an exponent outside +-500
#pragma unroll 1
                        for (int i = 0; i < 8; ++i) {
                            if (!inside(i, ch)) continue;
                            const int r = 4 * i + sr0;
                            double *e = cc + (size_t)(4 * i) * p.ldc;
                            *e = __dsub_rn(*e, oz_scale_far(core_of(r), exps[p.p_row0 + wrow + r],
                                                            exps[p.p_row0 + wcol + cb + sc0]));
                        }
                    }
                    __syncwarp();
                }
            }
        }
    }
    tc::fence_before_sync();
    __syncthreads();
    tc::fence_after_sync();
    if (warp == 1) tc::tmem_dealloc(tmem_base, OZ_TMEM_COLS);
}

// ---- splitting --------------------------------------------------------------
// One CTA (128 threads) per row of P (rows [0, m), k columns, stride ldp):
// exps[r], ns digit planes (row-major, kp >= k columns zero-padded, plane
// stride pstride bytes) and the row sum rsum[r] = S_r of the zero-point
// digits (per-plane integer sums, combined in FP64 in plane order). Each
// thread owns 8 consecutive columns per sweep.
constexpr int SL_TPB = 128;

__global__ void __launch_bounds__(SL_TPB)
ozaki_slice_kernel(const double *__restrict__ P, long long ldp, int m, int k, int kp, int ns,
                   int8_t *__restrict__ planes, long long pstride, long long ldpl,
                   int *__restrict__ exps, double *__restrict__ rsum,
                   const int *__restrict__ info) {
    __shared__ double red[SL_TPB / 32];
    __shared__ int tsum[OZAKI_MAX_SLICES][SL_TPB / 32];
    __shared__ int bad_row, abort_cta;
    const int r = blockIdx.x, tid = threadIdx.x;
    if (tid == 0) {
        abort_cta = info && *(volatile const int *)info != 0;
        bad_row = 0;
    }
    __syncthreads();
    if (abort_cta || r >= m) return;
    const double *row = P + (size_t)r * ldp;
    double mx = 0.0;
    for (int c = tid; c < k; c += SL_TPB) {
        const double v = row[c];
        if (!isfinite(v)) bad_row = 1;
        mx = fmax(mx, fabs(v));
    }
#pragma unroll
    for (int o = 16; o; o >>= 1) mx = fmax(mx, __shfl_xor_sync(0xffffffffu, mx, o));
    if ((tid & 31) == 0) red[tid >> 5] = mx;
    __syncthreads();
    mx = fmax(fmax(red[0], red[1]), fmax(red[2], red[3]));
    int e = 0;
    if (mx > 0.0) frexp(mx, &e);  // mx = f 2^e, f in [0.5, 1): |P[r, :]| < 2^e
    if (tid == 0) exps[r] = bad_row ? OZ_NONFINITE : e;
    int psum[OZAKI_MAX_SLICES];
#pragma unroll
    for (int t = 0; t < OZAKI_MAX_SLICES; ++t) psum[t] = 0;
    for (int c0 = tid * 8; c0 < kp; c0 += SL_TPB * 8) {
        double x[8];
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            const int c = c0 + i;
            const double v = c < k ? row[c] : 0.0;
            x[i] = (bad_row || !isfinite(v)) ? 0.0 : ldexp(v, -(e + 1));  // in (-1/2, 1/2)
        }
#pragma unroll
        for (int t = 0; t < OZAKI_MAX_SLICES; ++t) {
            if (t >= ns) break;
            uint64_t word = 0;
#pragma unroll
            for (int i = 0; i < 8; ++i) {
                x[i] *= 256.0;
                double d = floor(x[i]);             // [-128, 127] first, then [0, 255]
                x[i] -= d;
                // a tiny negative leading value gives d = -1 and a remainder
                // 1 - |x| that rounds to 1.0: carry it back into the digit
                if (x[i] >= 1.0) {
                    x[i] -= 1.0;
                    d += 1.0;
                }
                const int v = (int)d - (t ? 128 : 0);  // zero point of the lower planes
                psum[t] += v;
                word |= (uint64_t)((uint32_t)v & 0xffu) << (8 * i);
            }
            *reinterpret_cast<uint64_t *>(planes + t * pstride + (size_t)r * ldpl + c0) = word;
        }
    }
#pragma unroll
    for (int t = 0; t < OZAKI_MAX_SLICES; ++t) {
        int v = psum[t];
#pragma unroll
        for (int o = 16; o; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
        if ((tid & 31) == 0) tsum[t][tid >> 5] = v;
    }
    __syncthreads();
    if (tid == 0) {
        double sr = 0.0;
        for (int t = 0; t < ns; ++t) {
            const int tt = tsum[t][0] + tsum[t][1] + tsum[t][2] + tsum[t][3];
            sr = __dadd_rn(sr, ldexp((double)tt, -8 * (t + 1)));
        }
        rsum[r] = sr;
    }
}

int make_plane_map(CUtensorMap *map, const int8_t *base, int rows, long long ldpl, int kp,
                   long long pstride, int ns, int box_rows) {
    tc::EncodeTiledFn fn = tc::encode_tiled_fn();
    if (!fn) {
        set_error("cuTensorMapEncodeTiled is unavailable");
        return FMLB_ECUDA;
    }
    FMLB_REQUIRE(((uintptr_t)base % 16) == 0 && ldpl % 16 == 0 && pstride % 16 == 0,
                 "ozaki: digit planes not 16-byte aligned");
    const cuuint64_t gdim[3] = {(cuuint64_t)kp, (cuuint64_t)rows, (cuuint64_t)ns};
    const cuuint64_t gstride[2] = {(cuuint64_t)ldpl, (cuuint64_t)pstride};
    const cuuint32_t box[3] = {(cuuint32_t)OZ_KB, (cuuint32_t)box_rows, (cuuint32_t)ns};
    const cuuint32_t estride[3] = {1, 1, 1};
    CUresult res = fn(map, CU_TENSOR_MAP_DATA_TYPE_UINT8, 3, const_cast<int8_t *>(base), gdim,
                      gstride, box, estride, CU_TENSOR_MAP_INTERLEAVE_NONE,
                      CU_TENSOR_MAP_SWIZZLE_64B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                      CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (res != CUDA_SUCCESS) {
        set_error("ozaki: cuTensorMapEncodeTiled failed (%d)", (int)res);
        return FMLB_ECUDA;
    }
    return FMLB_OK;
}

// Deepest operand ring (<= OZ_MAX_STAGES) whose shared memory fits a CTA
// (three stages up to 4 planes, two at 5 or 6, one at 7 or 8).
int oz_stages(int ns) {
    const int sb = ns * (OZ_A_PLANE + OZ_B_PLANE);
    const int room = OZ_SMEM_LIMIT - OZ_CSTAGE_BYTES - OZ_BAR_BYTES - OZ_ALIGN;
    return std::max(1, std::min(OZ_MAX_STAGES, room / sb));
}

size_t oz_smem_bytes(int ns) {
    return (size_t)oz_stages(ns) * ns * (OZ_A_PLANE + OZ_B_PLANE) + OZ_CSTAGE_BYTES +
           OZ_BAR_BYTES + OZ_ALIGN;
}

thread_local tc::TestHooks t_hooks = {0, 0, 0, 0, 0};

// `move`: as built, the kernel can move registers between its warpgroups. That takes
// a start with OZ_REGS each (setmaxnreg.inc would wait for registers it cannot get), which
// depends on the compiler; otherwise the form without it runs (m = 16384, k = 1024, s = 6,
// with the split: 3.17 ms and 3.94).
template <int NS>
int launch_oz(const OzMaps &maps, const OzakiSlices &s, const OzParams &p, double *C, int *info,
              int grid, size_t smem, const tc::TestHooks &hooks, cudaStream_t st) {
    static_assert(NS <= OZAKI_MAX_SLICES, "digit planes");
    static int attr_dev = -1;
    static bool move = false;
    int dev = 0;
    FMLB_TRY(cuda_status(cudaGetDevice(&dev), "ozaki: cudaGetDevice"));
    if (attr_dev != dev) {
        FMLB_TRY(cuda_status(cudaFuncSetAttribute(ozaki_syrk_kernel<NS, true>,
                                                  cudaFuncAttributeMaxDynamicSharedMemorySize,
                                                  OZ_SMEM_LIMIT),
                             "ozaki: smem attribute"));
        FMLB_TRY(cuda_status(cudaFuncSetAttribute(ozaki_syrk_kernel<NS, false>,
                                                  cudaFuncAttributeMaxDynamicSharedMemorySize,
                                                  OZ_SMEM_LIMIT),
                             "ozaki: smem attribute"));
        cudaFuncAttributes fa;
        FMLB_TRY(cuda_status(cudaFuncGetAttributes(&fa, ozaki_syrk_kernel<NS, true>),
                             "ozaki: kernel attributes"));
        move = fa.numRegs == OZ_REGS;
        attr_dev = dev;
    }
    if (move && !hooks.fixed_regs)
        ozaki_syrk_kernel<NS, true><<<grid, OZ_THREADS, smem, st>>>(maps, s.exps, s.rsum, p, C, info,
                                                                    hooks.wait_budget);
    else
        ozaki_syrk_kernel<NS, false><<<grid, OZ_THREADS, smem, st>>>(maps, s.exps, s.rsum, p, C,
                                                                     info, hooks.wait_budget);
    return launch_status("ozaki_syrk_kernel");
}

}  // namespace

tc::TestHooks tc::test_hooks() {
    tc::TestHooks h = t_hooks;
    if (h.wait_budget <= 0) h.wait_budget = kOzDefaultBudget;
    return h;
}

int ozaki_split(const double *P, long long ldp, int m, int k, const OzakiSlices &s, const int *info,
                cudaStream_t st) {
    if (m <= 0) return FMLB_OK;
    FMLB_REQUIRE(m <= s.rows && k <= s.kp, "ozaki: panel %d x %d exceeds the slice buffer %d x %d",
                 m, k, s.rows, s.kp);
    ozaki_slice_kernel<<<m, SL_TPB, 0, st>>>(P, ldp, m, k, s.kp, s.ns, s.planes, s.pstride,
                                             s.ldpl, s.exps, s.rsum, info);
    return launch_status("ozaki_slice_kernel");
}

int ozaki_syrk(double *C, long long ldc, int m, const OzakiSlices &s, int p_row0, int strip_cols,
               int *info, cudaStream_t st) {
    if (m <= 0) return FMLB_OK;
    FMLB_REQUIRE(s.ns >= 1 && s.ns <= OZAKI_MAX_SLICES, "ozaki: 1..%d slices", OZAKI_MAX_SLICES);
    FMLB_REQUIRE(s.kp % OZ_MMA_K == 0 && s.kp <= 8192, "ozaki: k must be a multiple of 32, <= 8192");
    FMLB_REQUIRE(p_row0 >= 0 && p_row0 + m <= s.rows, "ozaki: rows outside the slice buffer");
    // boxes of 128 rows and the planes each pass reads (planes 0 .. q1-1 for
    // its last diagonal q1-1)
    OzMaps maps;
    memset(&maps, 0, sizeof maps);
    for (int ps = 0; ps < oz_passes(s.ns); ++ps)
        FMLB_TRY(make_plane_map(&maps.m[ps], s.planes, s.rows, s.ldpl, s.kp, s.pstride,
                                oz_pass_end(s.ns, ps), OZ_BM));
    OzParams p;
    p.m = m;
    p.p_row0 = p_row0;
    p.nkb = ceil_div(s.kp, OZ_KB);  // past kp the copies fill with zeros
    p.strip_cols = strip_cols > 0 ? std::min(strip_cols, m) : 0;
    const long long Tr = ceil_div(m, OZ_BM);
    p.strip_tiles = p.strip_cols > 0 ? ceil_div(p.strip_cols, OZ_BN) : 0;
    const long long nband = ceil_div(Tr, OZ_BAND);
    p.ntiles = p.strip_tiles ? nband * OZ_BAND * p.strip_tiles
                             : (long long)OZ_GROUP * nband * (nband + 1) / 2;
    p.ldc = ldc;
    double zc = ldexp(1.0, -8 * s.ns - 1);  // half an ulp of the last digit
    for (int t = 2; t <= s.ns; ++t) zc += ldexp(128.0, -8 * t);
    p.zp_c = zc;
    p.zp_kc2 = (double)s.kp * zc * zc;
    const tc::TestHooks hooks = tc::test_hooks();
    p.skip_loads = hooks.skip_loads;
    p.stages = oz_stages(s.ns);
    const size_t smem = oz_smem_bytes(s.ns);
    // four tiles per CTA: CTAs retire while the update runs, so the
    // factorisation's high-priority panel chain gets SMs (a persistent grid
    // held every SM until the update ended and serialised the lookahead)
    const int grid = (int)std::min<long long>(
        p.ntiles, std::max<long long>(sm_count(), (p.ntiles + 3) / 4));
    switch (s.ns) {
        case 1: return launch_oz<1>(maps, s, p, C, info, grid, smem, hooks, st);
        case 2: return launch_oz<2>(maps, s, p, C, info, grid, smem, hooks, st);
        case 3: return launch_oz<3>(maps, s, p, C, info, grid, smem, hooks, st);
        case 4: return launch_oz<4>(maps, s, p, C, info, grid, smem, hooks, st);
        case 5: return launch_oz<5>(maps, s, p, C, info, grid, smem, hooks, st);
        case 6: return launch_oz<6>(maps, s, p, C, info, grid, smem, hooks, st);
        case 7: return launch_oz<7>(maps, s, p, C, info, grid, smem, hooks, st);
        default: return launch_oz<8>(maps, s, p, C, info, grid, smem, hooks, st);
    }
}

size_t ozaki_slice_bytes(int rows, int kp, int ns) {
    return (size_t)ns * rows * kp + (size_t)rows * (sizeof(int) + sizeof(double)) + 512;
}

int ozaki_bind(void *ws, int rows, int kp, int ns, OzakiSlices &s) {
    FMLB_REQUIRE(kp % OZ_MMA_K == 0, "ozaki: padded k must be a multiple of 32");
    char *p = reinterpret_cast<char *>((reinterpret_cast<uintptr_t>(ws) + 255) & ~(uintptr_t)255);
    s.planes = reinterpret_cast<int8_t *>(p);
    s.rows = rows;
    s.kp = kp;
    s.ns = ns;
    s.ldpl = kp;
    s.pstride = (long long)rows * kp;
    s.rsum = reinterpret_cast<double *>(p + (size_t)ns * rows * kp);  // 8-byte aligned: kp % 32 == 0
    s.exps = reinterpret_cast<int *>(s.rsum + rows);
    return FMLB_OK;
}

}  // namespace fmlb

extern "C" size_t fmlb_syrk_ozaki_workspace_bytes(int m, int k, int nslices) {
    if (m <= 0 || k <= 0 || nslices <= 0) return 256;
    const int kp = (k + 31) / 32 * 32;
    return fmlb::ozaki_slice_bytes(m, kp, nslices);
}

extern "C" int fmlb_syrk_lower_ozaki(double *C, long long ldc, int m, const double *P,
                                     long long ldp, int k, int strip_cols, int nslices,
                                     void *work, size_t ws_bytes, int *info, void *stream) {
    using namespace fmlb;
    FMLB_REQUIRE(m >= 0 && k >= 0 && ldc >= m && ldp >= k && strip_cols >= 0,
                 "fmlb_syrk_lower_ozaki: bad sizes");
    FMLB_REQUIRE(nslices >= 1 && nslices <= OZAKI_MAX_SLICES,
                 "fmlb_syrk_lower_ozaki: nslices must be 1..%d", OZAKI_MAX_SLICES);
    FMLB_REQUIRE(k <= 8192, "fmlb_syrk_lower_ozaki: k=%d above 8192", k);
    if (m == 0 || k == 0) return FMLB_OK;
    FMLB_REQUIRE(C && P && info, "fmlb_syrk_lower_ozaki: null pointer");
    const size_t need = fmlb_syrk_ozaki_workspace_bytes(m, k, nslices);
    if (!work || ws_bytes < need) {
        set_error("fmlb_syrk_lower_ozaki: workspace %zu < %zu bytes", ws_bytes, need);
        return FMLB_ENOMEM;
    }
    OzakiSlices s;
    FMLB_TRY(ozaki_bind(work, m, (k + 31) / 32 * 32, nslices, s));
    cudaStream_t st = FMLB_STREAM(stream);
    FMLB_TRY(ozaki_split(P, ldp, m, k, s, info, st));
    return ozaki_syrk(C, ldc, m, s, 0, strip_cols, info, st);
}

extern "C" int fmlb_tc_test_hooks(long long wait_cycles, int skip_loads) {
    using namespace fmlb;
    FMLB_REQUIRE(wait_cycles >= 0, "fmlb_tc_test_hooks: negative wait budget");
    t_hooks.wait_budget = wait_cycles;
    t_hooks.skip_loads = skip_loads != 0 && skip_loads != 8;
    t_hooks.extra_block = (skip_loads & 2) != 0;
    t_hooks.withhold = (skip_loads & 4) != 0;
    t_hooks.fixed_regs = (skip_loads & 8) != 0;
    return FMLB_OK;
}
