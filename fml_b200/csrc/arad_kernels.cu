// ARAD molecular kernels: fget_kernels_arad / fget_symmetric_kernels_arad,
// fml/kernels/farad_kernels.f90:439-755, core atomic_distl2 :29-90.
//
//   K[s, I, J] = sum_{i1 < n_I, j1 < n_J} exp(-l2(i1, j1) / sigma_s^2)
//   l2 = self(I, i1) + self(J, j1) - 2 * S(i1, j1) * stoch(i1, j1), |l2| < eps -> 0
//   S  = sum over neighbour pairs (m1, m2) within the cut of
//        exp(-(r1 - r2)^2 / (4 w^2)) xi1 xi2 stoch(m1, m2) (1 + c1 c2 + s1 s2),
//        only where (r1 - r2)^2 < (8 w)^2.
//
// Stage 1 (arad_prep_kernel) turns each descriptor into its neighbour-list
// prefix length (the reference's early exit at r > cut), the sine factors xi
// and the self terms. Stage 2 evaluates molecule pairs.
//
// The FP64 path keeps the reference's operation order (explicit _rn
// intrinsics, no contracted FMA). The FP32 path is the fast path; its
// neighbour data is re-packed as float4 {r, xi, xi*c, xi*s} + float2 {row, col}.
#include <math.h>

#include <algorithm>

#include "common.cuh"

namespace fmlb {
namespace {

constexpr int MAXSIG = 16;

struct SigmaTable {
    double inv_sigma2[MAXSIG];  // -1 / sigma^2 (farad_kernels.f90:511)
};

struct AradParams {
    double width, cut, rw2, cw2, inv_width, maxg2, inv_cut;
    double eps;  // |l2| below eps counts as 0
};

// Per-set workspace views.
struct SetWs {
    int *nnb;             // (nm, amax)       neighbour prefix length
    double *xi;           // (nm, amax, amax) sine factors (FP64 path)
    double *self;         // (nm, amax)       self terms (FP64 path)
    float4 *pk;           // (nm, amax, amax) {r, xi, xi*c, xi*s} (FP32 paths)
    float2 *pz;           // (nm, amax, amax) {row, col}         (generic FP32 path)
    float *self32;        // (nm, amax)       self terms (generic FP32 path)
    signed char *asc;     // (nm, amax)       1: the neighbour list ascends in r (fast FP64 path)
    signed char *cls;     // (nm, amax, amax) element class of each neighbour (fast path)
    signed char *acls;    // (nm, amax)       element class of each atom (fast path)
    float *selff;         // (nm, amax)       self terms (fast path)
    float4 *spk;          // (nm, slots) records of each molecule by r, 64 to a group (paired path)
    unsigned short *smeta;  // (nm, slots)   atom | class << 8 | used << 15 of each
    float2 *band;         // (nm, slots / 64) lowest and highest r of each group
    int *nrec;            // (nm)             records per molecule
};

// Element classes (distinct periodic-table positions) of the fast paths: the
// stoichiometric factor between two classes comes from a small table.
constexpr int FC_MAXC = 16;
constexpr int FC_NPOS = 8 * 34;  // (row 0..7) * 34 + (col 0..33)
struct ClassInfo {
    int flag;                 // 0: fast path usable; otherwise why not
    int ncls;
    int present[FC_NPOS];
    signed char map[FC_NPOS]; // position -> class, -1 if absent
    float stoch[FC_MAXC * FC_MAXC];
    double stoch64[FC_MAXC * FC_MAXC];  // the factor as the pair loop forms it, in FP64
};

__host__ __device__ inline size_t align256(size_t x) { return (x + 255) & ~(size_t)255; }

// The FP32 pair kernel takes BD_REC records of molecule I at a time: the slots of
// nm molecules' records, each molecule's a multiple of that.
constexpr int BD_REC = 64;
__host__ __device__ inline int band_stride(int amax) {
    return (amax * amax + BD_REC - 1) / BD_REC * BD_REC;
}
inline size_t band_slots(int nm, int amax) { return (size_t)nm * band_stride(amax); }

size_t set_ws_bytes(int nm, int amax) {
    const size_t a2 = (size_t)nm * amax * amax, a1 = (size_t)nm * amax;
    return align256(a1 * sizeof(int)) + align256(a2 * sizeof(double)) +
           align256(a1 * sizeof(double)) + align256(a2 * sizeof(float4)) +
           align256(a2 * sizeof(float2)) + align256(a1 * sizeof(float)) + align256(a2) +
           align256(a1) + align256(a1 * sizeof(float)) +
           align256(band_slots(nm, amax) * sizeof(float4)) +
           align256(band_slots(nm, amax) * sizeof(unsigned short)) +
           align256(band_slots(nm, amax) / BD_REC * sizeof(float2)) +
           align256((size_t)nm * sizeof(int)) + align256(a1);
}

SetWs carve(char *&p, int nm, int amax) {
    const size_t a2 = (size_t)nm * amax * amax, a1 = (size_t)nm * amax;
    SetWs w;
    w.nnb = reinterpret_cast<int *>(p); p += align256(a1 * sizeof(int));
    w.xi = reinterpret_cast<double *>(p); p += align256(a2 * sizeof(double));
    w.self = reinterpret_cast<double *>(p); p += align256(a1 * sizeof(double));
    w.pk = reinterpret_cast<float4 *>(p); p += align256(a2 * sizeof(float4));
    w.pz = reinterpret_cast<float2 *>(p); p += align256(a2 * sizeof(float2));
    w.self32 = reinterpret_cast<float *>(p); p += align256(a1 * sizeof(float));
    w.cls = reinterpret_cast<signed char *>(p); p += align256(a2);
    w.acls = reinterpret_cast<signed char *>(p); p += align256(a1);
    w.selff = reinterpret_cast<float *>(p); p += align256(a1 * sizeof(float));
    const size_t slots = band_slots(nm, amax);
    w.spk = reinterpret_cast<float4 *>(p); p += align256(slots * sizeof(float4));
    w.smeta = reinterpret_cast<unsigned short *>(p); p += align256(slots * sizeof(unsigned short));
    w.band = reinterpret_cast<float2 *>(p); p += align256(slots / BD_REC * sizeof(float2));
    w.nrec = reinterpret_cast<int *>(p); p += align256((size_t)nm * sizeof(int));
    w.asc = reinterpret_cast<signed char *>(p); p += align256(a1);
    return w;
}

// exp(x) for the terms inside the window, x in [-16, 0] (the reduction holds to
// -700): x = k ln2 + r with ln2 in two parts, exp(r) by the polynomial of degree
// 11 that interpolates it at the Chebyshev nodes of [-ln2/2, ln2/2] widened by 0.05 %
// (k rounds a product that is itself rounded; relative error 1.5e-17; coefficients
// computed in 60 digits and rounded), the exponent added as an integer. Within 0.9 ulp (0.26 on average); half the instructions of the general
// function, which has to look after every argument.
__device__ __forceinline__ double exp_window(double x) {
    const double magic = 6755399441055744.0;  // 1.5 * 2^52: rounds to an integer
    const double kd = fma(x, 1.4426950408889634, magic);
    const int k = __double2loint(kd);
    const double n = kd - magic;
    const double r = fma(n, -2.3190468138462996e-17, fma(n, -0.6931471805599453, x));
    const double r2 = r * r;
    double e = fma(2.7632715071632255e-07, r2, 2.4801485278370062e-05);
    double o = fma(2.5110095611886237e-08, r2, 2.7557240761739257e-06);
    e = fma(e, r2, 0.0013888888952505406);
    o = fma(o, r2, 0.00019841269890193705);
    e = fma(e, r2, 0.04166666666648738);
    o = fma(o, r2, 0.008333333333319546);
    e = fma(e, r2, 0.5000000000000019);
    o = fma(o, r2, 0.1666666666666668);
    const double q = fma(o, r, e);
    const double p = fma(fma(q, r, 1.0), r, 1.0);
    return __hiloint2double(__double2hiint(p) + (k << 20), __double2loint(p));
}

// atomic_distl2 in FP64, reference order (farad_kernels.f90:58-88).
// x = descriptor of one atom (5, amax); xi = its sine factors.
__device__ double distl2_f64(const double *x1, const double *xi1, int n1, const double *x2,
                             const double *xi2, int n2, int amax, const AradParams &P) {
    double aad = 0.0;
    for (int m1 = 0; m1 < n1; ++m1) {
        const double r1 = x1[m1];
        const double p1 = x1[amax + m1], g1 = x1[2 * amax + m1];
        const double c1 = x1[3 * amax + m1], s1 = x1[4 * amax + m1];
        const double e1 = xi1[m1];
        for (int m2 = 0; m2 < n2; ++m2) {
            const double r2 = x2[m2];
            const double dr = __dsub_rn(r2, r1);
            const double t = __dmul_rn(dr, dr);
            if (t < P.maxg2) {
                double d = __dmul_rn(__dmul_rn(exp_window(__dmul_rn(t, P.inv_width)), e1), xi2[m2]);
                const double dp = __dsub_rn(p1, x2[amax + m2]);
                const double dg = __dsub_rn(g1, x2[2 * amax + m2]);
                const double st = __ddiv_rn(
                    __dmul_rn(__ddiv_rn(P.rw2, __dadd_rn(P.rw2, __dmul_rn(dp, dp))), P.cw2),
                    __dadd_rn(P.cw2, __dmul_rn(dg, dg)));
                d = __dmul_rn(d, st);
                const double ang = __dadd_rn(__dadd_rn(1.0, __dmul_rn(c1, x2[3 * amax + m2])),
                                             __dmul_rn(s1, x2[4 * amax + m2]));
                aad = __dadd_rn(aad, __dmul_rn(d, ang));
            }
        }
    }
    return aad;
}

// FP32 form over the packed neighbour records. The records hold the distance
// pre-scaled by rs = sqrt(-inv_width * log2 e), so exp(dr^2 inv_width) =
// exp2(-(dr')^2) and the window (dr)^2 < (8 w)^2 is (dr')^2 < maxg2s.
__device__ __forceinline__ float distl2_f32(const float4 *a, const float2 *za, int n1,
                                            const float4 *b, const float2 *zb, int n2,
                                            float maxg2s, float rw2, float cw2) {
    float aad = 0.0f;
    for (int m1 = 0; m1 < n1; ++m1) {
        const float4 u = a[m1];
        const float2 zu = za[m1];
        for (int m2 = 0; m2 < n2; ++m2) {
            const float4 v = b[m2];
            const float dr = v.x - u.x;
            const float t = dr * dr;
            if (t < maxg2s) {
                const float2 zv = zb[m2];
                const float dp = zu.x - zv.x, dg = zu.y - zv.y;
                const float st = __fdividef(rw2, rw2 + dp * dp) * __fdividef(cw2, cw2 + dg * dg);
                const float g = fmaf(u.z, v.z, fmaf(u.w, v.w, u.y * v.y));
                aad = fmaf(exp2f(-t) * st, g, aad);
            }
        }
    }
    return aad;
}

__host__ __device__ inline double fp32_scale(const AradParams &P) {
    return sqrt(-P.inv_width * 1.4426950408889634);
}

__device__ __forceinline__ int ptp_pos(double row, double col) {
    const double r = rint(row), c = rint(col);
    if (r != row || c != col || r < 0.0 || r > 7.0 || c < 0.0 || c > 33.0) return -1;
    return (int)r * 34 + (int)c;
}

// Marks a periodic-table position as present. The plain read first: nearly
// every mark repeats one already made, and thousands of atomics on the same
// few words serialise.
__device__ __forceinline__ void mark_class(ClassInfo *ci, int pos) {
    int *word = pos < 0 ? &ci->flag : &ci->present[pos];
    if (*(volatile int *)word == 0) atomicOr(word, 1);
}

// Stage 1: one warp per (molecule, atom), lanes over its neighbours
// (coalesced rows of the descriptor). With `ci` set, the periodic-table
// positions of the atom (Z) and of its neighbours are marked for the class
// tables in the same pass.
constexpr int PREP_WARPS = 4;
__global__ void __launch_bounds__(PREP_WARPS * 32)
arad_prep_kernel(const double *__restrict__ X, const double *__restrict__ Z,
                 const int *__restrict__ N, int nm, int amax, AradParams P, int conditional_sine,
                 SetWs w, ClassInfo *ci) {
    const long long gid = (long long)blockIdx.x * PREP_WARPS + (threadIdx.x >> 5);
    const int lane = threadIdx.x & 31;
    if (gid >= (long long)nm * amax) return;
    const int m = (int)(gid / amax), a = (int)(gid % amax);
    const int n = min(max(N[m], 0), amax);  // counts beyond amax are clamped
    const size_t base = (size_t)m * amax + a;
    if (a >= n) {
        if (lane == 0) w.nnb[base] = 0;
        return;
    }
    const double *x = X + base * 5 * amax;
    // neighbour prefix: the loop of atomic_distl2 exits at the first r > cut
    int cnt = n;
    for (int k0 = 0; k0 < n; k0 += 32) {
        const unsigned stop = __ballot_sync(0xffffffffu, k0 + lane < n && x[k0 + lane] > P.cut);
        if (stop) {
            cnt = k0 + __ffs(stop) - 1;
            break;
        }
    }
    double *xi = w.xi + base * amax;
    float4 *pk = w.pk + base * amax;
    float2 *pz = w.pz + base * amax;
    bool ascends = true;
    for (int k = lane; k < n; k += 32) {
        const double r = x[k];
        double s = 0.0;  // farad_kernels.f90:516 zero-initialised table
        if (!conditional_sine || r < P.cut) s = __dsub_rn(1.0, sin(__dmul_rn(r, P.inv_cut)));
        xi[k] = s;
        if (k < cnt) {
            const double c = x[3 * amax + k], sn = x[4 * amax + k];
            const double row = x[amax + k], col = x[2 * amax + k];
            pk[k] = make_float4((float)(r * fp32_scale(P)), (float)s, (float)(s * c),
                                (float)(s * sn));
            pz[k] = make_float2((float)row, (float)col);
            ascends = ascends && (k == 0 || r >= x[k - 1]);
            if (ci) mark_class(ci, ptp_pos(row, col));
        }
    }
    ascends = __all_sync(0xffffffffu, ascends);
    if (lane == 0) {
        w.nnb[base] = cnt;
        w.asc[base] = ascends ? 1 : 0;
        if (ci) mark_class(ci, ptp_pos(Z[base * 2 + 0], Z[base * 2 + 1]));
    }
}

// Self terms of the generic pair kernel, one thread per (molecule, atom).
// With `fast_ci` set they are needed only if the fast path is not usable.
__global__ void arad_generic_self_kernel(const double *__restrict__ X, const int *__restrict__ N,
                                         int nm, int amax, AradParams P, SetWs w,
                                         const ClassInfo *fast_ci) {
    if (fast_ci && fast_ci->flag == 0) return;
    const long long gid = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (gid >= (long long)nm * amax) return;
    const size_t base = (size_t)gid;
    const int cnt = w.nnb[base];
    const double *x = X + base * 5 * amax, *xi = w.xi + base * amax;
    const float4 *pk = w.pk + base * amax;
    const float2 *pz = w.pz + base * amax;
    w.self[base] = distl2_f64(x, xi, cnt, x, xi, cnt, amax, P);
    const float maxg2s = (float)(P.maxg2 * fp32_scale(P) * fp32_scale(P));
    w.self32[base] = distl2_f32(pk, pz, cnt, pk, pz, cnt, maxg2s, (float)P.rw2, (float)P.cw2);
}

__device__ __forceinline__ void pair_index(long long t, int symmetric, int nm2, int &I, int &J) {
    if (symmetric) {
        int j = (int)((sqrt(8.0 * (double)t + 1.0) - 1.0) * 0.5);
        while ((long long)j * (j + 1) / 2 > t) --j;
        while ((long long)(j + 1) * (j + 2) / 2 <= t) ++j;
        J = j;
        I = (int)(t - (long long)j * (j + 1) / 2);
    } else {
        I = (int)(t / nm2);
        J = (int)(t % nm2);
    }
}

// Stage 2: one warp per molecule pair; lanes stride over atom pairs.
// kDist: store every atom pair's l2 in D (nm1, nm2, amax, amax) instead of
// the kernel sums (atomic_arad_l2_distance_all, farad.f90:452-600).
// The bounds keep FP64 at four CTAs per SM, the distances at five: with the constants
// of the exponential in registers they took three and four (200 molecules of up to 33
// atoms, symmetric: 31.6 ms, 37.3 without the bound; 100 x 120 distances 28.9, 33.4). The
// lanes' atom pairs share j1 rather than i1 (28.2 ms; FP32, 40 atoms 14.3 instead of 38.7).
template <bool kF64, bool kDist = false>
__global__ void __launch_bounds__(128, kDist ? 5 : kF64 ? 4 : 0)
arad_pair_kernel(const double *__restrict__ X1, const double *__restrict__ Z1,
                 const int *__restrict__ N1, SetWs w1, int nm1, const double *__restrict__ X2,
                 const double *__restrict__ Z2, const int *__restrict__ N2, SetWs w2, int nm2,
                 int amax, AradParams P, SigmaTable sig, int nsig, int symmetric,
                 double *__restrict__ K, const ClassInfo *fast_ci,
                 double *__restrict__ D = nullptr) {
    // when the fast FP32 kernel handled this call, the generic one does nothing
    if (fast_ci && fast_ci->flag == 0) return;
    const int lane = threadIdx.x & 31;
    const long long npairs = symmetric ? (long long)nm1 * (nm1 + 1) / 2 : (long long)nm1 * nm2;
    const long long warp0 = ((long long)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const long long nwarps = ((long long)gridDim.x * blockDim.x) >> 5;
    const double eps = P.eps;
    const float maxg2s = (float)(P.maxg2 * fp32_scale(P) * fp32_scale(P));
    const float rw2f = (float)P.rw2, cw2f = (float)P.cw2;

    for (long long t = warp0; t < npairs; t += nwarps) {
        int I, J;
        pair_index(t, symmetric, nm2, I, J);
        const int nI = min(max(N1[I], 0), amax), nJ = min(max(N2[J], 0), amax);
        double acc[MAXSIG];
#pragma unroll
        for (int s = 0; s < MAXSIG; ++s) acc[s] = 0.0;
        const int P2 = nI * nJ;
        for (int p = lane; p < P2; p += 32) {
            // kernels: i1 fastest, the order in which the fast FP64 kernel sums its pairs too
            const int n1 = kDist ? nJ : nI, hi = p / n1, lo = p - hi * n1;
            const int i1 = kDist ? hi : lo, j1 = kDist ? lo : hi;
            const size_t b1 = (size_t)I * amax + i1, b2 = (size_t)J * amax + j1;
            const double dz1 = __dsub_rn(Z1[b1 * 2 + 0], Z2[b2 * 2 + 0]);
            const double dz2 = __dsub_rn(Z1[b1 * 2 + 1], Z2[b2 * 2 + 1]);
            const double stoch = __ddiv_rn(
                __dmul_rn(__ddiv_rn(P.rw2, __dadd_rn(P.rw2, __dmul_rn(dz1, dz1))), P.cw2),
                __dadd_rn(P.cw2, __dmul_rn(dz2, dz2)));
            double l2;
            if (kF64) {
                const double S = distl2_f64(X1 + b1 * 5 * amax, w1.xi + b1 * amax, w1.nnb[b1],
                                            X2 + b2 * 5 * amax, w2.xi + b2 * amax, w2.nnb[b2],
                                            amax, P);
                l2 = __dsub_rn(__dadd_rn(w1.self[b1], w2.self[b2]),
                               __dmul_rn(__dmul_rn(2.0, S), stoch));
            } else {
                const float S = distl2_f32(w1.pk + b1 * amax, w1.pz + b1 * amax, w1.nnb[b1],
                                           w2.pk + b2 * amax, w2.pz + b2 * amax, w2.nnb[b2],
                                           maxg2s, rw2f, cw2f);
                l2 = (double)(w1.self32[b1] + w2.self32[b2] - 2.0f * S * (float)stoch);
            }
            if (fabs(l2) < eps) l2 = 0.0;  // :594
            if (kDist) {  // farad.f90:589
                D[(((size_t)I * nm2 + J) * amax + i1) * amax + j1] = l2;
                continue;
            }
#pragma unroll
            for (int s = 0; s < MAXSIG; ++s)
                if (s < nsig) acc[s] += exp(l2 * sig.inv_sigma2[s]);
        }
        if (kDist) continue;
#pragma unroll
        for (int s = 0; s < MAXSIG; ++s) {
            if (s < nsig) {
                double v = acc[s];
                for (int o = 16; o; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
                if (lane == 0) {
                    K[((size_t)s * nm1 + I) * nm2 + J] = v;
                    if (symmetric) K[((size_t)s * nm1 + J) * nm2 + I] = v;  // :744
                }
            }
        }
    }
}

// ---------------------------------------------------------------------------
// Fast FP32 path.
//
// Molecule I's neighbour records (one record = one neighbour m1 of one atom
// i1) are packed, whole atoms at a time, into passes of 32 lanes; molecule J
// is staged in shared memory. A work item (pass p, atom j1 of J) lets every
// lane sum its record against all of j1's neighbours (broadcast reads), then a
// segmented warp scan forms S(i1, j1) for every atom i1 of the pass at the
// last lane of its segment, which applies the kernel exponentials for every
// sigma. Self terms come from the same code (J = I), so l2 cancels exactly for
// identical environments.
// ---------------------------------------------------------------------------
constexpr int FC_BM = 8, FC_WARPS = 8, FC_MAXREC = 1024, FC_MAXA = 32, FC_MAXSIG = 8;
constexpr int FC_SST = FC_MAXC + 1;

// One CTA: class ids in position order and the stoichiometric tables
// (farad_kernels.f90:80-81).
constexpr int CB_TPB = 288;  // >= FC_NPOS and FC_MAXC^2
static_assert(CB_TPB >= FC_NPOS && CB_TPB >= FC_MAXC * FC_MAXC, "one thread per entry");
__global__ void __launch_bounds__(CB_TPB)
arad_class_build_kernel(ClassInfo *ci, double rw2, double cw2) {
    __shared__ int rows[FC_MAXC], cols[FC_MAXC], before[CB_TPB / 32 + 1];
    const int pos = threadIdx.x, warp = pos >> 5, lane = pos & 31;
    const bool here = pos < FC_NPOS && ci->present[pos];
    const unsigned mask = __ballot_sync(0xffffffffu, here);
    if (lane == 0) before[warp + 1] = __popc(mask);
    if (pos == 0) before[0] = 0;
    __syncthreads();
    if (pos == 0)
        for (int q = 0; q < CB_TPB / 32; ++q) before[q + 1] += before[q];
    __syncthreads();
    const int nc = min(before[CB_TPB / 32], FC_MAXC);
    const int c = before[warp] + __popc(mask & ((1u << lane) - 1));
    if (pos < FC_NPOS) ci->map[pos] = here && c < FC_MAXC ? (signed char)c : -1;
    if (here && c < FC_MAXC) {
        rows[c] = pos / 34;
        cols[c] = pos % 34;
    }
    __syncthreads();
    if (pos == 0) {
        ci->ncls = nc;
        if (before[CB_TPB / 32] > FC_MAXC) ci->flag |= 2;
    }
    if (pos < FC_MAXC * FC_MAXC) {
        const int a = pos / FC_MAXC, b = pos % FC_MAXC;
        double v = 0.0;
        if (a < nc && b < nc) {
            const double dr = (double)(rows[a] - rows[b]), dc = (double)(cols[a] - cols[b]);
            // the operations of the pair loop (distl2_f64), so the same value
            v = __ddiv_rn(__dmul_rn(__ddiv_rn(rw2, __dadd_rn(rw2, __dmul_rn(dr, dr))), cw2),
                          __dadd_rn(cw2, __dmul_rn(dc, dc)));
        }
        ci->stoch64[pos] = v;
        ci->stoch[pos] = (float)v;
    }
}

// Element classes of every neighbour record and atom (after the class build);
// one thread per (molecule, atom, neighbour).
__global__ void arad_class_assign_kernel(const double *__restrict__ X, const double *__restrict__ Z,
                                         const int *__restrict__ N, int nm, int amax,
                                         const ClassInfo *ci, SetWs w) {
    const long long gid = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (gid >= (long long)nm * amax * amax) return;
    const size_t base = (size_t)(gid / amax);
    const int k = (int)(gid % amax);
    const int m = (int)(base / amax), a = (int)(base % amax);
    const int n = min(max(N[m], 0), amax);
    if (k == 0) {
        const int pos = a < n ? ptp_pos(Z[base * 2 + 0], Z[base * 2 + 1]) : -1;
        w.acls[base] = pos >= 0 ? max((int)ci->map[pos], 0) : 0;
    }
    if (a < n && k < w.nnb[base]) {
        const double *x = X + base * 5 * amax;
        const int pos = ptp_pos(x[amax + k], x[2 * amax + k]);
        w.cls[base * amax + k] = pos >= 0 ? (signed char)max((int)ci->map[pos], 0) : 0;
    }
}

// Paired path (at most FC_PC element classes): the records of J are stored two
// at a time, (r0, r1, xi0, xi1) and (xc0, xc1, xs0, xs1), so every lane
// evaluates two neighbour pairs per step with packed FP32x2 arithmetic
// (FADD2 / FMUL2 / FFMA2) and fetches both stoichiometric factors with one
// load from a per-class pair table. An atom with an odd neighbour count gets
// a padding record (r = 1e18, xi = 0) whose window test and exponential are 0.
constexpr int FC_PC = 8;
constexpr int FC_PTS = FC_PC * FC_PC + 1;  // pair-table row stride (float2): conflict-free rows
constexpr int FC_SS = FC_MAXA + 1;         // S row stride: lanes adding to different atoms i1
                                           // of one column j1 hit different banks

// Scalar path (more classes): one molecule pair at a time.
struct FastSmem {
    float4 recI[FC_MAXREC];      // molecule I, dense by atom, 32 records per pass
    int metaI[FC_MAXREC];        // atom | seg_start << 8 | cls << 16 | active << 24 | tail << 25
    float selfI[FC_MAXA];
    int aclsI[FC_MAXA];
    float4 recJ[FC_MAXREC];      // molecule J, dense by atom
    signed char clsJ[FC_MAXREC];  // element class of each record of J
    int offJ[FC_MAXA + 1];       // record offsets
    float selfJ[FC_MAXA];
    int aclsJ[FC_MAXA];
    float stoch[FC_MAXC * FC_SST];  // row stride 17: lanes of different classes hit distinct banks
    float S[FC_MAXA * FC_SS];       // S(i1, j1), row stride FC_SS
    float red[FC_WARPS][FC_MAXSIG];
    int npassI, nI, nJ;
};

// Molecule I, dense: pass p holds records [32 p, 32 p + 32). Whole CTA; the
// caller synchronises before the records are read.
__device__ void fast_load_I(FastSmem &sm, const SetWs &w, int I, int amax, int nI,
                            bool use_self) {
    __shared__ int offI[FC_MAXA + 1];
    if (threadIdx.x < 32) {  // exclusive prefix of the neighbour counts (nI <= 32)
        const int a = threadIdx.x;
        const int cnt = a < nI ? w.nnb[(size_t)I * amax + a] : 0;
        int incl = cnt;
        for (int d = 1; d < 32; d <<= 1) {
            const int o = __shfl_up_sync(0xffffffffu, incl, d);
            if (a >= d) incl += o;
        }
        offI[a] = incl - cnt;
        if (a == 31) {
            offI[32] = incl;
            sm.npassI = (incl + 31) / 32;
            sm.nI = nI;
        }
    }
    __syncthreads();
    const int nrec = offI[32];
    const int nslot = sm.npassI * 32;
    for (int slot = nrec + threadIdx.x; slot < nslot; slot += blockDim.x) {
        sm.metaI[slot] = ((slot & 31) << 8);  // inactive lane, own segment, no tail
        sm.recI[slot] = make_float4(0.f, 0.f, 0.f, 0.f);
    }
    for (int t = threadIdx.x; t < nI * amax; t += blockDim.x) {
        const int a = t / amax, k = t % amax;
        const int beg = offI[a], cnt = offI[a + 1] - beg;
        if (k < cnt) {
            const int slot = beg + k;
            // segment = this atom's records inside this pass
            const int seg = max(beg, slot & ~31) & 31;
            const bool tail = (k == cnt - 1) || ((slot & 31) == 31);
            const size_t src = ((size_t)I * amax + a) * amax + k;
            sm.metaI[slot] = a | (seg << 8) | ((int)w.cls[src] << 16) | (1 << 24) |
                             ((tail ? 1 : 0) << 25);
            sm.recI[slot] = w.pk[src];
        }
    }
    for (int a = threadIdx.x; a < nI; a += blockDim.x) {
        sm.selfI[a] = use_self ? w.selff[(size_t)I * amax + a] : 0.0f;
        sm.aclsI[a] = w.acls[(size_t)I * amax + a];
    }
}

// Molecule J, dense by atom. Whole CTA; the caller synchronises before the
// records are read.
__device__ void fast_load_J(FastSmem &sm, const SetWs &w, int J, int amax, int nJ,
                            bool use_self) {
    if (threadIdx.x < 32) {  // exclusive prefix of the neighbour counts (nJ <= 32)
        const int a = threadIdx.x;
        const int cnt = a < nJ ? w.nnb[(size_t)J * amax + a] : 0;
        int incl = cnt;
        for (int d = 1; d < 32; d <<= 1) {
            const int o = __shfl_up_sync(0xffffffffu, incl, d);
            if (a >= d) incl += o;
        }
        sm.offJ[a] = incl - cnt;
        if (a == 31) {
            sm.offJ[32] = incl;
            sm.nJ = nJ;
        }
    }
    __syncthreads();
    for (int t = threadIdx.x; t < nJ * amax; t += blockDim.x) {
        const int a = t / amax, k = t % amax;
        if (k < sm.offJ[a + 1] - sm.offJ[a]) {
            const int d = sm.offJ[a] + k;
            const size_t src = ((size_t)J * amax + a) * amax + k;
            sm.recJ[d] = w.pk[src];
            sm.clsJ[d] = w.cls[src];
        }
    }
    for (int a = threadIdx.x; a < nJ; a += blockDim.x) {
        sm.selfJ[a] = use_self ? w.selff[(size_t)J * amax + a] : 0.0f;
        sm.aclsJ[a] = w.acls[(size_t)J * amax + a];
    }
}

// Work item (pass p, atom j1): the segment sums of the pass against j1 are
// added into S[i1][j1] by each segment's last lane (an atom split across two
// passes contributes two partial sums; two terms commute, so the result does
// not depend on their order).
__device__ __forceinline__ void fast_item(FastSmem &sm, int p, int j1, float maxg2s) {
    const int lane = threadIdx.x & 31;
    const float4 u = sm.recI[p * 32 + lane];
    const int meta = sm.metaI[p * 32 + lane];
    const float *strow = sm.stoch + ((meta >> 16) & 0xff) * FC_SST;
    const int beg = sm.offJ[j1], end = sm.offJ[j1 + 1];
    float acc = 0.0f;
#pragma unroll 4
    for (int m2 = beg; m2 < end; ++m2) {
        const float4 q = sm.recJ[m2];
        const float dr = q.x - u.x;
        const float t = dr * dr;
        float e;
        asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(e) : "f"(-t));
        const float g = fmaf(u.w, q.w, fmaf(u.z, q.z, u.y * q.y));
        const float eg = e * strow[sm.clsJ[m2]];
        if (t < maxg2s) acc = fmaf(eg, g, acc);
    }
    const int seg = (meta >> 8) & 0xff;
    float v = acc;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
        const float o = __shfl_up_sync(0xffffffffu, v, d);
        if (lane - d >= seg) v += o;
    }
    if ((meta >> 25) & 1) atomicAdd(&sm.S[(meta & 0xff) * FC_SS + j1], v);
}

// All work items of one molecule pair, S cleared first. Whole CTA.
__device__ __forceinline__ void fast_pair_sums(FastSmem &sm, int nJ, float maxg2s) {
    for (int t = threadIdx.x; t < FC_MAXA * FC_SS; t += blockDim.x) sm.S[t] = 0.0f;
    __syncthreads();
    const int warp = threadIdx.x >> 5;
    const int items = sm.npassI * nJ;
    for (int it = warp; it < items; it += FC_WARPS) fast_item(sm, it / nJ, it % nJ, maxg2s);
    __syncthreads();
}

__device__ __forceinline__ void load_stoch(float *stoch, const ClassInfo *ci) {
    for (int t = threadIdx.x; t < FC_MAXC * FC_MAXC; t += blockDim.x)
        stoch[(t / FC_MAXC) * FC_SST + t % FC_MAXC] = ci->stoch[t];
}

__device__ __forceinline__ void pair_block(long long t, int symmetric, int nbj, int &bi, int &bj) {
    if (symmetric) {  // blocks bi <= bj
        int r = (int)((sqrt(8.0 * (double)t + 1.0) - 1.0) * 0.5);
        while ((long long)r * (r + 1) / 2 > t) --r;
        while ((long long)(r + 1) * (r + 2) / 2 <= t) ++r;
        bj = r;
        bi = (int)(t - (long long)r * (r + 1) / 2);
    } else {
        bi = (int)(t / nbj);
        bj = (int)(t % nbj);
    }
}

// Records of one molecule sorted by r (ties by atom, then neighbour index):
// the I-side layout of the paired path. One CTA per molecule, bitonic sort
// of 64-bit keys (r bits << 32 | atom * 32 + k) in shared memory.
__global__ void __launch_bounds__(FC_WARPS * 32)
arad_sort_records_kernel(SetWs w, const int *__restrict__ N, int nm, int amax,
                         const ClassInfo *ci) {
    __shared__ unsigned long long key[FC_MAXREC];
    __shared__ int off[FC_MAXA + 1];
    if (ci->flag || ci->ncls > FC_PC) return;
    const int I = blockIdx.x;
    if (I >= nm) return;
    const int nI = min(max(N[I], 0), amax);
    if (threadIdx.x < 32) {
        const int a = threadIdx.x;
        const int cnt = a < nI ? w.nnb[(size_t)I * amax + a] : 0;
        int incl = cnt;
        for (int d = 1; d < 32; d <<= 1) {
            const int o = __shfl_up_sync(0xffffffffu, incl, d);
            if (a >= d) incl += o;
        }
        off[a] = incl - cnt;
        if (a == 31) off[32] = incl;
    }
    __syncthreads();
    const int nrec = off[32];
    int len = 1;
    while (len < nrec) len <<= 1;
    for (int t = threadIdx.x; t < len; t += blockDim.x) key[t] = ~0ull;
    __syncthreads();
    for (int t = threadIdx.x; t < nI * amax; t += blockDim.x) {
        const int a = t / amax, k = t % amax;
        if (k < off[a + 1] - off[a]) {
            const float r = w.pk[((size_t)I * amax + a) * amax + k].x;
            key[off[a] + k] = ((unsigned long long)__float_as_uint(r) << 32) |
                              (unsigned)(a * FC_MAXA + k);
        }
    }
    __syncthreads();
    for (int size = 2; size <= len; size <<= 1)
        for (int stride = size >> 1; stride > 0; stride >>= 1) {
            for (int t = threadIdx.x; t < len; t += blockDim.x) {
                const int partner = t ^ stride;
                if (partner > t) {
                    const bool up = (t & size) == 0;
                    const unsigned long long x = key[t], y = key[partner];
                    if ((x > y) == up) {
                        key[t] = y;
                        key[partner] = x;
                    }
                }
            }
            __syncthreads();
        }
    // Inside a group of 64 two records of one atom go to one lane, as far as they
    // come in twos: the lane then adds to S once instead of twice. Twos take the
    // lanes in the order in which they are completed, then the atoms' odd records
    // in the order of the atoms; slots past them stay unused.
    const size_t base = (size_t)I * band_stride(amax);
    const int slots = (nrec + BD_REC - 1) / BD_REC * BD_REC;
    for (int t = threadIdx.x; t < slots; t += blockDim.x) {
        w.spk[base + t] = make_float4(0.f, 0.f, 0.f, 0.f);
        w.smeta[base + t] = 0;
    }
    __syncthreads();
    for (int t = threadIdx.x; t < nrec; t += blockDim.x) {
        const int beg = t / BD_REC * BD_REC, end = min(beg + BD_REC, nrec);
        const auto atom = [&](int q) { return (int)(key[q] & 0xffffffffu) / FC_MAXA; };
        const int a = atom(t), k = (int)(key[t] & 0xffffffffu) % FC_MAXA;
        int rank = 0, same = 0;  // among the group's records of this atom
        for (int q = beg; q < end; ++q) {
            rank += q < t && atom(q) == a;
            same += atom(q) == a;
        }
        const bool one = (same & 1) && rank == same - 1;
        int done = t;  // where t's two is completed
        if (one)
            done = end;
        else if (!(rank & 1))
            while (atom(++done) != a) {}
        int twos = 0;  // completed before that
        unsigned odd = 0;
        for (int q = beg; q < end; ++q) {
            const unsigned bit = 1u << atom(q);
            twos += q < done && (odd & bit);
            odd ^= bit;
        }
        const int ones = __popc(odd & ((1u << a) - 1));
        const int slot = one ? twos + (ones >> 1) + 32 * (ones & 1) : twos + 32 * (rank & 1);
        const size_t src = ((size_t)I * amax + a) * amax + k;
        const float4 rec = w.pk[src];
        w.spk[base + beg + slot] = rec;
        w.smeta[base + beg + slot] = (unsigned short)(a | ((int)w.cls[src] << 8) | (1 << 15));
        float2 *band = w.band + base / BD_REC + t / BD_REC;
        if (t == beg) band->x = rec.x;
        if (t == end - 1) band->y = rec.x;
    }
    if (threadIdx.x == 0) w.nrec[I] = nrec;
}

// ---- the paired path's pair sums ---------------------------------------------
// A CTA takes tiles of FC_BM molecules I and J, as many J at a time as its shared
// memory holds beside the records of one I:
//   1. for each group of 64 records of I and each atom j1 the range of j1's
//      record pairs inside the group's band widened by the (8 w)^2 window;
//   2. a warp keeps a group's records in registers, two to a lane, and walks the
//      atoms j1: each record pair of j1 is loaded once for four evaluations.
//      Terms outside a record's own window are masked, so that what is skipped
//      and what is masked are both exactly zero;
//   3. a lane's sums are added to S(i1, j1) in 2^-32 fixed point: the result does
//      not depend on the order of the additions. 64 bits as two 32-bit words
//      with a carry: the 64-bit shared-memory atomic is a compare-and-swap loop;
//   4. the kernel exponentials of every l2 and sigma, in an order that depends on
//      the two molecules' atoms alone.
// Bound by the instructions issued: 38 for a step of 2 (128 evaluations, of which 14
// packed FP32 and 4 exponentials, 8 cycles of their units each), about 45 to add a
// lane's sums, 5000 per molecule pair outside of the steps. 500 x 3001 molecules of
// at most 23 atoms, 5 sigmas: 29.7 ms; 39.7 with one J at a time, the ranges found
// by every warp for itself and the compare-and-swap loop, which took half of the
// shared memory's cycles.
constexpr int BD_JA = 96;     // atoms J at a time
struct BandSmem {
    float2 pt[FC_PC * FC_PTS];      // pt[c1][ca * FC_PC + cb] = (stoch(c1, ca), stoch(c1, cb))
    float stoch[FC_MAXC * FC_SST];  // row stride 17: lanes of different classes hit distinct banks
    float sc[FC_MAXSIG];            // log2 e / sigma^2, negative
    float selfI[FC_MAXA];
    float selfJ[BD_JA];
    float red[FC_BM][FC_WARPS][FC_MAXSIG];
    int aclsI[FC_MAXA];
    int nI[FC_BM], recI[FC_BM];     // molecules I of the tile: atoms, records
    int nJ[FC_BM], pairsJ[FC_BM];   // molecules J of the tile: atoms, record pairs
    short offJ[BD_JA + 1];          // first record pair of each atom J
    short atomJ[FC_BM + 1];         // first atom of each molecule J at a time
    unsigned char aclsJ[BD_JA];
};
// four CTAs per SM, with 1 KB for the system and the scalar path's offsets each
constexpr size_t kBandSmem = 56 * 1024 - 256;
constexpr size_t kBandArena = kBandSmem - (sizeof(BandSmem) + 15) / 16 * 16;

struct BandArena {
    float4 *rec;            // molecule I, groups of 64
    float4 *pair;           // molecules J: (r0, r1, xi0, xi1), (xc0, xc1, xs0, xs1) by turns
    unsigned *lo, *hi;      // S(i1, j1) in fixed point at j1 * ld + i1
    unsigned short *meta;   // as SetWs::smeta
    short2 *win;            // first and past-the-last record pair by group and atom j1
    unsigned char *pk;      // cls0 * FC_PC + cls1: column of the pair table
    int ld;                 // odd: lanes adding to different atoms i1 hit different banks
};
__host__ __device__ constexpr size_t band_bytes(int recs, int pairs, int atoms, int ld) {
    return (size_t)recs * 18 + (size_t)pairs * 33 + (size_t)atoms * ld * 8 +
           (size_t)atoms * (recs / BD_REC) * 4;
}
static_assert(band_bytes(FC_MAXREC, FC_MAXREC / 2, FC_MAXA, FC_MAXA + 1) <= kBandArena &&
              FC_MAXA <= BD_JA && FC_MAXREC / 2 < 32768 && FC_WARPS == FC_BM,
              "one pair of the largest molecules fits");
constexpr size_t kFastSmem =
    sizeof(FastSmem) > kBandSmem ? sizeof(FastSmem) : kBandSmem;  // whichever path the classes decide

__device__ __forceinline__ BandArena band_carve(unsigned char *p, int recs, int pairs, int atoms,
                                                int ld) {
    BandArena A;
    A.rec = reinterpret_cast<float4 *>(p);
    A.pair = A.rec + recs;
    A.lo = reinterpret_cast<unsigned *>(A.pair + 2 * pairs);
    A.hi = A.lo + atoms * ld;
    A.win = reinterpret_cast<short2 *>(A.hi + atoms * ld);
    A.meta = reinterpret_cast<unsigned short *>(A.win + atoms * (recs / BD_REC));
    A.pk = reinterpret_cast<unsigned char *>(A.meta + recs);
    A.ld = ld;
    return A;
}

__device__ __forceinline__ void band_load_tables(BandSmem &sm, const ClassInfo *ci) {
    load_stoch(sm.stoch, ci);
    for (int t = threadIdx.x; t < FC_PC * FC_PC * FC_PC; t += blockDim.x) {
        const int c1 = t / (FC_PC * FC_PC), k = t % (FC_PC * FC_PC);
        const int ca = k / FC_PC, cb = k % FC_PC;
        sm.pt[c1 * FC_PTS + k] =
            make_float2(ci->stoch[c1 * FC_MAXC + ca], ci->stoch[c1 * FC_MAXC + cb]);
    }
}

// Sizes of the tile's molecules: warp q takes the q-th of each side.
__device__ __forceinline__ void band_sizes(BandSmem &sm, const SetWs &w1, const int *N1, int I0,
                                           int nm1, const SetWs &w2, const int *N2, int J0,
                                           int nm2, int amax) {
    const int q = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int I = I0 + q, J = J0 + q;
    const int nJ = J < nm2 ? min(max(N2[J], 0), amax) : 0;
    int pairs = lane < nJ ? (w2.nnb[(size_t)J * amax + lane] + 1) >> 1 : 0;
    for (int o = 16; o; o >>= 1) pairs += __shfl_xor_sync(0xffffffffu, pairs, o);
    if (lane == 0) {
        sm.nI[q] = I < nm1 ? min(max(N1[I], 0), amax) : 0;
        sm.recI[q] = I < nm1 ? w1.nrec[I] : 0;
        sm.nJ[q] = nJ;
        sm.pairsJ[q] = pairs;
    }
}

// Molecules J .. J + count - 1 (the tile's from j0 on) in record pairs. Whole CTA,
// with a barrier inside; the caller synchronises before the records are read.
__device__ __forceinline__ void band_load_J(BandSmem &sm, const BandArena &A, const SetWs &w, int J,
                                            int j0, int count, int amax, bool use_self) {
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    if (warp < count) {  // offsets: warp q takes the q-th molecule
        int atoms = 0, beg = 0;
        for (int q = 0; q < warp; ++q) {
            atoms += sm.nJ[j0 + q];
            beg += sm.pairsJ[j0 + q];
        }
        const int n = sm.nJ[j0 + warp];
        const size_t a = (size_t)(J + warp) * amax + lane;
        const int np = lane < n ? (w.nnb[a] + 1) >> 1 : 0;
        int incl = np;
        for (int d = 1; d < 32; d <<= 1) {
            const int o = __shfl_up_sync(0xffffffffu, incl, d);
            if (lane >= d) incl += o;
        }
        if (lane < n) {
            sm.offJ[atoms + lane] = (short)(beg + incl - np);
            sm.selfJ[atoms + lane] = use_self ? w.selff[a] : 0.0f;
            sm.aclsJ[atoms + lane] = (unsigned char)w.acls[a];
        }
        if (lane == 31) {
            sm.atomJ[warp] = (short)atoms;
            if (warp == count - 1) {
                sm.atomJ[count] = (short)(atoms + n);
                sm.offJ[atoms + n] = (short)(beg + incl);
            }
        }
    }
    __syncthreads();
    // 16 threads per atom, a record pair each
    const int q = threadIdx.x & 15;
    int m = 0;
    for (int j = threadIdx.x >> 4; j < sm.atomJ[count]; j += FC_WARPS * 2) {
        while (j >= sm.atomJ[m + 1]) ++m;
        const int beg = sm.offJ[j];
        if (q >= sm.offJ[j + 1] - beg) continue;
        const size_t base = (size_t)(J + m) * amax + j - sm.atomJ[m], src = base * amax + 2 * q;
        const float4 r0 = w.pk[src];
        const int c0 = w.cls[src];
        float4 r1 = make_float4(1.0e18f, 0.0f, 0.0f, 0.0f);
        int c1 = 0;
        if (2 * q + 1 < w.nnb[base]) {
            r1 = w.pk[src + 1];
            c1 = w.cls[src + 1];
        }
        A.pair[2 * (beg + q)] = make_float4(r0.x, r1.x, r0.y, r1.y);
        A.pair[2 * (beg + q) + 1] = make_float4(r0.z, r1.z, r0.w, r1.w);
        A.pk[beg + q] = (unsigned char)(c0 * FC_PC + c1);
    }
}

// Molecule I of the tile (the i-th), S cleared, and the ranges of step 1 of its groups with the
// atoms J (loaded before). Whole CTA; the caller synchronises before use.
__device__ __forceinline__ void band_load_I(BandSmem &sm, const BandArena &A, const SetWs &w, int I,
                                            int i, int count, int amax, float wd, bool use_self) {
    const int nat = sm.atomJ[count], groups = (sm.recI[i] + BD_REC - 1) / BD_REC;
    const size_t base = (size_t)I * band_stride(amax);
    for (int t = threadIdx.x; t < groups * BD_REC; t += blockDim.x) {
        A.rec[t] = w.spk[base + t];
        A.meta[t] = w.smeta[base + t];
    }
    for (int t = threadIdx.x; t < nat * A.ld; t += blockDim.x) A.lo[t] = A.hi[t] = 0;
    for (int a = threadIdx.x; a < sm.nI[i]; a += blockDim.x) {
        sm.selfI[a] = use_self ? w.selff[(size_t)I * amax + a] : 0.0f;
        sm.aclsI[a] = w.acls[(size_t)I * amax + a];
    }
    for (int t = threadIdx.x; t < nat * groups; t += blockDim.x) {
        const int g = t / nat, j = t - g * nat;
        const float2 band = w.band[base / BD_REC + g];
        const float lo = band.x - wd, hi = band.y + wd;
        int below = sm.offJ[j], before = below;
        for (int q = below, end = sm.offJ[j + 1]; q < end; ++q) {
            const float2 r = *reinterpret_cast<const float2 *>(A.pair + 2 * q);
            below += !(r.y > lo);
            before += r.x < hi;
        }
        A.win[t] = make_short2((short)below, (short)before);
    }
}

// One record u (its r negated, as pairs of equals) against a record pair.
struct BandRec {
    float2 nx, y, z, w;
    __device__ explicit BandRec(const float4 &u)
        : nx(make_float2(-u.x, -u.x)), y(make_float2(u.y, u.y)), z(make_float2(u.z, u.z)),
          w(make_float2(u.w, u.w)) {}
};
__device__ __forceinline__ float2 band_terms(const BandRec &u, const float4 &a, const float4 &b,
                                             float2 st, float maxg2s, float2 acc) {
    const float2 dr = __fadd2_rn(make_float2(a.x, a.y), u.nx);
    const float2 t = __fmul2_rn(dr, dr);
    float e0, e1;  // outside the window exactly zero
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(e0) : "f"(t.x < maxg2s ? -t.x : -1.0e30f));
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(e1) : "f"(t.y < maxg2s ? -t.y : -1.0e30f));
    const float2 g = __ffma2_rn(make_float2(b.z, b.w), u.w,
                                __ffma2_rn(make_float2(b.x, b.y), u.z,
                                           __fmul2_rn(make_float2(a.z, a.w), u.y)));
    return __ffma2_rn(__fmul2_rn(make_float2(e0, e1), st), g, acc);
}

__device__ __forceinline__ void band_add(unsigned *lo, int hi, long long f) {
    const unsigned l = (unsigned)f;
    unsigned h = (unsigned)((unsigned long long)f >> 32);
    h += atomicAdd(lo, l) > ~l;  // the carry
    if (h) atomicAdd(lo + hi, h);
}

// Steps 2 and 3 for the atoms J from jfirst on. Whole CTA.
__device__ __forceinline__ void band_sums(const BandSmem &sm, const BandArena &A, int i, int jfirst,
                                          int nat, float maxg2s) {
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int groups = (sm.recI[i] + BD_REC - 1) / BD_REC, hi = (int)(A.hi - A.lo);
    for (int g = 0; g < groups; ++g) {
        const BandRec u0(A.rec[g * BD_REC + lane]), u1(A.rec[g * BD_REC + 32 + lane]);
        const int meta0 = A.meta[g * BD_REC + lane], meta1 = A.meta[g * BD_REC + 32 + lane];
        const float2 *pt0 = sm.pt + ((meta0 >> 8) & 0x7f) * FC_PTS;
        const float2 *pt1 = sm.pt + ((meta1 >> 8) & 0x7f) * FC_PTS;
        unsigned *s0 = A.lo + (meta0 & 0xff), *s1 = A.lo + (meta1 & 0xff);
        const bool both = ((meta0 ^ meta1) & 0x80ff) == 0;  // two records of one atom
        // the atoms that are left over after the eights go to other warps in each group
        for (int j = jfirst + ((warp + 3 * g) & (FC_WARPS - 1)); j < nat; j += FC_WARPS) {
            const short2 win = A.win[g * nat + j];
            float2 acc0 = make_float2(0.0f, 0.0f), acc1 = make_float2(0.0f, 0.0f);
#pragma unroll 2
            for (int m = win.x; m < win.y; ++m) {
                const float4 a = A.pair[2 * m], b = A.pair[2 * m + 1];
                const int k = A.pk[m];
                acc0 = band_terms(u0, a, b, pt0[k], maxg2s, acc0);
                acc1 = band_terms(u1, a, b, pt1[k], maxg2s, acc1);
            }
            // unused slots: records of zeros, whose sums are zero
            long long f0 = __float2ll_rn((acc0.x + acc0.y) * 4294967296.0f);
            const long long f1 = __float2ll_rn((acc1.x + acc1.y) * 4294967296.0f);
            if (both) f0 += f1;
            if (f0) band_add(s0 + j * A.ld, hi, f0);
            if (!both && f1) band_add(s1 + j * A.ld, hi, f1);
        }
    }
}

__device__ __forceinline__ float band_value(const BandArena &A, int idx) {
    const long long q = (long long)((unsigned long long)A.hi[idx] << 32 | A.lo[idx]);
    return (float)((double)q * 2.3283064365386963e-10);
}

// The paired path of a tile: molecules I0 .. and J0 .. (FC_BM of each).
__device__ __forceinline__ void band_tile(unsigned char *smem, const SetWs &w1, const int *N1,
                                          int nm1, const SetWs &w2, const int *N2, int nm2, int I0,
                                          int J0, int amax, float maxg2s, float eps,
                                          const ClassInfo *ci, const SigmaTable &sig, int nsig,
                                          int symmetric, double *K) {
    BandSmem &sm = *reinterpret_cast<BandSmem *>(smem);
    unsigned char *arena = smem + (sizeof(BandSmem) + 15) / 16 * 16;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const float wd = sqrtf(maxg2s) * 1.0001f;  // a little wider than the window
    band_load_tables(sm, ci);
#pragma unroll
    for (int s = 0; s < FC_MAXSIG; ++s)
        if (threadIdx.x == s && s < nsig)
            sm.sc[s] = (float)(sig.inv_sigma2[s] * 1.4426950408889634);
    band_sizes(sm, w1, N1, I0, nm1, w2, N2, J0, nm2, amax);
    __syncthreads();
    const int ni = min(FC_BM, nm1 - I0), nj = min(FC_BM, nm2 - J0);
    int recs = 0, ld = 1;
    for (int i = 0; i < ni; ++i) {
        recs = max(recs, (sm.recI[i] + BD_REC - 1) / BD_REC * BD_REC);
        ld = max(ld, sm.nI[i] | 1);
    }
    for (int j0 = 0, count; j0 < nj; j0 += count) {
        int atoms = sm.nJ[j0], pairs = sm.pairsJ[j0];
        for (count = 1; j0 + count < nj; ++count) {
            const int a = atoms + sm.nJ[j0 + count], p = pairs + sm.pairsJ[j0 + count];
            if (a > BD_JA || band_bytes(recs, p, a, ld) > kBandArena) break;
            atoms = a;
            pairs = p;
        }
        const BandArena A = band_carve(arena, recs, pairs, atoms, ld);
        __syncthreads();  // the molecules J before are done with
        band_load_J(sm, A, w2, J0 + j0, j0, count, amax, true);
        __syncthreads();
        for (int i = 0; i < ni; ++i) {
            const int I = I0 + i, nI = sm.nI[i];
            const int first = symmetric ? max(0, I - J0 - j0) : 0;  // J >= I
            if (first >= count) continue;
            band_load_I(sm, A, w1, I, i, count, amax, wd, true);
            __syncthreads();
            band_sums(sm, A, i, sm.atomJ[first], atoms, maxg2s);
            __syncthreads();
            for (int m = first; m < count; ++m) {
                // elements 32 part .. of every 256; which warp takes them does not matter
                const int part = (warp + 3 * m) & (FC_WARPS - 1);
                const int j1 = sm.atomJ[m], nJ = sm.atomJ[m + 1] - j1, n = nI * nJ;
                float kacc[FC_MAXSIG];
#pragma unroll
                for (int s = 0; s < FC_MAXSIG; ++s) kacc[s] = 0.0f;
                const float inv = 1.0f / (float)nJ;
                for (int t = part * 32 + lane; t < n; t += FC_WARPS * 32) {
                    const int a = (int)(((float)t + 0.5f) * inv), j = j1 + t - a * nJ;
                    const float stz = sm.stoch[sm.aclsI[a] * FC_SST + sm.aclsJ[j]];
                    float l2 = sm.selfI[a] + sm.selfJ[j] -
                               2.0f * band_value(A, j * A.ld + a) * stz;
                    if (fabsf(l2) < eps) l2 = 0.0f;  // farad_kernels.f90:594
#pragma unroll
                    for (int s = 0; s < FC_MAXSIG; ++s) {
                        if (s < nsig) {
                            float e;
                            asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(e) : "f"(l2 * sm.sc[s]));
                            kacc[s] += e;
                        }
                    }
                }
#pragma unroll
                for (int s = 0; s < FC_MAXSIG; ++s) {
                    if (s < nsig) {
                        float v = kacc[s];
                        if (part * 32 < n)
                            for (int o = 16; o; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
                        if (lane == 0) sm.red[m][part][s] = v;
                    }
                }
            }
            __syncthreads();
            for (int t = threadIdx.x; t < (count - first) * nsig; t += blockDim.x) {
                const int m = first + t / nsig, s = t % nsig, J = J0 + j0 + m;
                double v = 0.0;
                for (int q = 0; q < FC_WARPS; ++q) v += (double)sm.red[m][q][s];
                K[((size_t)s * nm1 + I) * nm2 + J] = v;
                if (symmetric) K[((size_t)s * nm1 + J) * nm2 + I] = v;
            }
        }
    }
}

// Self terms S(a, a) through the pair kernel's passes and sums, so that
// l2 = s + s - 2 S cancels exactly for an atom with itself.
__global__ void __launch_bounds__(FC_WARPS * 32, 4)
arad_fast_self_kernel(SetWs w, const int *__restrict__ N, int nm, int amax, AradParams P,
                      const ClassInfo *ci) {
    extern __shared__ __align__(16) unsigned char fc_smem_raw[];
    if (ci->flag) return;
    const int I = blockIdx.x;
    if (I >= nm) return;
    const float maxg2s = (float)(P.maxg2 * fp32_scale(P) * fp32_scale(P));
    if (ci->ncls <= FC_PC) {
        BandSmem &sm = *reinterpret_cast<BandSmem *>(fc_smem_raw);
        band_load_tables(sm, ci);
        band_sizes(sm, w, N, I, I + 1, w, N, I, I + 1, amax);
        __syncthreads();
        const int n = sm.nI[0], recs = (sm.recI[0] + BD_REC - 1) / BD_REC * BD_REC;
        const BandArena A = band_carve(fc_smem_raw + (sizeof(BandSmem) + 15) / 16 * 16, recs,
                                       sm.pairsJ[0], n, n | 1);
        band_load_J(sm, A, w, I, 0, 1, amax, false);
        __syncthreads();
        band_load_I(sm, A, w, I, 0, 1, amax, sqrtf(maxg2s) * 1.0001f, false);
        __syncthreads();
        band_sums(sm, A, 0, 0, n, maxg2s);
        __syncthreads();
        for (int a = threadIdx.x; a < n; a += blockDim.x)
            w.selff[(size_t)I * amax + a] = band_value(A, a * A.ld + a);
        return;
    }
    FastSmem &sm = *reinterpret_cast<FastSmem *>(fc_smem_raw);
    load_stoch(sm.stoch, ci);
    const int nI = min(max(N[I], 0), amax);
    fast_load_I(sm, w, I, amax, nI, false);
    fast_load_J(sm, w, I, amax, nI, false);
    __syncthreads();
    fast_pair_sums(sm, nI, maxg2s);
    for (int a = threadIdx.x; a < nI; a += blockDim.x)
        w.selff[(size_t)I * amax + a] = sm.S[a * FC_SS + a];
}

__global__ void __launch_bounds__(FC_WARPS * 32, 4)
arad_fast_pair_kernel(SetWs w1, const int *__restrict__ N1, int nm1, SetWs w2,
                      const int *__restrict__ N2, int nm2, int amax, AradParams P,
                      const ClassInfo *ci, SigmaTable sig, int nsig, int symmetric,
                      double *__restrict__ K) {
    extern __shared__ __align__(16) unsigned char fc_smem_raw[];
    if (ci->flag) return;
    const int nbj = (nm2 + FC_BM - 1) / FC_BM;
    int bi, bj;
    pair_block(blockIdx.x, symmetric, nbj, bi, bj);
    const float maxg2s = (float)(P.maxg2 * fp32_scale(P) * fp32_scale(P));
    const float eps = 5.0e-12f;
    if (ci->ncls <= FC_PC) {
        band_tile(fc_smem_raw, w1, N1, nm1, w2, N2, nm2, bi * FC_BM, bj * FC_BM, amax, maxg2s, eps,
                  ci, sig, nsig, symmetric, K);
        return;
    }
    FastSmem &sm = *reinterpret_cast<FastSmem *>(fc_smem_raw);
    load_stoch(sm.stoch, ci);
    float sc[FC_MAXSIG];
#pragma unroll
    for (int s = 0; s < FC_MAXSIG; ++s)
        sc[s] = s < nsig ? (float)(sig.inv_sigma2[s] * 1.4426950408889634) : 0.0f;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    for (int il = 0; il < FC_BM; ++il) {
        const int I = bi * FC_BM + il;
        if (I >= nm1) break;
        __syncthreads();
        const int nI = min(max(N1[I], 0), amax);
        fast_load_I(sm, w1, I, amax, nI, true);
        for (int jl = 0; jl < FC_BM; ++jl) {
            const int J = bj * FC_BM + jl;
            if (J >= nm2) break;
            if (symmetric && J < I) continue;
            __syncthreads();
            const int nJ = min(max(N2[J], 0), amax);
            fast_load_J(sm, w2, J, amax, nJ, true);
            __syncthreads();
            fast_pair_sums(sm, nJ, maxg2s);
            // phase 2: l2 and the kernel exponentials of every atom pair
            float kacc[FC_MAXSIG];
#pragma unroll
            for (int s = 0; s < FC_MAXSIG; ++s) kacc[s] = 0.0f;
            for (int t = threadIdx.x; t < nI * nJ; t += blockDim.x) {
                const int a = t / nJ, j1 = t - a * nJ;
                const float stz = sm.stoch[sm.aclsI[a] * FC_SST + sm.aclsJ[j1]];
                float l2 = sm.selfI[a] + sm.selfJ[j1] -
                           2.0f * sm.S[a * FC_SS + j1] * stz;
                if (fabsf(l2) < eps) l2 = 0.0f;  // farad_kernels.f90:594
#pragma unroll
                for (int s = 0; s < FC_MAXSIG; ++s) {
                    if (s < nsig) {
                        float e;
                        asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(e) : "f"(l2 * sc[s]));
                        kacc[s] += e;
                    }
                }
            }
#pragma unroll
            for (int s = 0; s < FC_MAXSIG; ++s) {
                float v = kacc[s];
                for (int o = 16; o; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
                if (lane == 0) sm.red[warp][s] = v;
            }
            __syncthreads();
            if (threadIdx.x < nsig) {
                const int s = threadIdx.x;
                double v = 0.0;
                for (int q = 0; q < FC_WARPS; ++q) v += (double)sm.red[q][s];
                K[((size_t)s * nm1 + I) * nm2 + J] = v;
                if (symmetric) K[((size_t)s * nm1 + J) * nm2 + I] = v;
            }
        }
    }
}

// ---- fast FP64 path ---------------------------------------------------------
// atomic_distl2 in FP64 for descriptors of at most FC_MAXA atoms and FC_MAXC
// element classes, bit for bit what the generic kernel gives: one thread sums
// an atom pair's terms in the reference's order with the reference's
// operations. At sigma 0.1 the exponent carries l2 / sigma^2 = 100 l2, and sums
// in any other order leave the 1e-12 agreement with the reference.
//
// A CTA takes one molecule I and a few molecules J, as many at a time as its
// shared memory holds:
//   1. the run of neighbours m2 of j1 inside the (8 w)^2 window of every
//      record (i1, m1), walking both ascending lists together (a list that
//      does not ascend keeps its whole length, and its terms are tested);
//   2. the atom pairs ordered by their number of terms, so that the 32 pairs
//      of a warp have nearly the same number (59 % of the lanes work with loops
//      over m1 and m2 in lockstep), and by atom j1 among equals, so that its
//      lanes read the same few records;
//   3. warps take 32 pairs at a time, longest first; a thread walks the runs of
//      its pair as one flat loop;
//   4. the kernel exponentials of every l2 and sigma, a warp per molecule J and
//      sigma, in a fixed order.
// 28 FP64 instructions per term, 16 of them the exponential. The stoichiometric
// factor comes from the class table, formed by the same operations (two FP64
// divisions per term before), and the operands from shared memory (per-lane
// gathers from global memory before), whose pipe is now as busy as the issue
// slots. One J at a time and 256 threads left half of the warps waiting for the
// one with the longest pairs.
constexpr int F6_TPB = 512;
constexpr int F6_ROWS = 65535;  // molecules I of a launch (the grid's limit in y)
constexpr int F6_AP = 1024;    // atom pairs at a time (a pair of the largest molecules)
constexpr int F6_WIN = 12288;  // runs at a time (24 KB): the atoms j1 go in chunks above that
constexpr int F6_JA = 128, F6_JM = 16;  // atoms and molecules J at a time
constexpr int F6_BUCKETS = 32, F6_CHUNKS = F6_AP / 32;
constexpr int F6_SST = FC_MAXC + 1;
static_assert(FC_MAXA * FC_MAXA <= F6_AP && FC_MAXA <= F6_JA, "one pair of molecules fits");
static_assert(F6_JM <= F6_TPB / 32 && F6_JM < 32, "a warp per molecule J, a lane each");

struct F64Side {
    double2 *A, *B;    // records by atom: (r, sine factor), (cos, sin)
    double *self;
    int *off, *end;    // records of the atoms
    int *acls, *asc;
    unsigned char *C;  // class of each record
};
struct F64View {
    F64Side i, j;
    double *l2;           // l2 of every atom pair
    double *st;           // stoichiometric table, row stride F6_SST
    int *tot;             // terms of every atom pair
    int *rank;            // F6_BUCKETS x F6_CHUNKS
    int *jatom, *jrec;    // first atom and record of each molecule J, and the ends
    int *ctl;             // molecules J, largest atom count, next 32 pairs
    unsigned short *win;  // F6_WIN: [m1][atom pair] first neighbour | length << 8
    unsigned short *perm; // atom pairs by number of terms
};

__host__ __device__ inline int f64_pad(int n) { return (n + 7) & ~7; }
// records of the molecules J at a time: about four of average size
__host__ __device__ inline int f64_pool(int amax) {
    return f64_pad(amax * amax) > 1072 ? f64_pad(amax * amax) : 1072;
}
inline size_t f64_smem_bytes(int amax) {
    const size_t R = (size_t)f64_pad(amax * amax), RJ = (size_t)f64_pool(amax);
    return (R + RJ) * 2 * sizeof(double2) +
           (F6_AP + FC_MAXC * F6_SST + FC_MAXA + F6_JA) * sizeof(double) +
           (F6_AP + F6_BUCKETS * F6_CHUNKS + 2 * (F6_JM + 2) + 4 + 4 * (FC_MAXA + F6_JA)) *
               sizeof(int) +
           (F6_WIN + F6_AP) * sizeof(unsigned short) + R + RJ;
}
// the self kernel: one side and the table
inline size_t f64_self_smem_bytes(int amax) {
    const size_t R = (size_t)f64_pad(amax * amax);
    return R * 2 * sizeof(double2) + (FC_MAXC * F6_SST + FC_MAXA) * sizeof(double) +
           4 * FC_MAXA * sizeof(int) + R;
}

__device__ __forceinline__ int *f64_atoms(F64Side &s, int *q, int atoms) {
    s.off = q;
    s.end = q + atoms;
    s.acls = q + 2 * atoms;
    s.asc = q + 3 * atoms;
    return q + 4 * atoms;
}

__device__ __forceinline__ F64View f64_view(unsigned char *p, int amax) {
    const int R = f64_pad(amax * amax), RJ = f64_pool(amax);
    F64View v;
    v.i.A = reinterpret_cast<double2 *>(p);
    v.i.B = v.i.A + R;
    v.j.A = v.i.B + R;
    v.j.B = v.j.A + RJ;
    v.l2 = reinterpret_cast<double *>(v.j.B + RJ);
    v.st = v.l2 + F6_AP;
    v.i.self = v.st + FC_MAXC * F6_SST;
    v.j.self = v.i.self + FC_MAXA;
    v.tot = reinterpret_cast<int *>(v.j.self + F6_JA);
    v.rank = v.tot + F6_AP;
    v.jatom = v.rank + F6_BUCKETS * F6_CHUNKS;
    v.jrec = v.jatom + F6_JM + 2;
    v.ctl = v.jrec + F6_JM + 2;
    int *q = f64_atoms(v.i, v.ctl + 4, FC_MAXA);
    q = f64_atoms(v.j, q, F6_JA);
    v.win = reinterpret_cast<unsigned short *>(q);
    v.perm = v.win + F6_WIN;
    v.i.C = reinterpret_cast<unsigned char *>(v.perm + F6_AP);
    v.j.C = v.i.C + R;
    return v;
}

// One warp: the record ranges of molecule m's n atoms, from entry `atom` of the
// side's lists and record `rec` on.
__device__ __forceinline__ void f64_offsets(const F64Side &s, const SetWs &w, int m, int amax, int n,
                                            int atom, int rec) {
    const int a = threadIdx.x & 31;
    const int cnt = a < n ? w.nnb[(size_t)m * amax + a] : 0;
    int incl = cnt;
    for (int d = 1; d < 32; d <<= 1) {
        const int o = __shfl_up_sync(0xffffffffu, incl, d);
        if (a >= d) incl += o;
    }
    if (a < n) {
        s.off[atom + a] = rec + incl - cnt;
        s.end[atom + a] = rec + incl;
    }
}

// Whole CTA (of any size): molecule m's records and atoms, its ranges being set.
__device__ __forceinline__ void f64_load(const F64Side &s, const double *__restrict__ X,
                                         const SetWs &w, int m, int amax, int n, int atom,
                                         bool use_self) {
    const size_t mol = (size_t)m * amax;
    for (int t = threadIdx.x; t < n * amax; t += blockDim.x) {
        const int a = t / amax, k = t - a * amax;
        const int at = s.off[atom + a] + k;
        if (at < s.end[atom + a]) {
            const double *x = X + (mol + a) * 5 * amax + k;
            s.A[at] = make_double2(x[0], w.xi[(mol + a) * amax + k]);
            s.B[at] = make_double2(x[3 * amax], x[4 * amax]);
            s.C[at] = (unsigned char)w.cls[(mol + a) * amax + k];
        }
    }
    for (int a = threadIdx.x; a < n; a += blockDim.x) {
        s.self[atom + a] = use_self ? w.self[mol + a] : 0.0;
        s.acls[atom + a] = w.acls[mol + a];
        s.asc[atom + a] = w.asc[mol + a];
    }
}

__device__ __forceinline__ void f64_load_table(double *st, const ClassInfo *ci) {
    for (int t = threadIdx.x; t < FC_MAXC * FC_MAXC; t += blockDim.x)
        st[(t / FC_MAXC) * F6_SST + t % FC_MAXC] = ci->stoch64[t];
}

// One term of atomic_distl2 (the operations and order of distl2_f64).
__device__ __forceinline__ double f64_term(double t, double inv_width, const double2 &A1,
                                           const double2 &B1, const double2 &A2, const double2 &B2,
                                           double st) {
    double d = __dmul_rn(__dmul_rn(exp_window(__dmul_rn(t, inv_width)), A1.y), A2.y);
    d = __dmul_rn(d, st);
    const double ang = __dadd_rn(__dadd_rn(1.0, __dmul_rn(B1.x, B2.x)), __dmul_rn(B1.y, B2.y));
    return __dmul_rn(d, ang);
}

// Self terms, one warp per molecule, one lane per atom.
__global__ void __launch_bounds__(32)
arad_f64_self_kernel(const double *__restrict__ X, SetWs w, const int *__restrict__ N, int nm,
                     int amax, AradParams P, const ClassInfo *ci) {
    extern __shared__ __align__(16) unsigned char fc_smem_raw[];
    if (ci->flag) return;
    const int m = blockIdx.x;
    if (m >= nm) return;
    const int R = f64_pad(amax * amax);
    F64Side s;
    s.A = reinterpret_cast<double2 *>(fc_smem_raw);
    s.B = s.A + R;
    double *st = reinterpret_cast<double *>(s.B + R);
    s.self = st + FC_MAXC * F6_SST;
    s.C = reinterpret_cast<unsigned char *>(
        f64_atoms(s, reinterpret_cast<int *>(s.self + FC_MAXA), FC_MAXA));
    const int n = min(max(N[m], 0), amax), a = threadIdx.x;
    f64_load_table(st, ci);
    f64_offsets(s, w, m, amax, n, 0, 0);
    __syncthreads();
    f64_load(s, X, w, m, amax, n, 0, false);
    __syncthreads();
    if (a >= n) return;
    double sum = 0.0;
    for (int k1 = s.off[a]; k1 < s.end[a]; ++k1) {
        const double2 A1 = s.A[k1], B1 = s.B[k1];
        const double *strow = st + s.C[k1] * F6_SST;
        for (int k2 = s.off[a]; k2 < s.end[a]; ++k2) {
            const double2 A2 = s.A[k2];
            const double dr = __dsub_rn(A2.x, A1.x);
            const double t = __dmul_rn(dr, dr);
            if (t < P.maxg2)
                sum = __dadd_rn(sum, f64_term(t, P.inv_width, A1, B1, A2, s.B[k2], strow[s.C[k2]]));
        }
    }
    w.self[(size_t)m * amax + a] = sum;
}

// Sum of atom pair ap = (i1, j1) of a chunk of nap over its runs, in (m1, m2)
// order. kTest: some list of J does not ascend, so terms outside the window
// occur in the runs.
template <bool kTest>
__device__ __forceinline__ double f64_pair_sum(const F64View &v, int i1, int j1, int ap, int nap,
                                               const AradParams &P) {
    const unsigned short *win = v.win + ap;
    double sum = 0.0;
    int k1 = v.i.off[i1] - 1, k2 = 0, rem = 0;
    const int jbeg = v.j.off[j1];
    double2 A1 = make_double2(0.0, 0.0), B1 = A1;
    const double *strow = v.st;
    for (int left = v.tot[ap]; left > 0; --left) {
        while (rem == 0) {  // the next run that holds a term
            const int w = *win;
            win += nap;
            ++k1;
            rem = w >> 8;
            k2 = jbeg + (w & 0xff);
            A1 = v.i.A[k1];
            B1 = v.i.B[k1];
            strow = v.st + v.i.C[k1] * F6_SST;
        }
        const double2 A2 = v.j.A[k2];
        const double dr = __dsub_rn(A2.x, A1.x);
        const double t = __dmul_rn(dr, dr);
        if (!kTest || t < P.maxg2)
            sum = __dadd_rn(sum, f64_term(t, P.inv_width, A1, B1, A2, v.j.B[k2],
                                          strow[v.j.C[k2]]));
        ++k2;
        --rem;
    }
    return sum;
}

// Molecule I = I0 + blockIdx.y against the bj molecules J of block blockIdx.x.
__global__ void __launch_bounds__(F6_TPB, 2)
arad_f64_pair_kernel(const double *__restrict__ X1, SetWs w1, const int *__restrict__ N1, int nm1,
                     const double *__restrict__ X2, SetWs w2, const int *__restrict__ N2, int nm2,
                     int amax, AradParams P, const ClassInfo *ci,
                     const __grid_constant__ SigmaTable sig, int nsig, int symmetric, int bj,
                     int I0, double *__restrict__ K) {
    extern __shared__ __align__(16) unsigned char fc_smem_raw[];
    if (ci->flag) return;
    const int I = I0 + (int)blockIdx.y, jb = (int)blockIdx.x;
    const int jend = min(nm2 - jb * bj, bj) + jb * bj;
    if (symmetric && jend <= I) return;  // below the diagonal
    const F64View v = f64_view(fc_smem_raw, amax);
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int nI = min(max(N1[I], 0), amax);
    f64_load_table(v.st, ci);
    if (warp == 1) f64_offsets(v.i, w1, I, amax, nI, 0, 0);
    __syncthreads();
    f64_load(v.i, X1, w1, I, amax, nI, 0, true);
    int J0 = symmetric ? max(jb * bj, I) : jb * bj;
    while (J0 < jend) {
        // as many molecules J as fit (the first always does); a lane each
        if (warp == 0) {
            const bool in = lane < F6_JM && J0 + lane < jend;
            const int n = in ? min(max(N2[J0 + lane], 0), amax) : 0;
            int atoms = n, recs = n * n;
            for (int d = 1; d < 32; d <<= 1) {
                const int oa = __shfl_up_sync(0xffffffffu, atoms, d);
                const int orc = __shfl_up_sync(0xffffffffu, recs, d);
                if (lane >= d) {
                    atoms += oa;
                    recs += orc;
                }
            }
            const bool fits = in && atoms * nI <= F6_AP && atoms <= F6_JA && recs <= f64_pool(amax);
            const int nj = __ffs(~__ballot_sync(0xffffffffu, fits || lane == 0)) - 1;
            int big = lane < nj ? n : 0;
            for (int d = 16; d; d >>= 1) big = max(big, __shfl_xor_sync(0xffffffffu, big, d));
            if (lane <= nj) {
                v.jatom[lane] = atoms - n;
                v.jrec[lane] = recs - n * n;
            }
            if (lane == 0) {
                v.ctl[0] = nj;
                v.ctl[1] = big;
            }
        }
        __syncthreads();
        const int nj = v.ctl[0], big = v.ctl[1], natom = v.jatom[nj];
        if (warp < nj)
            f64_offsets(v.j, w2, J0 + warp, amax, v.jatom[warp + 1] - v.jatom[warp],
                        v.jatom[warp], v.jrec[warp]);
        __syncthreads();
        for (int b = 0; b < nj; ++b)
            f64_load(v.j, X2, w2, J0 + b, amax, v.jatom[b + 1] - v.jatom[b], v.jatom[b], true);
        const int jstep = nI > 0 ? F6_WIN / (nI * nI) : F6_JA;
        for (int j0 = 0; j0 < natom; j0 += jstep) {
            const int jn = min(jstep, natom - j0), nap = nI * jn;
            for (int t = tid; t < F6_BUCKETS * F6_CHUNKS; t += F6_TPB) v.rank[t] = 0;
            if (tid == 0) v.ctl[2] = 0;
            __syncthreads();
            // 1. the runs; atom pair ap = (j1 - j0) nI + i1, a thread each. Both
            // ends of the window only move up while r1 ascends.
            for (int ap = tid; ap < nap; ap += F6_TPB) {
                const int jq = ap / nI, i1 = ap - jq * nI, j1 = j0 + jq;
                const double2 *J2 = v.j.A + v.j.off[j1];
                const int cnt = v.j.end[j1] - v.j.off[j1], k1 = v.i.off[i1];
                const bool ascends = v.j.asc[j1] != 0;
                int lo = 0, hi = ascends ? 0 : cnt, total = 0;
                double before = 0.0;
                for (int m1 = 0; m1 < v.i.end[i1] - k1; ++m1) {
                    const double r1 = v.i.A[k1 + m1].x;
                    if (ascends) {
                        if (!(r1 >= before)) lo = hi = 0;
                        before = r1;
                        while (lo < cnt) {  // to the first neighbour not below the window
                            const double dr = __dsub_rn(J2[lo].x, r1);
                            if (!(dr < 0.0) || __dmul_rn(dr, dr) < P.maxg2) break;
                            ++lo;
                        }
                        hi = max(hi, lo);
                        while (hi < cnt) {  // to the first neighbour above it
                            const double dr = __dsub_rn(J2[hi].x, r1);
                            if (!(dr < 0.0) && !(__dmul_rn(dr, dr) < P.maxg2)) break;
                            ++hi;
                        }
                    }
                    v.win[m1 * nap + ap] = (unsigned short)(lo | ((hi - lo) << 8));
                    total += hi - lo;
                }
                v.tot[ap] = total;
            }
            const bool test = __syncthreads_or(tid < jn && !v.j.asc[j0 + tid]);
            // 2. the order: per 32 pairs the count of each bucket (most terms
            // first), an exclusive prefix over buckets and 32s, then the places
            int bucket[F6_AP / F6_TPB], place[F6_AP / F6_TPB];
#pragma unroll
            for (int q = 0; q < F6_AP / F6_TPB; ++q) {
                const int ap = tid + q * F6_TPB;
                const bool in = ap < nap;
                bucket[q] = in ? F6_BUCKETS - 1 -
                                     min(F6_BUCKETS - 1, v.tot[ap] * F6_BUCKETS / (nI * big))
                               : F6_BUCKETS;
                const unsigned same = __match_any_sync(0xffffffffu, bucket[q]);
                place[q] = __popc(same & ((1u << lane) - 1));
                if (in && place[q] == 0) v.rank[bucket[q] * F6_CHUNKS + (ap >> 5)] = __popc(same);
            }
            __syncthreads();
            static_assert(F6_BUCKETS * F6_CHUNKS == 2 * F6_TPB, "two entries per thread");
            {
                const int c0 = v.rank[2 * tid], c1 = v.rank[2 * tid + 1];
                int incl = c0 + c1;
                for (int d = 1; d < 32; d <<= 1) {
                    const int o = __shfl_up_sync(0xffffffffu, incl, d);
                    if (lane >= d) incl += o;
                }
                __shared__ int part[F6_TPB / 32];
                if (lane == 31) part[warp] = incl;
                __syncthreads();
                int before = 0;
                for (int q = 0; q < warp; ++q) before += part[q];
                v.rank[2 * tid] = before + incl - c0 - c1;
                v.rank[2 * tid + 1] = before + incl - c1;
            }
            __syncthreads();
#pragma unroll
            for (int q = 0; q < F6_AP / F6_TPB; ++q) {
                const int ap = tid + q * F6_TPB;
                if (ap < nap)
                    v.perm[v.rank[bucket[q] * F6_CHUNKS + (ap >> 5)] + place[q]] =
                        (unsigned short)ap;
            }
            __syncthreads();
            // 3. the sums and l2 (which warp takes a pair does not change its sum)
            for (;;) {
                int t = lane == 0 ? atomicAdd(&v.ctl[2], 32) : 0;
                t = __shfl_sync(0xffffffffu, t, 0) + lane;
                if (t - lane >= nap) break;
                if (t < nap) {
                    const int ap = v.perm[t], jq = ap / nI, i1 = ap - jq * nI, j1 = j0 + jq;
                    const double S = test ? f64_pair_sum<true>(v, i1, j1, ap, nap, P)
                                          : f64_pair_sum<false>(v, i1, j1, ap, nap, P);
                    const double stz = v.st[v.i.acls[i1] * F6_SST + v.j.acls[j1]];
                    double l2 = __dsub_rn(__dadd_rn(v.i.self[i1], v.j.self[j1]),
                                          __dmul_rn(__dmul_rn(2.0, S), stz));
                    if (fabs(l2) < P.eps) l2 = 0.0;  // farad_kernels.f90:594
                    v.l2[j0 * nI + ap] = l2;
                }
                __syncwarp();
            }
            __syncthreads();
        }
        // 4. the kernel exponentials, a warp per molecule J and sigma
        for (int q = warp; q < nj * nsig; q += F6_TPB / 32) {
            const int b = q / nsig, s = q - b * nsig, J = J0 + b;
            const int beg = v.jatom[b] * nI, end = v.jatom[b + 1] * nI;
            double e = 0.0;
            for (int t = beg + lane; t < end; t += 32) e += exp(v.l2[t] * sig.inv_sigma2[s]);
            for (int o = 16; o; o >>= 1) e += __shfl_xor_sync(0xffffffffu, e, o);
            if (lane == 0) {
                K[((size_t)s * nm1 + I) * nm2 + J] = e;
                if (symmetric) K[((size_t)s * nm1 + J) * nm2 + I] = e;
            }
        }
        __syncthreads();  // the next molecules overwrite these
        J0 += nj;
    }
}

// Molecules J of a CTA: four, about what its shared memory holds at a time, once
// such blocks fill the GPU several times over.
inline int f64_block(long long npairs) { return npairs >= (1LL << 13) ? 4 : 1; }

// Small molecules keep the fast kernel's CTA waiting for itself: it orders and prepares a
// few dozen terms, and a warp per molecule pair does them in less. The fewer the pairs,
// the smaller the molecules for which that holds: a lone warp takes longer for its pair
// than a CTA. Both give the same bits. us of a warp per pair and of the fast kernel,
// symmetric: 5 atoms, 30 molecules 35, 53, 1000 2487, 5529; 6 atoms, 30 58, 59, 200 205,
// 301; 7 atoms, 30 74, 68, 200 292, 345; 8 atoms, 200 365, 388; 9 atoms, 200 526, 432, 1000
// 8246, 9043.
bool f64_generic(int amax, long long npairs) {
    return amax <= 5 || (amax <= 9 && npairs >= 1LL << (3 * amax - 10));
}

// The fast kernels' shared memory is dynamic (above the 48 KB static limit);
// the attribute is set once per device.
int fast_smem_attrs() {
    static int attr_dev = -1;
    int dev = 0;
    FMLB_TRY(cuda_status(cudaGetDevice(&dev), "fmlb_arad_kernels: cudaGetDevice"));
    if (attr_dev == dev) return FMLB_OK;
    FMLB_TRY(cuda_status(cudaFuncSetAttribute(arad_fast_self_kernel,
                                              cudaFuncAttributeMaxDynamicSharedMemorySize,
                                              (int)kFastSmem),
                         "fmlb_arad_kernels: self kernel smem attribute"));
    FMLB_TRY(cuda_status(cudaFuncSetAttribute(arad_fast_pair_kernel,
                                              cudaFuncAttributeMaxDynamicSharedMemorySize,
                                              (int)kFastSmem),
                         "fmlb_arad_kernels: pair kernel smem attribute"));
    FMLB_TRY(cuda_status(cudaFuncSetAttribute(arad_f64_self_kernel,
                                              cudaFuncAttributeMaxDynamicSharedMemorySize,
                                              (int)f64_self_smem_bytes(FC_MAXA)),
                         "fmlb_arad_kernels: FP64 self kernel smem attribute"));
    FMLB_TRY(cuda_status(cudaFuncSetAttribute(arad_f64_pair_kernel,
                                              cudaFuncAttributeMaxDynamicSharedMemorySize,
                                              (int)f64_smem_bytes(FC_MAXA)),
                         "fmlb_arad_kernels: FP64 pair kernel smem attribute"));
    attr_dev = dev;
    return FMLB_OK;
}

// ---- atom-level ARAD kernel (fget_atomic_kernels_arad, farad_kernels.f90:757-899)
// Every atom is its own environment: descriptor (5, amax), neighbour count n.
// Per atom: the prefix length of the neighbour list (the exit at r > cut of
// atomic_distl2, :68 / :72), the sine factors 1 - sin(r inv_cut) for every
// listed neighbour (:836-850, unconditional) and the self term (:855-868).
__global__ void arad_atom_prep_kernel(const double *__restrict__ Q, const int *__restrict__ N,
                                      int na, int amax, AradParams P, int *__restrict__ nnb,
                                      double *__restrict__ sines, double *__restrict__ self) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= na) return;
    const double *q = Q + (size_t)i * 5 * amax;
    const int n = min(max(N[i], 0), amax);
    double *si = sines + (size_t)i * amax;
    int pre = 0;
    while (pre < n && !(q[pre] > P.cut)) ++pre;
    for (int m = 0; m < amax; ++m) si[m] = m < n ? 1.0 - sin(__dmul_rn(q[m], P.inv_cut)) : 0.0;
    nnb[i] = pre;
    self[i] = distl2_f64(q, si, pre, q, si, pre, amax, P);
}

// K[s, i, j] = exp(l2(i, j) inv_sigma2[s]), l2 = self_i + self_j - 2 d(i, j) stoch
// (:873-891); thread per atom pair, j fastest (coalesced rows of K). With
// kDistance the l2 itself is stored, K[i, j] = l2(i, j) (the distances of
// fget_atomic_distance_arad, :902-1030).
template <bool kDistance>
__global__ void __launch_bounds__(128, 7)
arad_atom_pair_kernel(const double *__restrict__ Q1, const double *__restrict__ Z1,
                      const int *__restrict__ nnb1, const double *__restrict__ S1,
                      const double *__restrict__ self1, int na1,
                      const double *__restrict__ Q2, const double *__restrict__ Z2,
                      const int *__restrict__ nnb2, const double *__restrict__ S2,
                      const double *__restrict__ self2, int na2, int amax, AradParams P,
                      SigmaTable sig, int nsig, double *__restrict__ K) {
    const int j = blockIdx.x * blockDim.x + threadIdx.x;
    const double eps = (double)5.0e-12f;  // :823, a single-precision literal in the source
    for (int i = blockIdx.y; i < na1; i += gridDim.y) {
        if (j >= na2) continue;
        double l2 = distl2_f64(Q1 + (size_t)i * 5 * amax, S1 + (size_t)i * amax, nnb1[i],
                               Q2 + (size_t)j * 5 * amax, S2 + (size_t)j * amax, nnb2[j], amax,
                               P);
        const double dz1 = __dsub_rn(Z1[2 * i], Z2[2 * j]);
        const double dz2 = __dsub_rn(Z1[2 * i + 1], Z2[2 * j + 1]);
        const double st = __ddiv_rn(
            __dmul_rn(__ddiv_rn(P.rw2, __dadd_rn(P.rw2, __dmul_rn(dz1, dz1))), P.cw2),
            __dadd_rn(P.cw2, __dmul_rn(dz2, dz2)));
        l2 = __dsub_rn(__dadd_rn(self1[i], self2[j]), __dmul_rn(__dmul_rn(2.0, l2), st));
        if (fabs(l2) < eps) l2 = 0.0;
        if (kDistance) {
            K[(size_t)i * na2 + j] = l2;
        } else {
            for (int s = 0; s < nsig; ++s)
                K[((size_t)s * na1 + i) * na2 + j] = exp(__dmul_rn(l2, sig.inv_sigma2[s]));
        }
    }
}

size_t atom_ws_bytes(int na, int amax) {
    return align256((size_t)na * sizeof(int)) + align256((size_t)na * amax * sizeof(double)) +
           align256((size_t)na * sizeof(double));
}

}  // namespace
}  // namespace fmlb

extern "C" size_t fmlb_arad_atomic_workspace_bytes(int na1, int na2, int amax) {
    if (na1 < 0 || na2 < 0 || amax < 1) return 0;
    return fmlb::atom_ws_bytes(na1, amax) + fmlb::atom_ws_bytes(na2, amax);
}

static int arad_atomic_impl(const double *Q1, const double *Z1, const int *N1, int na1,
                            const double *Q2, const double *Z2, const int *N2, int na2, int amax,
                            const double *sigmas_host, int nsigma, double width,
                            double cut_distance, double r_width, double c_width, double *K,
                            void *workspace, size_t ws_bytes, bool distance, cudaStream_t st) {
    using namespace fmlb;
    const char *what = distance ? "fmlb_arad_atomic_distances" : "fmlb_arad_atomic_kernels";
    FMLB_REQUIRE(na1 >= 0 && na2 >= 0 && amax >= 1, "%s: bad sizes", what);
    if (!distance)
        FMLB_REQUIRE(nsigma >= 1 && nsigma <= MAXSIG && sigmas_host,
                     "%s: nsigma must be 1..%d", what, MAXSIG);
    const size_t need = fmlb_arad_atomic_workspace_bytes(na1, na2, amax);
    if (ws_bytes < need || (need && !workspace)) {
        set_error("%s: workspace %zu bytes < required %zu", what, ws_bytes, need);
        return FMLB_ENOMEM;
    }
    if (na1 == 0 || na2 == 0) return FMLB_OK;
    FMLB_REQUIRE(Q1 && Z1 && N1 && Q2 && Z2 && N2 && K, "%s: null pointer", what);
    AradParams P;
    P.width = width;
    P.cut = cut_distance;
    P.rw2 = r_width * r_width;
    P.cw2 = c_width * c_width;
    P.inv_width = -1.0 / (4.0 * width * width);      // :58
    P.maxg2 = (8.0 * width) * (8.0 * width);          // :60
    P.inv_cut = (4.0 * atan(1.0)) / (2.0 * cut_distance);  // :828
    P.eps = (double)5.0e-12f;                                // :823
    SigmaTable sig;
    for (int s = 0; s < (distance ? 0 : nsigma); ++s)
        sig.inv_sigma2[s] = -1.0 / (sigmas_host[s] * sigmas_host[s]);
    char *p = static_cast<char *>(workspace);
    int *nnb1 = reinterpret_cast<int *>(p); p += align256((size_t)na1 * sizeof(int));
    double *S1 = reinterpret_cast<double *>(p); p += align256((size_t)na1 * amax * sizeof(double));
    double *self1 = reinterpret_cast<double *>(p); p += align256((size_t)na1 * sizeof(double));
    int *nnb2 = reinterpret_cast<int *>(p); p += align256((size_t)na2 * sizeof(int));
    double *S2 = reinterpret_cast<double *>(p); p += align256((size_t)na2 * amax * sizeof(double));
    double *self2 = reinterpret_cast<double *>(p);
    arad_atom_prep_kernel<<<ceil_div(na1, 128), 128, 0, st>>>(Q1, N1, na1, amax, P, nnb1, S1,
                                                               self1);
    FMLB_TRY(launch_status("arad_atom_prep_kernel"));
    arad_atom_prep_kernel<<<ceil_div(na2, 128), 128, 0, st>>>(Q2, N2, na2, amax, P, nnb2, S2,
                                                               self2);
    FMLB_TRY(launch_status("arad_atom_prep_kernel"));
    const dim3 grid(ceil_div(na2, 128), std::min(na1, 65535));
    if (distance)
        arad_atom_pair_kernel<true><<<grid, 128, 0, st>>>(Q1, Z1, nnb1, S1, self1, na1, Q2, Z2,
                                                          nnb2, S2, self2, na2, amax, P, sig, 0,
                                                          K);
    else
        arad_atom_pair_kernel<false><<<grid, 128, 0, st>>>(Q1, Z1, nnb1, S1, self1, na1, Q2, Z2,
                                                           nnb2, S2, self2, na2, amax, P, sig,
                                                           nsigma, K);
    return launch_status("arad_atom_pair_kernel");
}

extern "C" int fmlb_arad_atomic_kernels(const double *Q1, const double *Z1, const int *N1, int na1,
                                        const double *Q2, const double *Z2, const int *N2, int na2,
                                        int amax, const double *sigmas_host, int nsigma,
                                        double width, double cut_distance, double r_width,
                                        double c_width, double *K, void *workspace,
                                        size_t ws_bytes, void *stream) {
    return arad_atomic_impl(Q1, Z1, N1, na1, Q2, Z2, N2, na2, amax, sigmas_host, nsigma, width,
                            cut_distance, r_width, c_width, K, workspace, ws_bytes, false,
                            FMLB_STREAM(stream));
}

extern "C" int fmlb_arad_atomic_distances(const double *Q1, const double *Z1, const int *N1,
                                          int na1, const double *Q2, const double *Z2,
                                          const int *N2, int na2, int amax, double width,
                                          double cut_distance, double r_width, double c_width,
                                          double *D, void *workspace, size_t ws_bytes,
                                          void *stream) {
    return arad_atomic_impl(Q1, Z1, N1, na1, Q2, Z2, N2, na2, amax, nullptr, 0, width,
                            cut_distance, r_width, c_width, D, workspace, ws_bytes, true,
                            FMLB_STREAM(stream));
}

extern "C" size_t fmlb_arad_workspace_bytes(int nm1, int nm2, int amax, int symmetric) {
    if (nm1 < 0 || nm2 < 0 || amax < 1) return 0;
    return fmlb::set_ws_bytes(nm1, amax) + (symmetric ? 0 : fmlb::set_ws_bytes(nm2, amax)) +
           fmlb::align256(sizeof(fmlb::ClassInfo));
}

static int arad_kernels_impl(const double *X1, const double *Z1, const int *N1, int nm1,
                             const double *X2, const double *Z2, const int *N2, int nm2,
                             int amax, const double *sigmas_host, int nsigma, double width,
                             double cut_distance, double r_width, double c_width, int symmetric,
                             int precision, double eps, double *K, void *workspace,
                             size_t ws_bytes, void *stream) {
    using namespace fmlb;
    cudaStream_t st = FMLB_STREAM(stream);
    FMLB_REQUIRE(nm1 >= 0 && amax >= 1, "fmlb_arad_kernels: bad sizes");
    FMLB_REQUIRE(nsigma >= 1 && sigmas_host, "fmlb_arad_kernels: need at least one sigma");
    FMLB_REQUIRE(precision == 0 || precision == 1, "fmlb_arad_kernels: precision must be 0 or 1");
    if (symmetric) {
        X2 = X1; Z2 = Z1; N2 = N1; nm2 = nm1;
    }
    FMLB_REQUIRE(nm2 >= 0, "fmlb_arad_kernels: bad nm2");
    const size_t need = fmlb_arad_workspace_bytes(nm1, nm2, amax, symmetric);
    if (ws_bytes < need || (need && !workspace)) {
        set_error("fmlb_arad_kernels: workspace %zu bytes < required %zu", ws_bytes, need);
        return FMLB_ENOMEM;
    }
    if (nm1 == 0 || nm2 == 0) return FMLB_OK;
    FMLB_REQUIRE(X1 && Z1 && N1 && X2 && Z2 && N2 && K, "fmlb_arad_kernels: null pointer");

    AradParams P;
    P.width = width;
    P.cut = cut_distance;
    P.rw2 = r_width * r_width;
    P.cw2 = c_width * c_width;
    P.inv_width = -1.0 / (4.0 * width * width);      // :58
    P.maxg2 = (8.0 * width) * (8.0 * width);          // :60
    P.inv_cut = (4.0 * atan(1.0)) / (2.0 * cut_distance);  // :502, :510
    P.eps = eps;

    char *p = static_cast<char *>(workspace);
    SetWs w1 = carve(p, nm1, amax);
    SetWs w2 = symmetric ? w1 : carve(p, nm2, amax);
    ClassInfo *ci = reinterpret_cast<ClassInfo *>(p);
    const int tpb = 128;
    const long long npairs = symmetric ? (long long)nm1 * (nm1 + 1) / 2 : (long long)nm1 * nm2;
    // fast paths: amax <= 32 and at most 16 element classes (decided on the device)
    const bool try_fast = amax <= FC_MAXA && !(precision == 0 && f64_generic(amax, npairs));
    ClassInfo *fast_ci = try_fast ? ci : nullptr;
    if (try_fast)
        FMLB_TRY(cuda_status(cudaMemsetAsync(ci, 0, sizeof(ClassInfo), st), "clear class info"));
    struct Set {
        const double *X, *Z;
        const int *N;
        int nm;
        SetWs w;
    } sets[2] = {{X1, Z1, N1, nm1, w1}, {X2, Z2, N2, nm2, w2}};
    const int nsets = symmetric ? 1 : 2;
    for (int q = 0; q < nsets; ++q) {
        const Set &s = sets[q];
        arad_prep_kernel<<<ceil_div((long long)s.nm * amax, PREP_WARPS), PREP_WARPS * 32, 0, st>>>(
            s.X, s.Z, s.N, s.nm, amax, P, symmetric ? 0 : 1, s.w, fast_ci);
        FMLB_TRY(launch_status("arad_prep_kernel"));
    }
    if (try_fast) {
        FMLB_TRY(fast_smem_attrs());
        arad_class_build_kernel<<<1, CB_TPB, 0, st>>>(ci, P.rw2, P.cw2);
        for (int q = 0; q < nsets; ++q) {
            const Set &s = sets[q];
            arad_class_assign_kernel<<<ceil_div((long long)s.nm * amax * amax, 256), 256, 0, st>>>(
                s.X, s.Z, s.N, s.nm, amax, ci, s.w);
            if (precision == 1) {
                arad_sort_records_kernel<<<s.nm, FC_WARPS * 32, 0, st>>>(s.w, s.N, s.nm, amax, ci);
                arad_fast_self_kernel<<<s.nm, FC_WARPS * 32, kFastSmem, st>>>(
                    s.w, s.N, s.nm, amax, P, ci);
            } else {
                arad_f64_self_kernel<<<s.nm, 32, f64_self_smem_bytes(amax), st>>>(
                    s.X, s.w, s.N, s.nm, amax, P, ci);
            }
        }
        FMLB_TRY(launch_status("arad fast-path preparation"));
    }
    for (int q = 0; q < nsets; ++q) {
        const Set &s = sets[q];
        arad_generic_self_kernel<<<ceil_div((long long)s.nm * amax, tpb), tpb, 0, st>>>(
            s.X, s.N, s.nm, amax, P, s.w, fast_ci);
        FMLB_TRY(launch_status("arad_generic_self_kernel"));
    }
    const int blocks = (int)std::min<long long>(ceil_div(npairs, tpb / 32), (long long)sm_count() * 64);
    const int chunk = try_fast && precision == 1 ? FC_MAXSIG : MAXSIG;
    for (int s0 = 0; s0 < nsigma; s0 += chunk) {
        const int ns = nsigma - s0 < chunk ? nsigma - s0 : chunk;
        SigmaTable sig;
        for (int s = 0; s < ns; ++s)
            sig.inv_sigma2[s] = -1.0 / (sigmas_host[s0 + s] * sigmas_host[s0 + s]);
        double *Ks = K + (size_t)s0 * nm1 * nm2;
        if (precision == 0) {
            if (try_fast) {
                const int bj = f64_block(npairs);
                for (int I0 = 0; I0 < nm1; I0 += F6_ROWS) {
                    const dim3 grid(ceil_div(nm2, bj), std::min(F6_ROWS, nm1 - I0));
                    arad_f64_pair_kernel<<<grid, F6_TPB, f64_smem_bytes(amax), st>>>(
                        X1, w1, N1, nm1, X2, w2, N2, nm2, amax, P, ci, sig, ns, symmetric, bj, I0,
                        Ks);
                    FMLB_TRY(launch_status("arad_f64_pair_kernel"));
                    if (nm1 - I0 <= F6_ROWS) break;  // I0 + F6_ROWS may pass 32 bits
                }
            }
            arad_pair_kernel<true><<<blocks, tpb, 0, st>>>(X1, Z1, N1, w1, nm1, X2, Z2, N2, w2, nm2,
                                                           amax, P, sig, ns, symmetric, Ks,
                                                           fast_ci);
        } else {
            if (try_fast) {
                const long long nbi = ceil_div(nm1, FC_BM), nbj = ceil_div(nm2, FC_BM);
                const long long nblk = symmetric ? nbi * (nbi + 1) / 2 : nbi * nbj;
                FMLB_REQUIRE(nblk < (1LL << 31), "fmlb_arad_kernels: too many molecule blocks");
                arad_fast_pair_kernel<<<(unsigned)nblk, FC_WARPS * 32, kFastSmem, st>>>(
                    w1, N1, nm1, w2, N2, nm2, amax, P, ci, sig, ns, symmetric, Ks);
                FMLB_TRY(launch_status("arad_fast_pair_kernel"));
            }
            arad_pair_kernel<false><<<blocks, tpb, 0, st>>>(X1, Z1, N1, w1, nm1, X2, Z2, N2, w2,
                                                            nm2, amax, P, sig, ns, symmetric, Ks,
                                                            fast_ci);
        }
        FMLB_TRY(launch_status("arad_pair_kernel"));
    }
    return FMLB_OK;
}

extern "C" int fmlb_arad_kernels(const double *X1, const double *Z1, const int *N1, int nm1,
                                 const double *X2, const double *Z2, const int *N2, int nm2,
                                 int amax, const double *sigmas_host, int nsigma, double width,
                                 double cut_distance, double r_width, double c_width,
                                 int symmetric, int precision, double *K, void *workspace,
                                 size_t ws_bytes, void *stream) {
    // eps: the single-precision literal 5.0e-12 of farad_kernels.f90:505 / :679
    return arad_kernels_impl(X1, Z1, N1, nm1, X2, Z2, N2, nm2, amax, sigmas_host, nsigma, width,
                             cut_distance, r_width, c_width, symmetric, precision,
                             (double)5.0e-12f, K, workspace, ws_bytes, stream);
}

// The kernel matrix of fget_alpha_arad (farad_kernels.f90:231-393): the
// symmetric FP64 ARAD kernel for one sigma with the routine's fixed
// parameters (width 0.2, cut 6, r_width 1, c_width 0.5, :237-240) and its eps
// (the single-precision literal 1.0e-11, :309), plus lambda on the diagonal
// (:385-389).
extern "C" int fmlb_arad_alpha_kernel_f64(const double *X, const double *Z, const int *N,
                                          int nm, int amax, double sigma, double lambda,
                                          double *K, void *workspace, size_t ws_bytes,
                                          void *stream) {
    using namespace fmlb;
    FMLB_REQUIRE(sigma > 0.0, "fmlb_arad_alpha_kernel_f64: sigma must be positive");
    FMLB_TRY(arad_kernels_impl(X, Z, N, nm, X, Z, N, nm, amax, &sigma, 1, 0.2, 6.0, 1.0, 0.5, 1,
                               0, (double)1.0e-11f, K, workspace, ws_bytes, stream));
    return fmlb_add_diagonal_f64(K, nm, nm, lambda, stream);
}

// atomic_arad_l2_distance_all (farad.f90:452-600), called by
// get_l2_distance_arad (fml/math/distance.py:120-189): D (nm1, nm2, amax, amax)
// with l2 of every atom pair, zero past each molecule's atoms. Sine factors
// for every listed neighbour in both sets (:519-539), eps the single-precision
// literal 5.0e-12 (:509).
extern "C" int fmlb_arad_distances(const double *X1, const double *Z1, const int *N1, int nm1,
                                   const double *X2, const double *Z2, const int *N2, int nm2,
                                   int amax, double width, double cut_distance, double r_width,
                                   double c_width, double *D, void *workspace, size_t ws_bytes,
                                   void *stream) {
    using namespace fmlb;
    cudaStream_t st = FMLB_STREAM(stream);
    FMLB_REQUIRE(nm1 >= 0 && nm2 >= 0 && amax >= 1, "fmlb_arad_distances: bad sizes");
    const size_t need = fmlb_arad_workspace_bytes(nm1, nm2, amax, 0);
    if (ws_bytes < need || (need && !workspace)) {
        set_error("fmlb_arad_distances: workspace %zu bytes < required %zu", ws_bytes, need);
        return FMLB_ENOMEM;
    }
    if (nm1 == 0 || nm2 == 0) return FMLB_OK;
    FMLB_REQUIRE(X1 && Z1 && N1 && X2 && Z2 && N2 && D, "fmlb_arad_distances: null pointer");
    AradParams P;
    P.width = width;
    P.cut = cut_distance;
    P.rw2 = r_width * r_width;
    P.cw2 = c_width * c_width;
    P.inv_width = -1.0 / (4.0 * width * width);
    P.maxg2 = (8.0 * width) * (8.0 * width);
    P.inv_cut = (4.0 * atan(1.0)) / (2.0 * cut_distance);  // farad.f90:515
    P.eps = (double)5.0e-12f;
    char *p = static_cast<char *>(workspace);
    SetWs w1 = carve(p, nm1, amax);
    SetWs w2 = carve(p, nm2, amax);
    const int tpb = 128;
    for (int q = 0; q < 2; ++q) {
        const double *X = q ? X2 : X1, *Z = q ? Z2 : Z1;
        const int *N = q ? N2 : N1, nm = q ? nm2 : nm1;
        const SetWs &w = q ? w2 : w1;
        arad_prep_kernel<<<ceil_div((long long)nm * amax, PREP_WARPS), PREP_WARPS * 32, 0, st>>>(
            X, Z, N, nm, amax, P, 0, w, nullptr);
        FMLB_TRY(launch_status("arad_prep_kernel"));
        arad_generic_self_kernel<<<ceil_div((long long)nm * amax, tpb), tpb, 0, st>>>(
            X, N, nm, amax, P, w, nullptr);
        FMLB_TRY(launch_status("arad_generic_self_kernel"));
    }
    FMLB_TRY(cuda_status(cudaMemsetAsync(D, 0, sizeof(double) * nm1 * nm2 * amax * amax, st),
                         "fmlb_arad_distances: clear D"));
    const long long npairs = (long long)nm1 * nm2;
    const int blocks =
        (int)std::min<long long>(ceil_div(npairs, tpb / 32), (long long)sm_count() * 64);
    SigmaTable sig{};
    arad_pair_kernel<true, true><<<blocks, tpb, 0, st>>>(X1, Z1, N1, w1, nm1, X2, Z2, N2, w2, nm2,
                                                         amax, P, sig, 0, 0, nullptr, nullptr,
                                                         D);
    return launch_status("arad_pair_kernel<distance>");
}
