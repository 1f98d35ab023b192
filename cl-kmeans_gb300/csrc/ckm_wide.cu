// Labels of any point set with 2 <= k <= 256 clusters and d <= 128 features,
// FP32 or FP64, on the tensor cores (tcgen05), with the reference's result.
//
// One persistent CTA per SM runs tiles of 128 points through three roles:
//   - producers (eight warps in teams, a team per tile; a warp takes eight
//     features of all the tile's points): the features, less a common origin
//     and times a power of two, as FP32 x; x = x_h + x_l in fp16 (residual at
//     most 2^-22 |x| + 2^-25) into K-major 128-byte-swizzled operand tiles in a
//     ring of stages, and |x|^2;
//   - one thread issues x_h.c_l and x_l.c_h, then x_h.c_h (tcgen05.mma
//     kind::f16, M = 128, N = the clusters, f32 accumulation) into one of four
//     accumulators in tensor memory (two for more than 128 clusters); the centroids' halves stay in shared
//     memory for the whole launch;
//   - epilogue (two groups of four warps, alternate tiles; a thread is a
//     point = a tensor-memory lane): the lowest score and the second lowest,
//     the certificate, the label.
// Each hand-over is an mbarrier, so the producers' loads, the MMAs and the
// epilogue of neighbouring tiles overlap.
// Every wait has a limit (2 s).  A role whose wait runs out stops the others, and
// the CTA labels its remaining points by the reference's arithmetic with all its
// warps: a failed hand-over costs time, not labels, so there is no error to
// report.
//
// Measured (labels, before: the generic kernel, n k d chained FP32 or FP64
// steps): n = 131072, d = 128, k = 64 330 -> 27 us; n = 300007, d = 21, k = 50
// 119 -> 22 us; n = 2^20, d = 64, k = 256 546 -> 141 us (1.9 TB/s); FP64 n =
// 2^20, d = 4, k = 16 281 -> 51 us.  Bound by issue slots and the latency of
// the epilogue's chain, not by memory or the MMAs (n = 3e6, d = 16, k = 64: 62 %
// of the issue slots, 2600 warp instructions per SM and tile).
//
// The epilogue costs the issue slots, so it keeps two sets of minima instead
// of a sorted pair per score: over the 16 scores of each group of 16 clusters
// (rows) and over the clusters of equal index modulo 16 (columns).  The lowest
// score is at the crossing of the lowest row and the lowest column; every
// other score is in another row or another column, so the second lowest of
// all is the lower of the two second-lowest minima.  That is one three-input
// minimum per two scores for the rows and one for the columns.  The index of
// the lowest column rides in the low four bits of (column minimum - m1).
//
// Certificate.  With x, c the shifted and scaled operands, a >= |x|, r = a + |c|, u
// = 2^-24, D = the features padded to 16, the score |c|^2 - 2 x.c of a cluster is
// off by at most half of
//   3.001 2^-22 r^2       the dropped x_l.c_l and the residuals of the split
//   1.01 gamma r^2        f32 accumulation, gamma = 2 d 2^-23: two ulps per
//                         addition; the 2 d cross products come first and
//                         stay below 2^-10 |x||c|, so d additions count
//   (D / 4 + 18) u r^2    |c|^2 in FP32 (5 steps, D / 8 partial sums, the factor
//                         below), the fma of the score, x and c rounded when
//                         shifted
//   4.1 2^-25 sqrt(D) r   fp16's subnormal range
//   for FP64 points, whose shift by the origin o rounds three times and whose
//   split leaves out 2^-46 |x| (|x_f| <= |t_f| + |o_f|, t = x - o) or 2^-126:
//   8 u r^2 and 8.2 sqrt(D) r (2^-43 max |o| + 2^-120) scale, in x.c and |c|^2
//   2^-40                 second order
// = t2 r^2 + t1 r + 2^-40. As r^2 <= 2 a^2 + 2 |c|^2 and |c| <= 2^-7 |c|^2 + 32, that is
// A + w |c|^2 with A = 2 t2 a^2 + t1 a + 32 t1 + 2^-40 and w = 2 t2 + 2^-7 t1. The cluster's
// own part is taken off its |c|^2 once (times 1 - w/2), so that the scores
// bound the exact ones from below up to A / 2, and a far centroid widens no other
// cluster's bound. The exact score of the lowest one's cluster c1 is at most A / 2
// + w |c1|^2 above its own: all differences hold up to S = A + w |c1|^2. With h = m1 +
// |x|^2, c1 is within h + S of x, squared, so |c1|^2 <= 2 a^2 + 2 (h + S) and S <= A +
// 1.003 2 w (a^2 + h).
// The reference's distance t = x - c, fma(t, t, acc) is within rho = (d + 4) u of the
// exact one (FP32; far less in FP64), plus underflow: T = S + 2.02 rho (h + S)
// + 2 (d + 8) 2^-149 scale^2.
// A second-lowest score more than T above the lowest, m1, proves the label.
// Other points take the reference's arithmetic over the clusters whose score
// is within T of the lowest if these are few. What is left, with more clusters in
// reach or a value that is not finite or too large, waits until the CTA's tiles
// are done and then takes all clusters, a warp's lanes over them; and where a
// warp meets many unproved points (equal centroids) the CTA gives the tensor
// cores up as after a failed wait. Labels, us, with each unproved point's clusters
// in its own thread and now, n = 2^20 (generic or low-d kernel): every hundredth
// point far out, d = 64, k = 256 7937, 195 (551), d = 16, k = 64 328, 51 (75); all
// centroids equal, d = 16, k = 64 483, 144 (75); two equal 98, 83 (75).
#include <cuda_fp16.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <cstdlib>
#include <mutex>

#include "ckm_device.cuh"
#include "ckm_internal.h"
#include "ckm_umma.cuh"

namespace ckm {
namespace {

constexpr uint32_t WM = 128;              // points per tile (tensor-memory lanes)
constexpr uint32_t W_MAX_K = 256;
constexpr uint32_t W_MAX_D = 128;
// Warps: EG groups of four for the epilogue, then eight producers, then four
// for the MMAs.
constexpr uint32_t w_threads(uint32_t EG) { return 32 * (4 * EG + 12); }
constexpr uint32_t W_TILE_BYTES = WM * 128u;  // one operand tile: 128 rows of 64 fp16
constexpr uint32_t W_NX_SLOTS = 8, W_NX_ROWS = 48;
constexpr float W_MAX_ABS = 32768.0f;         // |x| and |c| below: no fp16 overflow
constexpr unsigned long long W_WAIT_NS = 2000000000ull;
// What the tile loop does not resolve itself has this label until its end.
constexpr uint32_t W_LATER = 0xffffffffu;
constexpr uint32_t W_CANDIDATES = 4;          // fewer exact distances than this of a point in the tile loop
// Unproved points that a warp takes before the CTA gives the tensor cores up,
// some and a share of every tile's 32: beyond an eighth the exact labels by all
// of the CTA's warps cost less.
constexpr uint32_t W_UNPROVED_MIN = 16, W_UNPROVED_PER_TILE = 4;
// A poll of a barrier suspends its thread up to this long: labels of n = 2^20, d =
// 64, k = 256 142 us with 2 us (polls that run out within a tile), 141 with 6, 140.3
// with 20; a CTA that gives up leaves that much later (all centroids equal, d = 16,
// k = 64: 144, 144 and 162 us).
constexpr uint32_t W_POLL_NS = 6000;

template <typename T, typename L>
struct WideArgs {
    const T* points;
    const T* centroids;
    L* labels;
    unsigned long long* msum;  // counts are added here (nullptr: not counted)
    unsigned long long wait_ns;  // limit of every wait
    uint64_t n;
    uint32_t d, k, dk, kp, kblocks, stages, stages_log2, teams, tiles;
};

__device__ __forceinline__ unsigned long long w_now_ns() {
    unsigned long long t;
    asm volatile("mov.u64 %0, %globaltimer;" : "=l"(t));
    return t;
}

__device__ __forceinline__ bool w_try_wait(uint32_t bar, uint32_t parity, uint32_t poll) {
    uint32_t ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2, %3;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(ok)
        : "r"(bar), "r"(parity), "r"(poll)
        : "memory");
    return ok != 0;
}

// mbarrier wait with a time limit and a shared flag; false when another role
// gave the tensor cores up or the phase did not complete in time.
__device__ __forceinline__ bool w_wait(uint32_t bar, uint32_t parity, volatile unsigned int* abort_flag,
                                       unsigned long long limit) {
    const uint32_t poll = limit < W_POLL_NS ? (uint32_t)limit : W_POLL_NS;
    if (w_try_wait(bar, parity, poll)) return true;
    const unsigned long long t0 = w_now_ns();
    for (;;) {
        if (w_try_wait(bar, parity, poll)) return true;
        if (*abort_flag) return false;
        if (w_now_ns() - t0 >= limit) {
            *abort_flag = 1u;
            return false;
        }
    }
}

// True in one thread of a converged warp.
__device__ __forceinline__ bool w_elect() {
    uint32_t one;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "elect.sync _|p, 0xffffffff;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(one));
    return one != 0;
}

__device__ __forceinline__ void w_arrive(uint32_t bar) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory");
}

// Issues the load of 16 accumulator columns of this thread's lane; the values
// are there after w_ld_wait on the same array.
__device__ __forceinline__ void w_ld16(uint32_t taddr, float (&v)[16]) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
        : "=f"(v[0]), "=f"(v[1]), "=f"(v[2]), "=f"(v[3]), "=f"(v[4]), "=f"(v[5]), "=f"(v[6]), "=f"(v[7]),
          "=f"(v[8]), "=f"(v[9]), "=f"(v[10]), "=f"(v[11]), "=f"(v[12]), "=f"(v[13]), "=f"(v[14]), "=f"(v[15])
        : "r"(taddr));
}
__device__ __forceinline__ void w_ld_wait(float (&v)[16]) {
    asm volatile("tcgen05.wait::ld.sync.aligned;"
                 : "+f"(v[0]), "+f"(v[1]), "+f"(v[2]), "+f"(v[3]), "+f"(v[4]), "+f"(v[5]), "+f"(v[6]), "+f"(v[7]),
                   "+f"(v[8]), "+f"(v[9]), "+f"(v[10]), "+f"(v[11]), "+f"(v[12]), "+f"(v[13]), "+f"(v[14]),
                   "+f"(v[15])
                 :
                 : "memory");
}

__device__ __forceinline__ uint32_t w_idesc(uint32_t N) {  // kind::f16, fp16 A and B, f32 D, both K-major
    return (1u << 4) | ((N >> 3) << 17) | ((WM >> 4) << 24);
}

// Power of two that brings maxabs into [2^7, 2^8) (1 for 0), exponent kept
// within +-60 so that it and its square stay normal.
__device__ __forceinline__ float w_scale(float maxabs) {
    if (!(maxabs > 0.0f)) return 1.0f;
    int e = 0;
    frexpf(maxabs, &e);  // maxabs < 2^e
    const int s = 8 - e;
    return ldexpf(1.0f, s < -60 ? -60 : (s > 60 ? 60 : s));
}

// (v - mu) * scale as FP32, two features at a time.  FP32: one fma with
// shift = -mu * scale (exact: scale is a power of two), so the result is
// rounded once; FP64: both are cut into two floats (split64; shift holds those
// of mu, negated) and subtracted piecewise, as a subtraction and a conversion on
// the FP64 pipe took a third of the kernel's time (labels n = 600000 d = 16 k = 40
// 55 -> 43 us, d = 64 k = 64 178 -> 120, d = 33 k = 5 146 -> 87).
__device__ __forceinline__ float2 w_shift(float2 v, float2 shift, float scale) {
    return fma2(v, make_float2(scale, scale), shift);
}
__device__ __forceinline__ float2 w_floats(double v) {  // two floats in the place of a double
    return make_float2(__int_as_float(__double2loint(v)), __int_as_float(__double2hiint(v)));
}
__device__ __forceinline__ float2 w_shift(double2 v, double2 shift, float scale) {
    float2 h, l;
    split64(v.x, h.x, l.x);
    split64(v.y, h.y, l.y);
    const float2 sx = w_floats(shift.x), sy = w_floats(shift.y);
    const float2 t = add2(add2(h, make_float2(sx.x, sy.x)), add2(l, make_float2(sx.y, sy.y)));
    return make_float2(t.x * scale, t.y * scale);
}
// The shift of a feature from its origin.
__device__ __forceinline__ float w_shift_of(float mu, float scale) { return -mu * scale; }
__device__ __forceinline__ double w_shift_of(double mu, float) {
    const float h = (float)mu;
    return __hiloint2double(__float_as_int(isinf(h) ? 0.0f : -(float)(mu - (double)h)), __float_as_int(-h));
}
template <typename T> struct Pair;
template <> struct Pair<float> { using type = float2; };
template <> struct Pair<double> { using type = double2; };

// Eight consecutive features of row r as fp16 halves into the hi and lo
// tiles; adds their squares to ss.
__device__ __forceinline__ void w_store8(uint32_t hi, uint32_t lo, uint32_t off, const float2 (&x)[4], float2& ss) {
    uint32_t h[4], l[4];
#pragma unroll
    for (int e = 0; e < 4; ++e) {
        ss = fma2(x[e], x[e], ss);
        const __half2 hh = __floats2half2_rn(x[e].x, x[e].y);
        const float2 lf = sub2(x[e], __half22float2(hh));
        const __half2 ll = __floats2half2_rn(lf.x, lf.y);
        h[e] = *reinterpret_cast<const uint32_t*>(&hh);
        l[e] = *reinterpret_cast<const uint32_t*>(&ll);
    }
    asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(hi + off), "r"(h[0]), "r"(h[1]), "r"(h[2]), "r"(h[3])
                 : "memory");
    asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(lo + off), "r"(l[0]), "r"(l[1]), "r"(l[2]), "r"(l[3])
                 : "memory");
}

__device__ __forceinline__ float w_tag(float v, uint32_t i) {
    return __uint_as_float((__float_as_uint(v) & 0xfffffff0u) | i);
}

// Lowest (with its index in the low four bits) and second lowest of 16.
__device__ __forceinline__ void w_lowest2(const float (&v)[16], float& lo, float& hi) {
    float l[8], h[8];
#pragma unroll
    for (int i = 0; i < 8; ++i) {
        const float a = w_tag(v[2 * i], 2 * i), b = w_tag(v[2 * i + 1], 2 * i + 1);
        l[i] = fminf(a, b);
        h[i] = fmaxf(a, b);
    }
#pragma unroll
    for (int w = 4; w >= 1; w >>= 1)
#pragma unroll
        for (int i = 0; i < w; ++i) {
            const float t = fmaxf(l[i], l[i + w]);
            h[i] = fmin3(t, h[i], h[i + w]);
            l[i] = fminf(l[i], l[i + w]);
        }
    lo = l[0];
    hi = h[0];
}

// The reference's distance of point p to cluster c, f ascending.
template <typename T>
__device__ __forceinline__ T w_distance(const T* __restrict__ P, uint64_t n, uint64_t p, const T* __restrict__ C,
                                        uint32_t k, uint32_t c, uint32_t d) {
    T acc = T(0);
    uint32_t f = 0;
    for (; f + 8 <= d; f += 8) {
        T t[8];
#pragma unroll
        for (int e = 0; e < 8; ++e)
            t[e] = __ldg(P + (uint64_t)(f + e) * n + p) - __ldg(C + (uint64_t)(f + e) * k + c);
#pragma unroll
        for (int e = 0; e < 8; ++e) acc = fma(t[e], t[e], acc);
    }
    for (; f < d; ++f) {
        const T t = __ldg(P + (uint64_t)f * n + p) - __ldg(C + (uint64_t)f * k + c);
        acc = fma(t, t, acc);
    }
    return acc;
}

// acc[j] = fma(t, t, acc[j]), t = x - row[j], for eight clusters; WORDS: row is
// 16-byte aligned and readable to the eighth (else the first `left` are read).
template <bool WORDS>
__device__ __forceinline__ void w_step8(float x, const float* row, uint32_t left, float (&acc)[8]) {
    float c[8];
    if constexpr (WORDS) {
        const float4 u = *reinterpret_cast<const float4*>(row), v = *reinterpret_cast<const float4*>(row + 4);
        c[0] = u.x, c[1] = u.y, c[2] = u.z, c[3] = u.w, c[4] = v.x, c[5] = v.y, c[6] = v.z, c[7] = v.w;
    } else {
#pragma unroll
        for (uint32_t j = 0; j < 8; ++j) c[j] = j < left ? __ldg(row + j) : 0.0f;
    }
#pragma unroll
    for (uint32_t j = 0; j < 8; j += 2) {
        const float2 t = sub2(make_float2(x, x), make_float2(c[j], c[j + 1]));
        const float2 s = fma2(t, t, make_float2(acc[j], acc[j + 1]));
        acc[j] = s.x;
        acc[j + 1] = s.y;
    }
}
template <bool WORDS>
__device__ __forceinline__ void w_step8(double x, const double* row, uint32_t left, double (&acc)[8]) {
    double c[8];
#pragma unroll
    for (uint32_t j = 0; j < 8; j += 2) {
        if constexpr (WORDS) {
            const double2 u = *reinterpret_cast<const double2*>(row + j);
            c[j] = u.x, c[j + 1] = u.y;
        } else {
            c[j] = j < left ? __ldg(row + j) : 0.0;
            c[j + 1] = j + 1 < left ? __ldg(row + j + 1) : 0.0;
        }
    }
#pragma unroll
    for (uint32_t j = 0; j < 8; ++j) {
        const double t = x - c[j];
        acc[j] = fma(t, t, acc[j]);
    }
}

// The reference's label of point p + lane by all clusters, eight at a time; the
// centroid of feature f and cluster c is at C[f * stride + c].  Past the last
// point the last one is labelled.
template <typename T, bool SHARED>
__device__ __noinline__ uint32_t w_exact32(const T* __restrict__ P, uint64_t n, uint64_t p, const T* C, uint32_t stride,
                                           uint32_t k, uint32_t d) {
    const uint64_t at = p + (threadIdx.x & 31u);
    const T* first = P + (at < n ? at : n - 1);
    T best = TypeMax<T>::v();
    uint32_t label = 0;
    for (uint32_t c0 = 0; c0 < k; c0 += 8) {
        T acc[8];
#pragma unroll
        for (uint32_t j = 0; j < 8; ++j) acc[j] = T(0);
        const T* src = first;
        const T* row = C + c0;
#pragma unroll 4
        for (uint32_t f = 0; f < d; ++f, src += n, row += stride) w_step8<SHARED>(__ldg(src), row, k - c0, acc);
#pragma unroll
        for (uint32_t j = 0; j < 8; ++j)
            if (c0 + j < k && acc[j] < best) {
                best = acc[j];
                label = c0 + j;
            }
    }
    return label;
}

// The reference's label of one point by all clusters: the lanes of a warp over
// the clusters, J per lane, U features' loads in flight.
template <typename T, bool SHARED, uint32_t J, uint32_t U>
__device__ __forceinline__ uint32_t w_exact1(const T* __restrict__ P, uint64_t n, uint64_t p, const T* C,
                                             uint32_t stride, uint32_t k, uint32_t d) {
    const uint32_t lane = threadIdx.x & 31u;
    T best = TypeMax<T>::v();
    uint32_t label = 0;
    for (uint32_t c0 = lane; c0 < k + lane; c0 += 32 * J) {
        T acc[J];
#pragma unroll
        for (uint32_t j = 0; j < J; ++j) acc[j] = T(0);
        for (uint32_t f0 = 0; f0 < d; f0 += 32) {
            const T mine = f0 + lane < d ? __ldg(P + (uint64_t)(f0 + lane) * n + p) : T(0);
            const uint32_t left = min(32u, d - f0);
            for (uint32_t f = 0; f < left; f += U) {
                T c[U][J];
#pragma unroll
                for (uint32_t u = 0; u < U; ++u)
#pragma unroll
                    for (uint32_t j = 0; j < J; ++j)
                        if (f + u < left && c0 + 32 * j < k) {
                            const T* at = C + (size_t)(f0 + f + u) * stride + c0 + 32 * j;
                            c[u][j] = SHARED ? *at : __ldg(at);
                        } else {
                            c[u][j] = T(0);
                        }
#pragma unroll
                for (uint32_t u = 0; u < U; ++u) {
                    const T x = __shfl_sync(0xffffffffu, mine, (f + u) & 31u);
                    if (f + u < left)
#pragma unroll
                        for (uint32_t j = 0; j < J; ++j) {
                            const T t = x - c[u][j];
                            acc[j] = fma(t, t, acc[j]);
                        }
                }
            }
        }
#pragma unroll
        for (uint32_t j = 0; j < J; ++j)
            if (c0 + 32 * j < k && acc[j] < best) {
                best = acc[j];
                label = c0 + 32 * j;
            }
    }
    // the lowest cluster of the lowest distance; none below the type's maximum: 0
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        const T b = __shfl_xor_sync(0xffffffffu, best, o);
        const uint32_t l = __shfl_xor_sync(0xffffffffu, label, o);
        if (b < best || (b == best && l < label)) {
            best = b;
            label = l;
        }
    }
    return label;
}
template <typename T, bool SHARED>
__device__ __noinline__ uint32_t w_by_all(const T* __restrict__ P, uint64_t n, uint64_t p, const T* C, uint32_t stride,
                                          uint32_t k, uint32_t d) {
    if (k <= 64) return w_exact1<T, SHARED, 2, 8>(P, n, p, C, stride, k, d);
    return w_exact1<T, SHARED, 8, 16 / sizeof(T)>(P, n, p, C, stride, k, d);
}

// EG epilogue groups, ACCS accumulators (a multiple of EG).
template <typename T, typename L, int EG, int ACCS>
__global__ void __launch_bounds__(w_threads(EG), 1) wide_label_kernel(const WideArgs<T, L> a) {
    constexpr uint32_t W_THREADS = w_threads(EG), W_EPI_WARPS = 4 * EG, W_MMA_WARP = W_EPI_WARPS + 8;
    extern __shared__ unsigned char smem_raw[];
    __shared__ __align__(8) uint64_t bar_af[4], bar_ae[4], bar_tf[4], bar_te[4], bar_nx[W_NX_SLOTS], bar_fin;
    __shared__ uint32_t s_tmem;
    __shared__ unsigned int s_abort, s_later, s_cabs, s_cn_max, s_bad, s_omax;
    __shared__ __align__(16) float s_cn[W_MAX_K];
    __shared__ __align__(16) T s_mu[W_MAX_D];     // the origin, then the shift of w_shift
    __shared__ uint32_t s_invalid[W_MAX_K / 32];
    __shared__ float s_nx[W_NX_ROWS][WM];  // partial |x|^2: [slot][part][point]
    __shared__ unsigned int s_mass[W_MAX_K];
    __shared__ uint32_t s_next[W_EPI_WARPS];  // the first tile that an epilogue warp has not labelled
    volatile unsigned int* abort_flag = &s_abort;

    // the warp index as a value the compiler knows to be the same in the whole
    // warp: the roles' branches and addresses stay on the uniform datapath
    const uint32_t tid = threadIdx.x, warp = __shfl_sync(0xffffffffu, tid >> 5, 0), lane = tid & 31u;
    const uint32_t d = a.d, k = a.k, dk = a.dk, kp = a.kp;
    const uint64_t n = a.n;
    const uint32_t sB = (umma::smem_u32(smem_raw) + 1023u) & ~1023u;
    const uint32_t b_part = a.kblocks * kp * 128u;      // one half (hi or lo) of the centroids
    const uint32_t sA = sB + 2u * b_part;
    const uint32_t a_part = a.kblocks * W_TILE_BYTES;   // one half of a tile
    const uint32_t a_bytes = 2u * a_part;
    uint32_t cols = 32;
    while (cols < kp) cols <<= 1;
    constexpr uint32_t accs = ACCS;
    // producers: `teams` teams of `team_warps`; a tile's items are its chunks
    // of 8 features (times two halves of its points in FP64), of which a
    // warp takes every team_warps-th; the warps with any are the members
    constexpr uint32_t PPT = 16 / sizeof(T), HALVES = 4 / PPT;  // points per thread, parts of a tile
    const uint32_t used = (d + 7) / 8, items = used * HALVES;
    const uint32_t team_warps = 8 / a.teams, members = min(team_warps, items);
    // MMA warps: a warp meets every phase of the barriers it waits on, so
    // their number divides those of the stages and of the accumulators
    const uint32_t mma_warps = min(a.stages, accs);
    // the |x|^2 parts of a tile are read after its stage is free again, by an
    // epilogue group whose previous tile has left its accumulator: the slots
    // go round after stages + accumulators tiles (an even number, as a group
    // takes every other tile)
    const uint32_t nx_slots = (a.stages + accs + 1u) & ~1u, nx_parts = members / HALVES;

    if (tid == 0) {
        for (int i = 0; i < 4; ++i) {
            umma::mbar_init(umma::smem_u32(&bar_af[i]), members);
            umma::mbar_init(umma::smem_u32(&bar_ae[i]), 1);
        }
        for (int i = 0; i < 4; ++i) {
            umma::mbar_init(umma::smem_u32(&bar_tf[i]), 1);
            umma::mbar_init(umma::smem_u32(&bar_te[i]), 4);
        }
        for (uint32_t i = 0; i < W_NX_SLOTS; ++i) umma::mbar_init(umma::smem_u32(&bar_nx[i]), members);
        umma::mbar_init(umma::smem_u32(&bar_fin), mma_warps);
        umma::mbar_fence_init();
        s_abort = 0u;
        s_later = 0u;
        s_cabs = 0u;
        s_omax = 0u;
        s_cn_max = 0u;
        s_bad = 0u;
    }
    if (warp == W_MMA_WARP) umma::tmem_alloc(umma::smem_u32(&s_tmem), accs * cols);
    for (uint32_t i = tid; i < W_MAX_K; i += W_THREADS) {
        s_cn[i] = 0.0f;
        s_mass[i] = 0u;
    }
    for (uint32_t i = tid; i < W_MAX_D; i += W_THREADS) s_mu[i] = T(0);
    if (tid < W_MAX_K / 32) s_invalid[tid] = 0u;
    umma::fence_before_sync();
    __syncthreads();
    umma::fence_after_sync();
    const uint32_t tmem = s_tmem;

    // ---- centroids: origin, validity, scale, fp16 halves, |c|^2 ----
    // A centroid with a coordinate that is not finite never wins in the
    // reference (its distance is not below the type's maximum): a zero row
    // with a huge |c|^2.  The origin is a median of medians of 27 of the
    // centroids, which a few far ones do not move; any finite value would do.
    for (uint32_t f = warp; f < d; f += W_THREADS / 32) {
        const T* row = a.centroids + (uint64_t)f * k;
        for (uint32_t c = lane; c < k; c += 32)
            if (!isfinite(__ldg(row + c))) atomicOr(&s_invalid[c >> 5], 1u << (c & 31u));
        T m = __ldg(row + (lane < 27 ? lane * k / 27 : 0u));
#pragma unroll
        for (uint32_t i = 0; i < 3; ++i) {  // medians of three, of 9 threes, then 3, then 1
            const T x = __shfl_sync(0xffffffffu, m, 3 * lane), y = __shfl_sync(0xffffffffu, m, 3 * lane + 1),
                    z = __shfl_sync(0xffffffffu, m, 3 * lane + 2);
            m = fmax(fmin(x, y), fmin(fmax(x, y), z));
        }
        if (lane == 0) s_mu[f] = isfinite(m) ? m : T(0);
    }
    __syncthreads();
    {
        float m = 0.0f;
        for (uint32_t f = warp; f < d; f += W_THREADS / 32)
            for (uint32_t c = lane; c < k; c += 32)
                if (!((s_invalid[c >> 5] >> (c & 31u)) & 1u)) {
                    const float v = fabsf((float)(__ldg(a.centroids + (uint64_t)f * k + c) - s_mu[f]));
                    if (isfinite(v)) m = fmaxf(m, v);
                    else s_bad = 1u;  // no FP32 image of a finite centroid: exact labels for every point
                }
        const uint32_t mb = __reduce_max_sync(0xffffffffu, __float_as_uint(m));
        if (lane == 0) atomicMax(&s_cabs, mb);
    }
    __syncthreads();
    const float scale = w_scale(__uint_as_float(s_cabs));
    if (sizeof(T) == 8)  // max |origin|, for the certificate
        for (uint32_t f = tid; f < d; f += W_THREADS) atomicMax(&s_omax, __float_as_uint(__double2float_ru(fabs((double)s_mu[f]))));
    __syncthreads();
    using T2 = typename Pair<T>::type;
    for (uint32_t f = tid; f < W_MAX_D; f += W_THREADS) s_mu[f] = w_shift_of(s_mu[f], scale);
    __syncthreads();
    for (uint32_t u = warp; u < (dk / 8) * ((kp + 31) / 32); u += W_THREADS / 32) {
        const uint32_t j = u % (dk / 8), c = u / (dk / 8) * 32 + lane;
        if (c >= kp) continue;
        const bool valid = c < k && !((s_invalid[c >> 5] >> (c & 31u)) & 1u) && !s_bad;
        float2 x[4];
#pragma unroll
        for (int e = 0; e < 4; ++e) {
            T2 v, shift;
            const uint32_t f = 8 * j + 2 * e;
            shift.x = s_mu[f];
            shift.y = s_mu[f + 1];
            v.x = valid && f < d ? __ldg(a.centroids + (uint64_t)f * k + c) : T(0);
            v.y = valid && f + 1 < d ? __ldg(a.centroids + (uint64_t)(f + 1) * k + c) : T(0);
            x[e] = w_shift(v, shift, scale);
            if (!valid) x[e] = make_float2(0.0f, 0.0f);
        }
        float2 ss = make_float2(0.0f, 0.0f);
        const uint32_t off = (j >> 3) * kp * 128u + umma::sw128_offset(c, (j & 7u) * 8u);
        w_store8(sB, sB + b_part, off, x, ss);
        if (valid) atomicAdd(&s_cn[c], ss.x + ss.y);
    }
    __syncthreads();
    // the certificate's constants, and |c|^2 less each cluster's part of the bound
    const float fd = (float)d, fk = (float)dk;
    const float t2 = (3.001f * 0x1p-22f + 1.01f * 2.0f * fd * 0x1p-23f * 1.005f + (0.25f * fk + (sizeof(T) == 4 ? 18.0f : 26.0f)) * 0x1p-24f) *
                     1.002f;
    const float origin = sizeof(T) == 4 ? 0.0f : fmaf(__uint_as_float(s_omax), 0x1p-43f, 0x1p-120f) * scale;
    const float t1 = (4.1f * 0x1p-25f + 8.2f * origin) * sqrtf(fk) * 1.001f;
    const float w = (2.0f * t2 + t1 * 0x1p-7f) * 1.001f;
    for (uint32_t c = tid; c < kp; c += W_THREADS) {
        const bool valid = c < k && !((s_invalid[c >> 5] >> (c & 31u)) & 1u) && !s_bad;
        if (valid) atomicMax(&s_cn_max, __float_as_uint(s_cn[c]));
        s_cn[c] = valid ? s_cn[c] * (1.0f - (0.5f * w + 0x1p-24f)) : 0x1p126f;
    }
    // the padding features of the point tiles stay zero
    for (uint32_t u = warp; u < a.stages * 2 * 4; u += W_THREADS / 32)
        for (uint32_t j = used; j < dk / 8; ++j) {
            const uint32_t r = (u & 3u) * 32 + lane;
            const uint32_t at = sA + (u >> 2) * a_part + (j >> 3) * W_TILE_BYTES + umma::sw128_offset(r, (j & 7u) * 8u);
            asm volatile("st.shared.v4.b32 [%0], {%1, %1, %1, %1};" ::"r"(at), "r"(0u) : "memory");
        }
    umma::fence_proxy_async_smem();
    __syncthreads();

    if (warp >= W_EPI_WARPS && warp < W_MMA_WARP) {
        // ---- producers ----
        // The loads of a warp's next item (of its next tile, after the last)
        // are issued as soon as the current one is converted.
        const uint32_t pw = warp - W_EPI_WARPS, team = pw / team_warps, m = pw % team_warps;
        const uint64_t row_bytes = n * sizeof(T);
        T v[8][PPT];
        auto load = [&](uint32_t t, uint32_t item) {
            if (t >= a.tiles) return;
            const uint32_t j = item / HALVES;
            const uint64_t p = (uint64_t)t * WM + (item % HALVES) * (32 * PPT) + lane;
            const char* src = reinterpret_cast<const char*>(a.points + (uint64_t)j * 8 * n + p);
            if ((uint64_t)t * WM + WM <= n && j * 8 + 8 <= d) {
#pragma unroll
                for (uint32_t e = 0; e < 8; ++e) {
#pragma unroll
                    for (uint32_t i = 0; i < PPT; ++i) v[e][i] = __ldg(reinterpret_cast<const T*>(src) + 32 * i);
                    src += row_bytes;
                }
            } else {
#pragma unroll
                for (uint32_t e = 0; e < 8; ++e) {
#pragma unroll
                    for (uint32_t i = 0; i < PPT; ++i)
                        v[e][i] = j * 8 + e < d && p + 32 * i < n ? __ldg(reinterpret_cast<const T*>(src) + 32 * i) : T(0);
                    src += row_bytes;
                }
            }
        };
        const uint32_t stride = a.teams * gridDim.x;
        uint32_t it = team, slot = team;
        if (m < members) {
            load(blockIdx.x + team * gridDim.x, m);
            for (uint32_t t = blockIdx.x + team * gridDim.x; t < a.tiles; t += stride, it += a.teams) {
                // the team's next tile but one into L2 (128 bytes per thread)
                const uint64_t pn = ((uint64_t)t + 2 * stride) * WM;
                for (uint32_t i = m * 32 + lane; i < d * 4 * (uint32_t)(sizeof(T) / 4) && pn < n; i += members * 32) {
                    constexpr uint32_t LINE = 128 / sizeof(T);
                    const uint64_t pp = pn + (i % (WM / LINE)) * LINE;
                    if (pp < n)
                        asm volatile("prefetch.global.L2 [%0];" ::"l"(a.points + (uint64_t)(i / (WM / LINE)) * n + pp));
                }
                // the stage is free once the MMAs of the tile `stages` before are done
                const uint32_t stage = it & (a.stages - 1u);
                const bool ok = w_wait(umma::smem_u32(&bar_ae[stage]), ((it >> a.stages_log2) & 1u) ^ 1u, abort_flag, a.wait_ns);
                if (!__all_sync(0xffffffffu, ok)) break;
                const uint32_t hi = sA + stage * a_bytes;
                float2 ss[PPT];
#pragma unroll
                for (uint32_t i = 0; i < PPT; ++i) ss[i] = make_float2(0.0f, 0.0f);
#pragma unroll 1
                for (uint32_t item = m; item < items; item += team_warps) {
                    const uint32_t j = item / HALVES;
                    const uint32_t row = (item % HALVES) * (32 * PPT) + lane;
                    const uint32_t off = (j >> 3) * W_TILE_BYTES + umma::sw128_offset(row, (j & 7u) * 8u);
                    T2 shift[4];
#pragma unroll
                    for (int e = 0; e < 4; ++e) shift[e] = *reinterpret_cast<const T2*>(&s_mu[8 * j + 2 * e]);
#pragma unroll
                    for (uint32_t i = 0; i < PPT; ++i) {
                        float2 x[4];
#pragma unroll
                        for (int e = 0; e < 4; ++e) {
                            x[e] = make_float2(0.0f, 0.0f);
                            if (sizeof(T) == 4 || 8 * j + 2 * e < d) {  // (FP64 points take some 30 operations)
                                T2 vv;
                                vv.x = v[2 * e][i];
                                vv.y = v[2 * e + 1][i];
                                x[e] = w_shift(vv, shift[e], scale);
                            }
                        }
                        w_store8(hi + i * 32u * 128u, hi + a_part + i * 32u * 128u, off, x, ss[i]);
                    }
                    if (item + team_warps < items) load(t, item + team_warps);
                    else load(t + stride, m);
                }
#pragma unroll
                for (uint32_t i = 0; i < PPT; ++i)
                    s_nx[slot * nx_parts + m / HALVES][(m % HALVES) * (32 * PPT) + i * 32 + lane] = ss[i].x + ss[i].y;
                umma::fence_proxy_async_smem();
                __syncwarp();
                if (lane == 0) {
                    w_arrive(umma::smem_u32(&bar_nx[slot]));
                    w_arrive(umma::smem_u32(&bar_af[stage]));
                }
                slot += a.teams;
                if (slot >= nx_slots) slot -= nx_slots;
            }
        }
    } else if (warp >= W_MMA_WARP) {
        // ---- MMA issue: warps take tiles in turn (the waits and the issue of
        // a tile are a serial chain of some 1000 cycles), each keeps its
        // control flow uniform and one elected thread issues ----
        const uint32_t mw = warp - W_MMA_WARP;
        const uint32_t idesc = w_idesc(kp), steps = dk / 16;
        const uint64_t bh = umma::sw128_desc(sB), bl = umma::sw128_desc(sB + b_part);
        const uint64_t bblock = (kp * 128u) >> 4, ablock = W_TILE_BYTES >> 4;  // descriptor steps to the next 64 features
        for (uint32_t it = mw; mw < mma_warps; it += mma_warps) {
            if ((uint64_t)blockIdx.x + (uint64_t)it * gridDim.x >= a.tiles) break;
            const uint32_t b = it % accs, stage = it & (a.stages - 1u);
            // lane 0 polls the operands' barrier, the others the accumulator's
            const uint32_t bar = lane == 0 ? umma::smem_u32(&bar_af[stage]) : umma::smem_u32(&bar_te[b]);
            const uint32_t parity = lane == 0 ? (it >> a.stages_log2) & 1u : ((it / accs) & 1u) ^ 1u;
            const bool ok = w_wait(bar, parity, abort_flag, a.wait_ns);
            if (!__all_sync(0xffffffffu, ok)) break;
            __syncwarp();
            umma::fence_after_sync();
            const uint32_t acc = tmem + b * cols;
            const uint64_t ah = umma::sw128_desc(sA + stage * a_bytes), al = umma::sw128_desc(sA + stage * a_bytes + a_part);
            if (w_elect()) {
                // the cross products first, then x_h c_h; a small loop, as this
                // warp's instructions share the cache with the other roles'
#pragma unroll 1
                for (uint32_t pass = 0; pass < 3; ++pass) {
                    uint64_t ad = pass == 1 ? al : ah, bd = pass == 0 ? bl : bh;
#pragma unroll 1
                    for (uint32_t ks = 0; ks < steps; ++ks) {
                        umma::mma_bf16(acc, ad, bd, idesc, pass + ks);
                        const bool block = (ks & 3u) == 3u;  // the next 64 features
                        ad += block ? ablock - 6 : 2;
                        bd += block ? bblock - 6 : 2;
                    }
                }
                umma::mma_commit(umma::smem_u32(&bar_tf[b]));
                umma::mma_commit(umma::smem_u32(&bar_ae[stage]));
            }
            __syncwarp();
        }
        // every MMA issued has completed before tensor memory is freed
        if (mw < mma_warps && w_elect()) {
            umma::mma_commit(umma::smem_u32(&bar_fin));
            umma::mbar_wait(umma::smem_u32(&bar_fin), 0u, 1u << 22);
        }
        __syncwarp();
    } else {
        // ---- epilogue ----
        const uint32_t g = warp >> 2, q = warp & 3u, row = q * 32 + lane;
        const float INF = __int_as_float(0x7f800000);
        const float cm = s_bad ? INF : sqrtf(__uint_as_float(s_cn_max)) * (1.0f + 0x1p-16f);
        const float t00 = t1 * 32.0f + 0x1p-40f, wc = 2.0f * (w * 1.001f + 0x1p-22f) * 1.003f;
        const float ta = 2.0f * t2 + wc;
        const float rho = sizeof(T) == 4 ? 2.02f * (fd + 4.0f) * 0x1p-24f * 1.001f : 0x1p-40f;
        const float t0 = 2.0f * (fd + 8.0f) * 0x1p-149f * scale * scale;
        const float rmax = 0x1p60f * scale;
        const float2 two = make_float2(-2.0f, -2.0f);
        uint32_t b = g, phase = 0, slot = g, nx_phase = 0;  // the slots go round as the tiles of all groups do
        uint32_t t = blockIdx.x + g * gridDim.x;
        uint32_t allowed = W_UNPROVED_MIN;
        for (; t < a.tiles; t += EG * gridDim.x) {
            const uint32_t taddr = tmem + b * cols + ((q * 32u) << 16);
            const uint32_t bar_full = umma::smem_u32(&bar_tf[b]), bar_empty = umma::smem_u32(&bar_te[b]);
            // lane 0 polls the scores' barrier, the others the norms'
            const bool ok = w_wait(lane == 0 ? bar_full : umma::smem_u32(&bar_nx[slot]), lane == 0 ? phase : nx_phase,
                                   abort_flag, a.wait_ns);
            if (!__all_sync(0xffffffffu, ok)) break;
            __syncwarp();
            umma::fence_after_sync();
            float v0[16], v1[16], col[16];
            float m1 = INF, m2 = INF;
            uint32_t r1 = 0;
#pragma unroll
            for (int i = 0; i < 16; ++i) col[i] = INF;
            // scores of one group of 16 clusters, in place; its minimum
            auto score = [&](float (&s)[16], uint32_t cc) {
                const float4* cn4 = reinterpret_cast<const float4*>(s_cn + cc);
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    const float4 c = cn4[i];
                    const float2 lo2 = fma2(make_float2(s[4 * i], s[4 * i + 1]), two, make_float2(c.x, c.y));
                    const float2 hi2 = fma2(make_float2(s[4 * i + 2], s[4 * i + 3]), two, make_float2(c.z, c.w));
                    s[4 * i] = lo2.x;
                    s[4 * i + 1] = lo2.y;
                    s[4 * i + 2] = hi2.x;
                    s[4 * i + 3] = hi2.y;
                }
                const float x0 = fmin3(s[0], s[1], s[2]), x1 = fmin3(s[3], s[4], s[5]), x2 = fmin3(s[6], s[7], s[8]),
                            x3 = fmin3(s[9], s[10], s[11]), x4 = fmin3(s[12], s[13], s[14]);
                const float gm = fminf(fmin3(x0, x1, x2), fmin3(x3, x4, s[15]));
                m2 = fminf(m2, fmaxf(m1, gm));
                if (gm < m1) r1 = cc;
                m1 = fminf(m1, gm);
            };
            // 32 clusters at a time; the next 32 scores are on their way
            // while these are compared
            auto load32 = [&](float (&x)[16], float (&y)[16], uint32_t cc) {
                w_ld16(taddr + cc, x);
                if (cc + 16 < kp) w_ld16(taddr + cc + 16, y);
            };
            auto wait32 = [&](float (&x)[16], float (&y)[16]) {
                w_ld_wait(x);
                w_ld_wait(y);
            };
            auto take32 = [&](float (&x)[16], float (&y)[16], uint32_t cc) {
                score(x, cc);
                if (cc + 16 < kp) {
                    score(y, cc + 16);
#pragma unroll
                    for (int i = 0; i < 16; ++i) col[i] = fmin3(col[i], x[i], y[i]);
                } else {
#pragma unroll
                    for (int i = 0; i < 16; ++i) col[i] = fminf(col[i], x[i]);
                }
            };
            if constexpr (EG == 4) {  // enough warps to hide the loads
#pragma unroll 1
                for (uint32_t cc = 0; cc < kp; cc += 32) {
                    load32(v0, v1, cc);
                    wait32(v0, v1);
                    take32(v0, v1, cc);
                }
            } else {
                float w0[16], w1[16];
                load32(v0, v1, 0);
                wait32(v0, v1);
#pragma unroll 1
                for (uint32_t cc = 0;; cc += 64) {
                    if (cc + 32 < kp) load32(w0, w1, cc + 32);
                    take32(v0, v1, cc);
                    if (cc + 32 >= kp) break;
                    wait32(w0, w1);
                    if (cc + 64 < kp) load32(v0, v1, cc + 64);
                    take32(w0, w1, cc + 32);
                    if (cc + 64 >= kp) break;
                    wait32(v0, v1);
                }
            }
            // columns as distances from the lowest score: the lowest column is
            // (nearly) zero and the index in its low bits costs no precision
#pragma unroll
            for (int i = 0; i < 16; i += 2) {
                const float2 e = sub2(make_float2(col[i], col[i + 1]), make_float2(m1, m1));
                col[i] = e.x;
                col[i + 1] = e.y;
            }
            float c1, c2;
            w_lowest2(col, c1, c2);
            uint32_t label = r1 + (__float_as_uint(c1) & 15u);
            const float gap = fminf(m2 - m1, c2);

            const uint64_t p = (uint64_t)t * WM + row;
            const bool in = p < n;
            float nx = 0.0f;
            for (uint32_t i = 0; i < nx_parts; ++i) nx += s_nx[slot * nx_parts + i][row];
            nx *= 1.0f + 0x1p-15f;
            const float aa = sqrtf(nx) * (1.0f + 0x1p-16f);
            const float h = fmaxf(m1 + nx, 0.0f);
            const float S = fmaf(ta * aa, aa, fmaf(t1, aa, fmaf(wc, h, t00)));
            const float T_ = (S + fmaf(rho, h + S, t0)) * (1.0f + 0x1p-10f);
            const bool fin = m1 < INF && aa < W_MAX_ABS && cm < W_MAX_ABS && aa + cm < rmax && T_ < INF;
            const bool proved = fin && gap > T_;
            allowed += W_UNPROVED_PER_TILE;
            const uint32_t open = __ballot_sync(0xffffffffu, in && !proved);
            if (open) {
                if (__popc(open) > allowed) {  // (this tile is labelled below, with the rest)
                    *abort_flag = 1u;
                    break;
                }
                allowed -= __popc(open);
                // candidates of the unproved points, exact distances, the
                // lexicographic (distance, index) minimum
                const float cut = m1 + T_;
                T best = TypeMax<T>::v();
                uint32_t bc = 0, tries = in && !proved && fin ? W_CANDIDATES : 0u;
                bool later = in && !proved && !fin;
                if (__any_sync(0xffffffffu, tries))
#pragma unroll 1
                    for (uint32_t cc = 0; cc < kp; cc += 16) {
                        w_ld16(taddr + cc, v0);
                        w_ld_wait(v0);
                        uint32_t mask = 0;
                        if (tries) {
#pragma unroll
                            for (int i = 0; i < 16; ++i)
                                if (cc + i < k && fmaf(-2.0f, v0[i], s_cn[cc + i]) <= cut) mask |= 1u << i;
                        }
                        while (mask) {
                            const uint32_t c = cc + __ffs(mask) - 1;
                            mask &= mask - 1;
                            if (--tries == 0u) {
                                later = true;
                                break;
                            }
                            const T dist = w_distance(a.points, n, p, a.centroids, k, c, d);
                            if (dist < best) {  // ascending clusters: the lowest index wins a tie
                                best = dist;
                                bc = c;
                            }
                        }
                        __syncwarp();
                    }
                if (!proved) label = later ? W_LATER : bc;
                if (later) s_later = 1u;
            }
            umma::fence_before_sync();
            __syncwarp();
            if (lane == 0) w_arrive(bar_empty);
            b += EG;
            if (b >= accs) {
                b = g;
                phase ^= 1u;
            }
            slot += EG;
            if (slot >= nx_slots) {
                slot -= nx_slots;
                nx_phase ^= 1u;
            }
            if (in) {
                a.labels[p] = (L)label;
                if (a.msum && label != W_LATER) atomicAdd(&s_mass[label], 1u);
            }
        }
        if (lane == 0) s_next[warp] = t;
    }

    umma::fence_before_sync();
    __syncthreads();
    if (warp == W_MMA_WARP) {
        __syncwarp();
        umma::fence_after_sync();
        umma::tmem_dealloc(tmem, accs * cols);
    }
    if (s_abort || s_later) {
        // The reference's labels by all clusters, with the centroids in the
        // operands' place if they fit.
        constexpr uint32_t WARPS = W_THREADS / 32;
        T* s_c = reinterpret_cast<T*>(smem_raw + (sB - umma::smem_u32(smem_raw)));
        const uint32_t padded = (k + 7u) & ~7u;
        const bool fits = (size_t)d * padded * sizeof(T) <= 2u * b_part + a.stages * a_bytes;
        if (fits)
            for (uint32_t i = tid; i < d * k; i += W_THREADS) s_c[i / k * padded + i % k] = __ldg(a.centroids + i);
        __syncthreads();
        const uint64_t step = (uint64_t)EG * gridDim.x;
        // points that the tile loop left for later, one by one
        if (s_later)
            for (uint32_t w = 0; w < W_EPI_WARPS; ++w)
                for (uint64_t t = blockIdx.x + (w >> 2) * (uint64_t)gridDim.x + warp * step; t < s_next[w]; t += WARPS * step) {
                    const uint64_t p = t * WM + (w & 3u) * 32u;
                    for (uint32_t left = __ballot_sync(0xffffffffu, p + lane < n && a.labels[p + lane] == (L)W_LATER); left;
                         left &= left - 1u) {
                        const uint32_t l = __ffs(left) - 1u;
                        const uint32_t label = fits ? w_by_all<T, true>(a.points, n, p + l, s_c, padded, k, d)
                                                    : w_by_all<T, false>(a.points, n, p + l, a.centroids, k, k, d);
                        if (lane == l) {
                            a.labels[p + l] = (L)label;
                            if (a.msum) atomicAdd(&s_mass[label], 1u);
                        }
                    }
                }
        // The tensor cores were given up, because too few points were proved or
        // because a wait ran out: the CTA's other points, a warp per 32.
        if (s_abort)
            for (uint32_t w = 0; w < W_EPI_WARPS; ++w)
                for (uint64_t t = s_next[w] + warp * step; t < a.tiles; t += WARPS * step) {
                    const uint64_t p = t * WM + (w & 3u) * 32u;
                    if (p >= n) continue;
                    const uint32_t label = fits ? w_exact32<T, true>(a.points, n, p, s_c, padded, k, d)
                                                : w_exact32<T, false>(a.points, n, p, a.centroids, k, k, d);
                    if (p + lane < n) {
                        a.labels[p + lane] = (L)label;
                        if (a.msum) atomicAdd(&s_mass[label], 1u);
                    }
                }
        __syncthreads();
    }
    if (a.msum)
        for (uint32_t c = tid; c < k; c += W_THREADS)
            if (s_mass[c]) atomicAdd(&a.msum[c], (unsigned long long)s_mass[c]);
}

// Dynamic shared memory of a shape: alignment, centroid halves, point stages.
size_t wide_smem(uint32_t dk, uint32_t kp, uint32_t stages) {
    const size_t kb = (dk + 63) / 64;
    return 1024 + 2 * kb * kp * 128 + (size_t)stages * 2 * kb * W_TILE_BYTES;
}

constexpr size_t W_STATIC = 30 * 1024;  // above the kernel's static shared memory

template <typename T, typename L, int EG, int ACCS>
int launch_wide_v(const WideArgs<T, L>& a, size_t smem, cudaStream_t s) {
    auto kern = wide_label_kernel<T, L, EG, ACCS>;
    const DeviceInfo& di = device_info();
    {
        static std::mutex mu;
        static bool done[64] = {false};
        int dev = 0;
        cudaGetDevice(&dev);
        std::lock_guard<std::mutex> lock(mu);
        if (dev < 0 || dev >= 64 || !done[dev]) {
            const cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                                       (int)(di.smem_optin - W_STATIC));
            if (e != cudaSuccess) return cuda_fail(e, "cudaFuncSetAttribute(wide)");
            if (dev >= 0 && dev < 64) done[dev] = true;
        }
    }
    const uint32_t grid = std::min<uint32_t>(a.tiles, (uint32_t)di.sm_count);
    kern<<<grid, w_threads(EG), smem, s>>>(a);
    count_launch();
    const cudaError_t e = cudaGetLastError();
    return e == cudaSuccess ? CKM_OK : cuda_fail(e, "wide label launch");
}

template <typename T, typename L>
int launch_wide_t(const T* points, const T* centroids, L* labels, unsigned long long* msum, uint64_t n, uint32_t d,
                  uint32_t k, cudaStream_t s) {
    const DeviceInfo& di = device_info();
    // CKM_WIDE_TEST_WAIT_NS (tests only): the limit of the waits, which run out
    // at 0, to check that the labels do not depend on them
    const char* wait = std::getenv("CKM_WIDE_TEST_WAIT_NS");
    WideArgs<T, L> a{points, centroids, labels, msum, wait ? std::strtoull(wait, nullptr, 10) : W_WAIT_NS, n, d, k,
                     0, 0, 0, 0, 0, 0, 0};
    a.dk = (d + 15) / 16 * 16;
    a.kp = (k + 15) / 16 * 16;
    a.kblocks = (a.dk + 63) / 64;
    // d <= 32: four stages filled by four teams of two warps (a warp's fixed
    // cost per tile spreads over more features than in larger teams: n = 2e6,
    // d = 20, k = 10 in 86 us, 118 with two teams, 177 with one); else one
    // team and two stages (n = 2^18, d = 100, k = 100: 50 us, 57 with two
    // teams), one where two do not fit
    const uint32_t chunks = (d + 7) / 8;
    a.stages = chunks <= 4 ? 4 : 2;
    a.teams = chunks <= 4 ? 4 : 1;
    while (a.stages > 1 && wide_smem(a.dk, a.kp, a.stages) + W_STATIC > di.smem_optin) a.stages >>= 1;
    a.teams = std::min(a.teams, a.stages);
    a.stages_log2 = a.stages == 4 ? 2 : a.stages - 1;
    a.tiles = (uint32_t)((n + WM - 1) / WM);
    const size_t smem = wide_smem(a.dk, a.kp, a.stages);
    if (a.kp > 128) return launch_wide_v<T, L, 2, 2>(a, smem, s);
    if (chunks <= 4) return launch_wide_v<T, L, 4, 4>(a, smem, s);
    return launch_wide_v<T, L, 2, 4>(a, smem, s);
}

}  // namespace

// The ends in d and k are those of the kernel's shared and tensor memory: at d =
// 129 or k = 257 the generic kernel takes over, some ten times slower. Nothing in
// the kernel needs the end in n; larger sets have not been run here.
bool wide_supported(uint64_t n, uint32_t d, uint32_t k) {
    const DeviceInfo& di = device_info();
    if (di.cc_major != 10 || n == 0 || n >= ((uint64_t)1 << 29) || d > W_MAX_D || k < 2 || k > W_MAX_K) return false;
    return wide_smem((d + 15) / 16 * 16, (k + 15) / 16 * 16, 1) + W_STATIC <= di.smem_optin;
}

// Where the lines lie: the other kernel against this one, us (fused: with the
// sums pass). A tile of this kernel costs most of its time whatever k and d
// are, so it wins where k*d is large, and labels alone also want enough tiles
// to pay for its set-up of 3 to 4 us.
//   low-d kernel (fused):    n = 5000 d = 8 k = 64 27 / 19, n = 10^5 level, n = 2^20 64 /
//                            72, k = 80 level, k = 100 1.45 times the speed; n =
//                            1.1e6 d = 16 k = 40 84 / 75, d = 12 k = 45 73 / 82
//                (labels):   d = 8 k = 64 n = 5e4 7.1 / 10.5, n = 10^6 38 / 37;
//                            d = 16 k = 32 n = 5e4 5.0 / 6.7, n = 5e5 21 / 19;
//                            d = 16 k = 64 n = 5000 7.5 / 6.6, d = 8 k = 128 n =
//                            5e4 12 / 15; at n = 2^20 d = 16 k = 16 25 / 33, d = 4
//                            k = 128 51 / 74
//   rows kernel (fused):     d = 32 k = 20 n = 5000 24 / 19; at n = 2^20 d = 32
//                            k = 16 90 / 97, d = 64 k = 16 151 / 140
//               (labels):    d = 32 k = 20 n = 10^5 9.5 / 11, d = 64 k = 10 n = 3e5
//                            21 / 23; d = 32 k = 64 n = 5000 5.8 / 8.2, n = 20000
//                            8.5 / 8.3, n = 3e5 38 / 19
//   generic kernel (fused):  n = 5000 d = 10 k = 4 18 / 14, d = 40 k = 3 47 / 15; d = 10 n
//                            = 20000 0.75 to 0.9 times the speed for k = 8 to 24, 1.1
//                            for k = 32; n = 10^5 0.9 for k = 8 to 16, n = 4e5 above 1
//                            (its shared atomics meet most in two or three rows)
//               (labels):    d = 20 k = 20 n = 5000 10.3 / 7.1, d = 33 k = 10 8.2 /
//                            7.0; d = 20 k = 10 n = 5000 6.0 / 7.1, n = 3e5 23 / 17;
//                            at n = 2^20 d = 17 k = 8 49 / 47, d = 28 k = 4 43 / 52, d
//                            = 33 k = 5 58 / 65, d = 48 k = 5 81 / 63, k = 3 56 / 63; d = 80
//                            k = 5 n = 10^5 0.9, n = 4e5 1.3, k = 2 n = 4e5 0.7
bool wide_pays_f32(uint64_t n, uint32_t d, uint32_t k, bool fused) {
    const uint64_t kd = (uint64_t)k * d;
    if (lowd_supported(d, k)) {
        // (a second chunk of four features costs like one of eight)
        const uint64_t from = d == 12 || (d == 8 && n >= 65536) ? 640 : 512;
        return (fused || n >= (1u << 19)) ? d >= 8 && kd >= from : d >= 12 && kd >= 1024;
    }
    if ((d == 32 || d == 64) && rows_supported(d, k)) return fused ? kd >= 640 : kd >= 1024 && n >= 16384;
    if (fused) return d >= 16 || k <= 4 || kd >= 300 || n >= (1u << 18);
    if (k >= 8) return kd >= 330 || (kd >= 136 && n * kd >= (1u << 25));
    return k >= 4 && (kd >= 480 || (kd >= 176 && n * kd >= (1u << 26)));
}
// FP64 (the generic kernel against this one; d <= 16 mostly goes to
// ckm_lowd64.cu): its FP64 distances grow with k*d, so few of them want many points.
//   labels: d = 16 k = 50 n = 2500 117 / 13; d = 24 k = 10 n = 10^4 36 / 15; d = 32
//           k = 2 n = 10^4 11 / 18; n = 6e5 d = 8 k = 8 160 / 33, d = 2 k = 8 49 / 33
//   fused:  d = 8 k = 12 n = 10^4 29 / 23; n = 10^5 d = 2 k = 8 24 / 23, n = 1.8e5
//           d = 10 k = 2 143 / 38
bool wide_pays_f64(uint64_t n, uint32_t d, uint32_t k, bool fused) {
    const uint64_t kd = (uint64_t)k * d;
    if (fused) return kd >= 96 || n >= 98304;
    return n >= 65536 ? kd >= 32 || n >= (1u << 18) : kd >= 64 && k >= 4;
}

int launch_wide_f32(const FusedF32& a, bool count, cudaStream_t s) {
    return launch_wide_t<float, uint32_t>(a.points, a.centroids, a.labels, count ? a.scratch.masses : nullptr,
                                          a.n, a.d, a.k, s);
}

int launch_wide_f64(const FusedF64& a, bool count, cudaStream_t s) {
    return launch_wide_t<double, uint64_t>(a.points, a.centroids, a.labels, count ? a.scratch.masses : nullptr,
                                           a.n, a.d, a.k, s);
}

}  // namespace ckm
