// FP64 labels for d <= 16: an FP32 screen in front of the FP64 distances.
//
// FP64 arithmetic runs at two lanes per clock and SM here, so even the d
// conversions of a point on that pipe cost more than reading the point.  Each
// coordinate is cut by integer operations into two floats, x = xh + xl (24 and
// 23 bits), the centroids likewise once per CTA, and
//   t = (xh - ch) + (xl - cl),  s = sum of t^2
// is computed in FP32, two points at a time in packed operations.  The lowest
// two scores and the bound below prove the label for all but about one point
// in a million; the others get FP64 distances (the reference's: t = x - c, acc =
// fma(t, t, acc), f ascending, strict '<' from cluster 0) for the clusters that
// the screen cannot rule out.
//
// Bound.  With ax >= |x_f|, cm >= |c_f| and E = 2^-44 (ax + cm) + 2^-120: the split
// leaves out at most 2^-46 |x_f| (2^-126 at the lower end of the float range)
// and 2^-48 |c_f|, |xl - cl| <= 2^-23 (|x_f| + |c_f|), and the three FP32
// roundings give |t' - t| <= 1.01 2^-23 |t| + E.  Squared and summed by D fused
// multiply-adds,
//   |s - S| <= alpha S + 2.05 E sqrt(D S) + 1.01 D E^2,
//   alpha = 1.02 (1.03 2^-22 + 1.01 D 2^-24),
// and 2.05 E sqrt(D S) <= alpha S + 4.3e6 D E^2, so |s - S| <= 2 alpha S + kappa with
// kappa = 4.4e6 D E^2.  The reference's FP64 distance is S up to (D + 3) 2^-53.
// Hence a cluster with s > cut = m1 (1 + 4.5 alpha) + 2.2 kappa + 2^-120 (m1 the lowest
// score; the last term covers the squares' underflow) has a larger reference
// distance than the lowest one's cluster.  The proof wants m1 and cut finite;
// an infinite or NaN coordinate, or one beyond the float range, makes them not
// so.  A centroid that is not finite is never the nearest: its score is +inf.
//
// What bounds it: issue slots (66 % at d = 4, k = 16), of which the lowest two and
// the integer split take the ALU pipe to 52 %, the 4 d k packed operations per two
// points the FMA pipe to 29 %.  n = 2^20, d = 4, k = 16 18 us, with the 42 MB read
// and written 7 (the tensor-core labels 51, the generic kernel 278).
#include "ckm_device.cuh"
#include "ckm_internal.h"

#include <algorithm>
#include <cfloat>

namespace ckm {
namespace {

constexpr int L64_BLK = 256;
constexpr uint32_t L64_TILE = 2 * L64_BLK;  // two points per thread
constexpr size_t LOWD64_SMEM_LIMIT = 40 * 1024;  // (below 48 KB with the static part: no attribute needed)

constexpr int l64_ctas(int d) { return d <= 4 ? 4 : d <= 8 ? 3 : 2; }  // per SM, by registers

struct Lowd64Args {
    const double* points;
    const double* centroids;
    uint64_t* labels;
    unsigned long long* msum;  // counts are added here (nullptr: not counted)
    uint64_t n;
    uint32_t k;
    int vec, vec_labels;  // 16-byte loads and stores of two points
};

template <int D>
struct Lowd64Bound {
    static constexpr float alpha = 1.02f * (1.03f * 0x1p-22f + 1.01f * (float)D * 0x1p-24f);
    static constexpr float grow = 1.0f + 4.5f * alpha;
    static constexpr float kappa = 2.2f * 4.4e6f * (float)D;
};

// The label of point p by FP64 distances of the clusters with s <= cut (all of
// them where the screen proved nothing).
template <int D>
__device__ __noinline__ uint32_t exact_label64(const Lowd64Args a, const float4* s_c, uint64_t p, float cut) {
    double x[D];
    float xh[D], xl[D];
#pragma unroll
    for (int f = 0; f < D; ++f) {
        x[f] = __ldg(a.points + (uint64_t)f * a.n + p);
        split64(x[f], xh[f], xl[f]);
    }
    double best = DBL_MAX;
    uint32_t lab = 0;
    for (uint32_t c = 0; c < a.k; ++c) {
        float s = 0.0f;
#pragma unroll
        for (int f = 0; f < D; ++f) {
            const float4 m = s_c[c * D + f];
            const float t = (xh[f] + m.x) + (xl[f] + m.z);
            s = fmaf(t, t, s);
        }
        if (s > cut) continue;  // (not for a NaN)
        double acc = 0.0;
#pragma unroll
        for (int f = 0; f < D; ++f) {
            const double t = x[f] - __ldg(a.centroids + (uint64_t)f * a.k + c);
            acc = fma(t, t, acc);
        }
        if (acc < best) {
            best = acc;
            lab = c;
        }
    }
    return lab;
}

template <int D>
__global__ void __launch_bounds__(L64_BLK, l64_ctas(D)) lowd64_kernel(const Lowd64Args a, const uint64_t tiles) {
    extern __shared__ __align__(16) unsigned char smem[];
    __shared__ unsigned int s_cm;
    const uint32_t k = a.k;
    const uint64_t n = a.n;
    float4* s_c = reinterpret_cast<float4*>(smem);  // [c][f]: (-ch, -ch, -cl, -cl)
    unsigned int* s_mass = reinterpret_cast<unsigned int*>(s_c + (size_t)k * D);
    if (threadIdx.x == 0) s_cm = 0u;
    __syncthreads();
    for (uint32_t c = threadIdx.x; c < k; c += L64_BLK) {
        double v[D];
        bool finite = true;
#pragma unroll
        for (int f = 0; f < D; ++f) {
            v[f] = __ldg(a.centroids + (uint64_t)f * k + c);
            finite = finite && (__double2hiint(v[f]) & 0x7ff00000) != 0x7ff00000;
        }
        float cm = 0.0f;
#pragma unroll
        for (int f = 0; f < D; ++f) {
            const float h = finite ? (float)v[f] : __int_as_float(0x7f800000);
            const float l = isinf(h) ? 0.0f : (float)(v[f] - (double)h);
            s_c[c * D + f] = make_float4(-h, -h, -l, -l);
            cm = fmaxf(cm, fabsf(h));
        }
        if (finite) atomicMax(&s_cm, __float_as_uint(cm));
        s_mass[c] = 0u;
    }
    __syncthreads();
    const float cm = __uint_as_float(s_cm);
    const float INF = __int_as_float(0x7f800000);

    for (uint64_t tile = blockIdx.x; tile < tiles; tile += gridDim.x) {
        const uint64_t p = tile * L64_TILE + 2u * threadIdx.x;
        float2 xh[D], xl[D];
        float axa = 0.0f, axb = 0.0f;
        {
            double xa[D], xb[D];
#pragma unroll
            for (int f = 0; f < D; ++f) {
                const double* src = a.points + (uint64_t)f * n + p;
                if (a.vec && p + 1 < n) {
                    const double2 v = __ldg(reinterpret_cast<const double2*>(src));
                    xa[f] = v.x;
                    xb[f] = v.y;
                } else {
                    xa[f] = p < n ? __ldg(src) : 0.0;
                    xb[f] = p + 1 < n ? __ldg(src + 1) : 0.0;
                }
            }
#pragma unroll
            for (int f = 0; f < D; ++f) {
                split64(xa[f], xh[f].x, xl[f].x);
                split64(xb[f], xh[f].y, xl[f].y);
                axa = fmaxf(axa, fabsf(xh[f].x));
                axb = fmaxf(axb, fabsf(xh[f].y));
            }
        }
        float m1a = INF, m2a = INF, m1b = INF, m2b = INF;
        uint32_t ia = 0, ib = 0;
#pragma unroll 2
        for (uint32_t c = 0; c < k; ++c) {
            float2 s;
#pragma unroll
            for (int f = 0; f < D; ++f) {
                const float4 m = s_c[c * D + f];
                const float2 t = add2(add2(xh[f], make_float2(m.x, m.y)), add2(xl[f], make_float2(m.z, m.w)));
                s = f == 0 ? fma2(t, t, make_float2(0.0f, 0.0f)) : fma2(t, t, s);
            }
            m2a = fminf(m2a, fmaxf(m1a, s.x));
            m2b = fminf(m2b, fmaxf(m1b, s.y));
            if (s.x < m1a) { m1a = s.x; ia = c; }
            if (s.y < m1b) { m1b = s.y; ib = c; }
        }
        auto cut_of = [&](float m1, float ax) {
            const float e = fmaf(ax * 1.000001f + cm * 1.000001f, 0x1p-44f, 0x1p-120f);
            const float q = e * e * Lowd64Bound<D>::kappa + 0x1p-120f;
            const float cut = fmaf(m1, Lowd64Bound<D>::grow, q);
            return cut < 1e38f ? cut : INF;  // NaN and overflow: nothing ruled out
        };
        if (p < n) {
            // (a NaN score hides neither of the two: the point's own NaN leaves m1
            // infinite, a centroid's is replaced above)
            const float ca = cut_of(m1a, axa), cb = cut_of(m1b, axb);
            if (!(m2a > ca) || !(ca < INF)) ia = exact_label64<D>(a, s_c, p, ca);
            if (p + 1 < n && (!(m2b > cb) || !(cb < INF))) ib = exact_label64<D>(a, s_c, p + 1, cb);
            if (a.vec_labels && p + 1 < n) {
                *reinterpret_cast<ulonglong2*>(a.labels + p) = make_ulonglong2(ia, ib);
            } else {
                a.labels[p] = ia;
                if (p + 1 < n) a.labels[p + 1] = ib;
            }
            if (a.msum) {
                atomicAdd(&s_mass[ia], 1u);
                if (p + 1 < n) atomicAdd(&s_mass[ib], 1u);
            }
        }
    }
    if (a.msum) {
        __syncthreads();
        for (uint32_t c = threadIdx.x; c < k; c += L64_BLK)
            if (s_mass[c]) atomicAdd(&a.msum[c], (unsigned long long)s_mass[c]);
    }
}

size_t lowd64_smem(uint32_t d, uint32_t k) { return (size_t)k * (d * sizeof(float4) + sizeof(unsigned int)); }

template <int D>
int launch_lowd64_d(const Lowd64Args& a, cudaStream_t s) {
    const uint64_t tiles = (a.n + L64_TILE - 1) / L64_TILE;
    const uint64_t grid = std::min<uint64_t>(tiles, (uint64_t)device_info().sm_count * l64_ctas(D));
    lowd64_kernel<D><<<(unsigned)grid, L64_BLK, lowd64_smem(D, a.k), s>>>(a, tiles);
    count_launch();
    const cudaError_t e = cudaGetLastError();
    return e == cudaSuccess ? CKM_OK : cuda_fail(e, "lowd64 launch");
}

}  // namespace

// Its time grows with k (4 d + 9), that of the tensor-core labels hardly (51 us for
// 2^20 points of d <= 8, 70 for d <= 16; 9 to 12 for few): n = 2^20 d = 4 k = 16
// (units 400) 18 us, d = 8 k = 32 (1312) 56, d = 4 k = 100 (2500) 77, d = 2 k = 200
// (3400) 109; d = 10 k = 20 (980) 46, d = 16 k = 17 (1241) 66, k = 22 (1606) 80; n = 5000
// d = 8 k = 32 7.2 against 9, d = 8 k = 100 (4100) 14 against 11.5, d = 12 k = 30 (1710)
// 8.7 against 11, n = 2000 d = 4 k = 60 6.3 against 13.  The generic kernel is slower
// everywhere (n = 1000 d = 1 k = 4 2.1 against 2.8, n = 2^20 d = 3 k = 3 8.5 against
// 43), so what the tensor-core labels do not take comes here too as far as the
// centroids fit.
bool lowd64_pays(uint64_t n, uint32_t d, uint32_t k) {
    if (n == 0 || d < 1 || d > 16 || k < 1 || lowd64_smem(d, k) > LOWD64_SMEM_LIMIT) return false;
    return (uint64_t)k * (4 * d + 9) <= (n < 32768 ? 2600 : 1300) || !wide_supported(n, d, k);
}

int launch_lowd64(const FusedF64& a, bool count, cudaStream_t s) {
    Lowd64Args g{a.points, a.centroids, a.labels, count ? a.scratch.masses : nullptr, a.n, a.k, 0, 0};
    g.vec = a.n % 2 == 0 && reinterpret_cast<uintptr_t>(a.points) % 16 == 0;
    g.vec_labels = reinterpret_cast<uintptr_t>(a.labels) % 16 == 0;
    switch (a.d) {
        case 1: return launch_lowd64_d<1>(g, s);
        case 2: return launch_lowd64_d<2>(g, s);
        case 3: return launch_lowd64_d<3>(g, s);
        case 4: return launch_lowd64_d<4>(g, s);
        case 5: return launch_lowd64_d<5>(g, s);
        case 6: return launch_lowd64_d<6>(g, s);
        case 7: return launch_lowd64_d<7>(g, s);
        case 8: return launch_lowd64_d<8>(g, s);
        case 9: return launch_lowd64_d<9>(g, s);
        case 10: return launch_lowd64_d<10>(g, s);
        case 11: return launch_lowd64_d<11>(g, s);
        case 12: return launch_lowd64_d<12>(g, s);
        case 13: return launch_lowd64_d<13>(g, s);
        case 14: return launch_lowd64_d<14>(g, s);
        case 15: return launch_lowd64_d<15>(g, s);
        case 16: return launch_lowd64_d<16>(g, s);
        default: return fail(CKM_ERR_UNSUPPORTED, "lowd64: unsupported feature count");
    }
}

}  // namespace ckm
