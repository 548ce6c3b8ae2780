// Device helpers of the neighbour searches: (distance, index) keys, warp-wide sorting networks, point and
// box distances.
#pragma once
#include "common.cuh"

namespace hgc {

// A candidate is one 64-bit word: squared-distance bits in the high half, hit index in the low
// half, so that ordering the words orders by (distance, index).  The word is held as a double:
// for non-negative floats in the high half the IEEE-754 order of the doubles equals the order of
// the 64-bit integers (distances are never NaN), and a 64-bit comparison then is one FP64
// instruction instead of a chain of integer compares on the (half-rate, saturated) integer pipe.
typedef double knn_key;
#define HGC_KNN_INF_KEY 1.7976931348623157e308  /* DBL_MAX: above every real key, even distance = +inf */

__device__ __forceinline__ knn_key make_key(float distsq, int j)
{
    return __hiloint2double((int)__float_as_uint(distsq), j);
}
__device__ __forceinline__ float key_distsq(knn_key k) { return __int_as_float(__double2hiint(k)); }
__device__ __forceinline__ int key_index(knn_key k) { return __double2loint(k); }

__device__ __forceinline__ knn_key shfl_key(knn_key v, int src) { return __shfl_sync(0xffffffffu, v, src); }
__device__ __forceinline__ knn_key shfl_xor_key(knn_key v, int m) { return __shfl_xor_sync(0xffffffffu, v, m); }

// Keeps the smaller of (v, o) when `lower`, else the larger.
__device__ __forceinline__ knn_key cmp_exchange(knn_key v, knn_key o, bool lower)
{
    return ((v < o) == lower) ? v : o;
}

// Smallest / largest float of the warp (NaN operands are ignored).
__device__ __forceinline__ float warp_min_f32(float v)
{
    float r;
    asm("redux.sync.min.f32 %0, %1, 0xffffffff;" : "=f"(r) : "f"(v));
    return r;
}
__device__ __forceinline__ float warp_max_f32(float v)
{
    float r;
    asm("redux.sync.max.f32 %0, %1, 0xffffffff;" : "=f"(r) : "f"(v));
    return r;
}

// Ascending bitonic sort of one key per lane.  Each merge starts with the mirrored partner, so
// every step is "the lower lane keeps the smaller key" and only five lane-bit tests are needed.
__device__ __forceinline__ knn_key warp_sort(knn_key v, int lane)
{
#pragma unroll
    for (int k = 2; k <= 32; k <<= 1) {
        v = cmp_exchange(v, shfl_xor_key(v, k - 1), (lane & (k >> 1)) == 0);
#pragma unroll
        for (int j = k >> 2; j > 0; j >>= 1) v = cmp_exchange(v, shfl_xor_key(v, j), (lane & j) == 0);
    }
    return v;
}

// Ascending sort of one 32-bit word per lane (same network).
__device__ __forceinline__ unsigned warp_sort_u32(unsigned v, int lane)
{
#pragma unroll
    for (int k = 2; k <= 32; k <<= 1) {
        unsigned o = __shfl_xor_sync(0xffffffffu, v, k - 1);
        v = ((lane & (k >> 1)) == 0) ? min(v, o) : max(v, o);
#pragma unroll
        for (int j = k >> 2; j > 0; j >>= 1) {
            o = __shfl_xor_sync(0xffffffffu, v, j);
            v = ((lane & j) == 0) ? min(v, o) : max(v, o);
        }
    }
    return v;
}

__device__ __forceinline__ unsigned warp_bitonic_merge_u32(unsigned v, int lane)
{
#pragma unroll
    for (int j = 16; j > 0; j >>= 1) {
        const unsigned o = __shfl_xor_sync(0xffffffffu, v, j);
        v = ((lane & j) == 0) ? min(v, o) : max(v, o);
    }
    return v;
}

// Sorts a bitonic sequence (one key per lane) ascending.
__device__ __forceinline__ knn_key warp_bitonic_merge(knn_key v, int lane)
{
#pragma unroll
    for (int j = 16; j > 0; j >>= 1) v = cmp_exchange(v, shfl_xor_key(v, j), (lane & j) == 0);
    return v;
}

// Merges an ascending block `b` of 32 keys into the ascending striped list, keeping the smallest.
template <int L>
__device__ __forceinline__ void merge_into_list(knn_key (&list)[L], knn_key b, int lane)
{
#pragma unroll
    for (int r = 0; r < L; r++) {
        // a register whose largest key is not above b's smallest stays as it is
        const knn_key reg_max = shfl_key(list[r], 31);
        const knn_key b_min = shfl_key(b, 0);
        if (b_min >= reg_max) continue;
        const knn_key rev = shfl_xor_key(b, 31);
        const bool keep = list[r] < rev;
        const knn_key lo = keep ? list[r] : rev;
        const knn_key hi = keep ? rev : list[r];
        list[r] = warp_bitonic_merge(lo, lane);
        if (r + 1 < L) b = warp_bitonic_merge(hi, lane);
    }
}

// list[reg] for a runtime `reg`, without indexing the register array dynamically
template <int L>
__device__ __forceinline__ knn_key list_reg(const knn_key (&list)[L], int reg)
{
    knn_key v = list[0];
#pragma unroll
    for (int r = 1; r < L; r++)
        if (r == reg) v = list[r];
    return v;
}

// Merges two ascending runs of M registers each (striped: rank r in register r / 32 of lane r % 32) into
// one run of 2 M registers.
template <int M>
__device__ __forceinline__ void merge_runs(knn_key *a, int lane)
{
    // compare with the mirrored second run, smaller keys to the front: two bitonic halves
#pragma unroll
    for (int i = 0; i < M; i++) {
        const knn_key lo = a[i], hi = a[2 * M - 1 - i];
        const knn_key rev = shfl_xor_key(hi, 31), rlo = shfl_xor_key(lo, 31);
        a[i] = rev < lo ? rev : lo;
        a[2 * M - 1 - i] = rlo < hi ? hi : rlo;
    }
#pragma unroll
    for (int st = M / 2; st > 0; st >>= 1)
#pragma unroll
        for (int i = 0; i < 2 * M; i++)
            if ((i & st) == 0) {
                const knn_key lo = a[i], hi = a[i + st];
                const bool sw = hi < lo;
                a[i] = sw ? hi : lo;
                a[i + st] = sw ? lo : hi;
            }
#pragma unroll
    for (int i = 0; i < 2 * M; i++) a[i] = warp_bitonic_merge(a[i], lane);
}

// Ascending sort of 32 * L keys, striped over the lanes.
template <int L>
__device__ __forceinline__ void sort_striped(knn_key (&k)[L], int lane)
{
#pragma unroll
    for (int r = 0; r < L; r++) k[r] = warp_sort(k[r], lane);
    if (L >= 2) {
#pragma unroll
        for (int r = 0; r + 2 <= L; r += 2) merge_runs<1>(k + r, lane);
    }
    if (L >= 4) {
#pragma unroll
        for (int r = 0; r + 4 <= L; r += 4) merge_runs<2>(k + r, lane);
    }
    if (L >= 8) {
#pragma unroll
        for (int r = 0; r + 8 <= L; r += 8) merge_runs<4>(k + r, lane);
    }
    if (L >= 16) merge_runs<8>(k, lane);
}

template <int NV4>
struct Point {
    float4 v[NV4];
};

template <int NV4>
__device__ __forceinline__ Point<NV4> load_point(const float4 *__restrict__ pts, size_t i)
{
    Point<NV4> p;
#pragma unroll
    for (int u = 0; u < NV4; u++) p.v[u] = __ldg(pts + i * NV4 + u);
    return p;
}

// sum over coordinates of (a-b)^2, each operation rounded on its own, in coordinate order.  The
// zero padding of the last float4 adds +0 terms, which change nothing.
// Packed float32x2 subtract / multiply (two individually rounded float32 operations per instruction).
__device__ __forceinline__ float2 sub2(float ax, float ay, float bx, float by)
{
    float2 r;
    asm("{ .reg .b64 ra, rb, rr; mov.b64 ra, {%2,%3}; mov.b64 rb, {%4,%5}; sub.rn.f32x2 rr, ra, rb; "
        "mov.b64 {%0,%1}, rr; }"
        : "=f"(r.x), "=f"(r.y) : "f"(ax), "f"(ay), "f"(bx), "f"(by));
    return r;
}
__device__ __forceinline__ float2 sqr2(float2 a)
{
    float2 r;
    asm("{ .reg .b64 ra, rr; mov.b64 ra, {%2,%3}; mul.rn.f32x2 rr, ra, ra; mov.b64 {%0,%1}, rr; }"
        : "=f"(r.x), "=f"(r.y) : "f"(a.x), "f"(a.y));
    return r;
}

template <int NV4>
__device__ __forceinline__ float distsq(const Point<NV4> &a, const Point<NV4> &b)
{
    float s = 0.f;
#pragma unroll
    for (int u = 0; u < NV4; u++) {
        const float2 q01 = sqr2(sub2(a.v[u].x, a.v[u].y, b.v[u].x, b.v[u].y));
        const float2 q23 = sqr2(sub2(a.v[u].z, a.v[u].w, b.v[u].z, b.v[u].w));
        s = u == 0 ? q01.x : __fadd_rn(s, q01.x);  // 0 + square is the square
        s = __fadd_rn(s, q01.y);
        s = __fadd_rn(s, q23.x);
        s = __fadd_rn(s, q23.y);
    }
    return s;
}

// Squared distance from q to the box [lo, hi], with the operation sequence of distsq: a lower
// bound of the computed distance to any point inside the box.
__device__ __forceinline__ float gap1(float q, float lo, float hi)
{
    return fmaxf(fmaxf(__fsub_rn(lo, q), __fsub_rn(q, hi)), 0.f);
}
template <int NV4>
__device__ __forceinline__ float box_distsq(const Point<NV4> &q, const float4 *__restrict__ lo,
                                            const float4 *__restrict__ hi, size_t chunk)
{
    float s = 0.f;
#pragma unroll
    for (int u = 0; u < NV4; u++) {
        const float4 l = __ldg(lo + chunk * NV4 + u), h = __ldg(hi + chunk * NV4 + u);
        float g;
        g = gap1(q.v[u].x, l.x, h.x); s = __fadd_rn(s, __fmul_rn(g, g));
        g = gap1(q.v[u].y, l.y, h.y); s = __fadd_rn(s, __fmul_rn(g, g));
        g = gap1(q.v[u].z, l.z, h.z); s = __fadd_rn(s, __fmul_rn(g, g));
        g = gap1(q.v[u].w, l.w, h.w); s = __fadd_rn(s, __fmul_rn(g, g));
    }
    return s;
}

}  // namespace hgc
