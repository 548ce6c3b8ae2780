// Kernels over the edges of a neighbour table that the backward ops and PushKnn have in common.
#pragma once
#include "common.cuh"

namespace hgc {

enum EdgeSum {
    kSumPlain,    // x[i,f] * w[e]
    kSumMean,     // (x[i,f] / K) * w[e]
    kSumMeanMax   // the same plus, where the target is the maximum of (i, f), x[i,F+f] * w[e]
};

// out[m,f] = sum over the edges e = (i, slot) that point at m, in ascending order.  One warp per target, lanes over
// a slab of up to 32 * FPL features starting at f0.  Every lane fetches one edge with its weight and flags, then
// the warp walks the 32 edges, the rows of 8 of them in flight.  The terms are added one by one, in edge
// order.  Which features of a source have the target as their maximum comes as bits (arg_flags_kernel): reading
// the arg-max row of every edge instead doubled the gathered bytes.
// 12.8 M edges, F = 64, hits in the search's order: 0.91 ms.  Half of the gathered lines miss L1, and the registers of 8 rows
// in flight leave 24 warps per SM to hide that; 60 % of the issue slots.
// POW2: K is a power of two, so that the division is an exact scaling.
template <int FPL, int MODE, bool POW2>
__global__ void __launch_bounds__(256)
edge_sum_kernel(const float *__restrict__ x, int ldx, const float *__restrict__ weights,
                const unsigned *__restrict__ flags, const int *__restrict__ nidx, const int *__restrict__ bounds,
                const int *__restrict__ edges, float *__restrict__ out, int n_vert, int K, int F, int f0,
                const int *__restrict__ order)
{
    pdl_begin();
    constexpr int U = 8;
    const int lane = threadIdx.x & 31;
    const int slot = blockIdx.x * 8 + (threadIdx.x >> 5);
    if (slot >= n_vert) return;
    const int m = order ? order[slot] : slot;  // processing order only: every target is visited once
    const int begin = bounds[m], end = bounds[m + 1];
    const float kf = (float)K, inv = 1.f / kf;
    float acc[FPL];
    bool mine[FPL];
#pragma unroll
    for (int u = 0; u < FPL; u++) {
        acc[u] = 0.f;
        mine[u] = f0 + u * 32 + lane < F;
    }
    const float *__restrict__ xl = x + f0 + lane;
    for (int p = begin; p < end; p += 32) {
        const int e = p + lane < end ? edges[p + lane] : 0;
        const int my_i = e / K;
        float my_w = 0.f;
        unsigned my_flag[FPL];
#pragma unroll
        for (int u = 0; u < FPL; u++) my_flag[u] = 0u;
        if (p + lane < end) {
            my_w = weights[e];
            if (MODE == kSumMeanMax) {
                bool counts = true;
                if (my_i == m) {
                    // the hit is its own neighbour: only its first occurrence in the row counts for the maximum
                    for (int k = e - my_i * K - 1; k >= 0; k--) counts = counts && nidx[(size_t)my_i * K + k] != m;
                }
                if (counts) {
                    const uint2 b = *reinterpret_cast<const uint2 *>(flags + 2 * (size_t)e);
                    my_flag[0] = b.x;
                    if (FPL > 1) my_flag[FPL - 1] = b.y;
                }
            }
        }
        const int n_here = min(32, end - p);
        for (int q0 = 0; q0 < n_here; q0 += U) {
            float g[U][FPL], h[U][FPL], w[U];
#pragma unroll
            for (int q = 0; q < U; q++) {
                // beyond the last edge: i = 0 with weight 0, not added below
                const int i = __shfl_sync(0xffffffffu, my_i, (q0 + q) & 31);
                w[q] = __shfl_sync(0xffffffffu, my_w, (q0 + q) & 31);
                const float *row = xl + (size_t)i * ldx;
#pragma unroll
                for (int u = 0; u < FPL; u++) {
                    g[q][u] = mine[u] ? __ldg(row + u * 32) : 0.f;
                    h[q][u] = 0.f;
                    if (MODE == kSumMeanMax) {
                        const unsigned b = __shfl_sync(0xffffffffu, my_flag[u], (q0 + q) & 31);
                        if ((b >> lane) & 1u) h[q][u] = __ldg(row + F + u * 32);
                    }
                }
            }
#pragma unroll
            for (int q = 0; q < U; q++) {
                if (q0 + q >= n_here) break;  // uniform
#pragma unroll
                for (int u = 0; u < FPL; u++) {
                    float t = MODE == kSumPlain ? g[q][u] : POW2 ? __fmul_rn(g[q][u], inv) : __fdiv_rn(g[q][u], kf);
                    t = __fmul_rn(t, w[q]);
                    if (MODE == kSumMeanMax && h[q][u] != 0.f) t = __fadd_rn(t, __fmul_rn(h[q][u], w[q]));
                    acc[u] = __fadd_rn(acc[u], t);
                }
            }
        }
    }
#pragma unroll
    for (int u = 0; u < FPL; u++)
        if (mine[u]) out[(size_t)m * F + f0 + u * 32 + lane] = acc[u];
}

// flags[e][2]: for every edge e = (i, slot) with target m, the features f0 .. f0 + 63 of hit i whose arg-max is m.
// One warp per hit; the two words of an edge are ballots over the lanes' arg-max entries.
static __global__ void __launch_bounds__(256)
arg_flags_kernel(const int *__restrict__ arg, const int *__restrict__ nidx, unsigned *__restrict__ flags, int n_vert,
                 int K, int F, int f0)
{
    pdl_begin();
    const int lane = threadIdx.x & 31;
    const int i = blockIdx.x * 8 + (threadIdx.x >> 5);
    if (i >= n_vert) return;
    constexpr int kNone = (int)0x80000000;  // not a hit
    const int a0 = f0 + lane < F ? arg[(size_t)i * F + f0 + lane] : kNone;
    const int a1 = f0 + 32 + lane < F ? arg[(size_t)i * F + f0 + 32 + lane] : kNone;
    for (int k0 = 0; k0 < K; k0 += 32) {
        int my_m = k0 + lane < K ? nidx[(size_t)i * K + k0 + lane] : -1;
        if (my_m < 0) my_m = kNone + 1;
        uint2 mine = make_uint2(0u, 0u);
#pragma unroll 8
        for (int q = 0; q < 32; q++) {
            if (k0 + q >= K) break;  // uniform
            const int m = __shfl_sync(0xffffffffu, my_m, q);
            const unsigned b0 = __ballot_sync(0xffffffffu, a0 == m), b1 = __ballot_sync(0xffffffffu, a1 == m);
            if (lane == q) mine = make_uint2(b0, b1);
        }
        if (k0 + lane < K) *reinterpret_cast<uint2 *>(flags + 2 * ((size_t)i * K + k0 + lane)) = mine;
    }
}

// out[i,k] = scale * sum over f, in order, of own[i,f] * x[m,f] for the neighbour m in slot k of hit i, plus (MAX) the
// same sum of own[i,F+f] * x[m,f] over the features whose arg-max is m.  One lane per (hit, slot), whose sum runs
// through the features one by one; the rows of the warp's 32 neighbours are read coalesced, 32 features at
// a time, into shared memory, from where every lane reads its own (rows 36 floats apart: no bank conflicts).
// A lane reading its row from global memory directly touched 32 lines with every load.
// 12.8 M edges, F = 64: 0.84 ms, bound by issue (80 % of the slots) and the L1 data stage (79 %): 32 loads, shuffles and
// shared-memory stores per warp and 32 features.
// MAX also writes the edge's bits for edge_sum_kernel (features 0 .. 63), which it compares for anyway.
template <bool GRAD, bool MAX>
__global__ void __launch_bounds__(256)
edge_dot_kernel(const float *__restrict__ own, int ld_own, const float *__restrict__ x, const int *__restrict__ arg,
                const int *__restrict__ nidx, float *__restrict__ out, long long n_edges, int n_vert, int K, int F,
                bool vec4, const int *__restrict__ order, unsigned *__restrict__ flags)
{
    pdl_begin();
    constexpr int kRow = 36;
    __shared__ __align__(16) float s_x[8][32 * kRow];
    const int lane = threadIdx.x & 31;
    float *__restrict__ s = s_x[threadIdx.x >> 5];
    const long long t0 = (long long)blockIdx.x * 256 + (threadIdx.x & ~31);
    if (t0 >= n_edges) return;
    const long long t = t0 + lane;
    int i = 0, m = -1;
    long long e = 0;
    if (t < n_edges) {
        const int row = (int)(t / K);
        i = order ? order[row] : row;  // processing order only
        e = (long long)i * K + (t - (long long)row * K);
        m = nidx[e];
        if (m >= n_vert) m = -1;
    }
    const float *__restrict__ g = own + (size_t)i * ld_own;
    const int *__restrict__ am = MAX ? arg + (size_t)i * F : nullptr;
    float mean_part = 0.f, max_part = 0.f;
    uint2 bits = make_uint2(0u, 0u);
    for (int f0 = 0; f0 < F; f0 += 32) {
        unsigned hit = 0u;
        __syncwarp();
        const bool in = f0 + lane < F;
#pragma unroll 8
        for (int q = 0; q < 32; q++) {
            const int mq = __shfl_sync(0xffffffffu, m, q);
            s[q * kRow + lane] = in && mq >= 0 ? __ldg(x + (size_t)mq * F + f0 + lane) : 0.f;
        }
        __syncwarp();
#pragma unroll
        for (int c = 0; c < 32; c += 4) {
            if (f0 + c >= F) break;  // uniform
            const float4 xv = *reinterpret_cast<const float4 *>(s + lane * kRow + c);
            float4 gv = make_float4(0.f, 0.f, 0.f, 0.f);
            int4 av = make_int4(-1, -1, -1, -1);
            const int left = F - f0 - c;
            if (vec4) {
                gv = __ldg(reinterpret_cast<const float4 *>(g + f0 + c));
                if (MAX) av = __ldg(reinterpret_cast<const int4 *>(am + f0 + c));
            } else {
                gv.x = g[f0 + c];
                if (left > 1) gv.y = g[f0 + c + 1];
                if (left > 2) gv.z = g[f0 + c + 2];
                if (left > 3) gv.w = g[f0 + c + 3];
                if (MAX) {
                    av.x = am[f0 + c];
                    if (left > 1) av.y = am[f0 + c + 1];
                    if (left > 2) av.z = am[f0 + c + 2];
                    if (left > 3) av.w = am[f0 + c + 3];
                }
            }
            // features beyond the last are zeros on both sides and change nothing
            mean_part = __fadd_rn(mean_part, __fmul_rn(gv.x, xv.x));
            mean_part = __fadd_rn(mean_part, __fmul_rn(gv.y, xv.y));
            mean_part = __fadd_rn(mean_part, __fmul_rn(gv.z, xv.z));
            mean_part = __fadd_rn(mean_part, __fmul_rn(gv.w, xv.w));
            if (MAX && m >= 0) {
                const float *h = g + F + f0 + c;
                hit |= (av.x == m ? 1u : 0u) << c | (av.y == m ? 2u : 0u) << c | (av.z == m ? 4u : 0u) << c | (av.w == m ? 8u : 0u) << c;
                if (av.x == m) max_part = __fadd_rn(max_part, __fmul_rn(h[0], xv.x));
                if (av.y == m) max_part = __fadd_rn(max_part, __fmul_rn(h[1], xv.y));
                if (av.z == m) max_part = __fadd_rn(max_part, __fmul_rn(h[2], xv.z));
                if (av.w == m) max_part = __fadd_rn(max_part, __fmul_rn(h[3], xv.w));
            }
        }
        if (f0 == 0) bits.x = hit;
        if (f0 == 32) bits.y = hit;
    }
    if (t >= n_edges) return;
    if (MAX && flags) *reinterpret_cast<uint2 *>(flags + 2 * (size_t)e) = bits;
    if (m < 0) {
        out[e] = 0.f;
    } else if (GRAD) {
        // the reference scales by the double 1./(float)K
        out[e] = __fadd_rn((float)__dmul_rn((double)mean_part, 1.0 / (double)(float)K), max_part);
    } else {
        out[e] = mean_part;
    }
}

// Features per lane and division mode of edge_sum_kernel; slabs of 64 features.
template <int MODE>
int launch_edge_sum_slab(const float *x, int ldx, const float *weights, const unsigned *flags, const int *nidx,
                         const int *bounds, const int *edges, float *out, int n_vert, int K, int F, int f0,
                         const int *order, cudaStream_t stream)
{
    const int blocks = div_up(n_vert, 8);
#define HGC_SUM(FPL, P) HGC_CUDA_TRY(launch_overlapped(n_vert, edge_sum_kernel<FPL, MODE, P>, blocks, 256, 0, stream, x, ldx, weights, flags, nidx, bounds, edges, out, n_vert, K, F, f0, order))
    const bool pow2 = MODE == kSumPlain || (K & (K - 1)) == 0;
    if (F - f0 <= 32) { if (pow2) HGC_SUM(1, true); else HGC_SUM(1, false); }
    else              { if (pow2) HGC_SUM(2, true); else HGC_SUM(2, false); }
#undef HGC_SUM
    HGC_LAUNCH_CHECK();
    return HGC_OK;
}

}  // namespace hgc
