// Kernels over the edges of a neighbour table that the backward ops and PushKnn have in common.
#pragma once
#include <type_traits>

#include "common.cuh"
#include "incoming.cuh"

namespace hgc {

// (ax * bx, ay * by), rounded one by one.  Sums stay with __fadd_rn: ptxas contracts a packed addition of a packed product
// to a fused one although both ask for rounding.
__device__ __forceinline__ float2 mul2(float ax, float ay, float bx, float by)
{
    float2 r;
    asm("{ .reg .b64 ra, rb, rr; mov.b64 ra, {%2,%3}; mov.b64 rb, {%4,%5}; mul.rn.f32x2 rr, ra, rb; mov.b64 {%0,%1}, rr; }"
        : "=f"(r.x), "=f"(r.y) : "f"(ax), "f"(ay), "f"(bx), "f"(by));
    return r;
}
enum EdgeSum {
    kSumPlain,    // x[i,f] * w[e]
    kSumMean,     // (x[i,f] / K) * w[e]
    kSumMeanMax   // the same plus, where the target is the maximum of (i, f), x[i,F+f] * w[e]
};

constexpr int VW = 4;  // features per lane of edge_sum_kernel
struct EdgeVec { float v[VW]; };
__device__ __forceinline__ EdgeVec load_edge_vec(const float *p)
{
    const float4 q = __ldg(reinterpret_cast<const float4 *>(p));
    return {{q.x, q.y, q.z, q.w}};
}

// The same if any bit of `wanted` is set; otherwise, and (not WHOLE) in places whose bit is not set, the values do not count.
template <bool WHOLE>
__device__ __forceinline__ EdgeVec load_edge_vec_if(const float *p, unsigned wanted)
{
    EdgeVec r = {{0.f, 0.f, 0.f, 0.f}};
    if constexpr (WHOLE) {
        asm volatile("{ .reg .pred q; setp.ne.u32 q, %5, 0; @q ld.global.nc.v4.f32 {%0,%1,%2,%3}, [%4]; }"
                     : "+f"(r.v[0]), "+f"(r.v[1]), "+f"(r.v[2]), "+f"(r.v[3]) : "l"(p), "r"(wanted));
    } else {
#pragma unroll
        for (int v = 0; v < VW; v++)
            if ((wanted >> v) & 1u) r.v[v] = __ldg(p + v);
    }
    return r;
}

// Source, weight and (kSumMeanMax) the two words of flags of an edge that points at m.
template <int MODE>
__device__ __forceinline__ uint4 edge_record(int e, int m, int K, const float *__restrict__ weights,
                                             const unsigned *__restrict__ flags, const int *__restrict__ nidx)
{
    const int i = e / K;
    uint4 ed = make_uint4((unsigned)i, __float_as_uint(weights[e]), 0u, 0u);
    if (MODE == kSumMeanMax) {
        bool counts = true;
        if (i == m) {
            // the hit is its own neighbour: only its first occurrence in the row counts for the maximum
            for (int k = e - i * K - 1; k >= 0; k--) counts = counts && nidx[(size_t)i * K + k] != m;
        }
        if (counts) {
            const uint2 b = *reinterpret_cast<const uint2 *>(flags + 2 * (size_t)e);
            ed.z = b.x;
            ed.w = b.y;
        }
    }
    return ed;
}

// What an edge adds to VW features: g, times 1 / K where SCALE, and h where a bit of b is set, both times the weight.
template <int MODE, bool SCALE>
__device__ __forceinline__ EdgeVec edge_terms(const EdgeVec &g, const EdgeVec &h, float w, unsigned b, float inv)
{
    EdgeVec t;
#pragma unroll
    for (int v = 0; v < VW; v += 2) {
        float2 r = make_float2(g.v[v], g.v[v + 1]);
        if (SCALE) r = mul2(r.x, r.y, inv, inv);
        r = mul2(r.x, r.y, w, w);
        t.v[v] = r.x;
        t.v[v + 1] = r.y;
        if (MODE == kSumMeanMax) {
            r = mul2(h.v[v], h.v[v + 1], w, w);
            if (b & (1u << v)) t.v[v] = __fadd_rn(t.v[v], r.x);
            if (b & (2u << v)) t.v[v + 1] = __fadd_rn(t.v[v + 1], r.y);
        }
    }
    return t;
}

// out[m,f] = sum over the edges e = (i, slot) that point at m, in ascending order, for the features f0 .. f0 + LPT * VW - 1.
// LPT lanes work on one target, VW neighbouring features each; a warp has 32 / LPT targets.  Every lane fetches one edge with
// its weight and flags and puts them into shared memory, from where all lanes read them with one broadcast load per edge
// (four shuffles before); the rows of two edges are in flight.  The terms are added one by one, in edge order.
// Rows lie `ldr` floats apart in `rows`, whole vectors in every row; SCALE multiplies them with 1 / K.  In the mode kSumMeanMax
// `maxima` (rows `ldm` floats apart, HVEC: whole vectors) holds what goes to the maximum alone.  Which features of a source
// have the target as their maximum comes as bits (arg_flags_kernel): reading the arg-max row of every edge instead doubled
// the gathered bytes.
// 12.8 M edges, F = 64, hits in the search's order: 0.55 ms; a warp per target with 4-byte loads and 8 rows in flight took
// 0.91, its 77 registers leaving 24 warps per SM.  Half of the gathered lines miss L1 and resident warps hide that better than
// rows in flight: 16 lanes x 4 features with 2 rows and 40 warps per SM beat 4 rows (+1 %), 8 rows (+20 %), a warp x 2 features
// (+10 %), and 64 warps, which spill (+27 %).  PushKnn, 200k hits, K = 40, F = 32: 433 -> 341 us.
// Wide lists (wide_list) are worked on by whole blocks, before their other targets: every LPT lanes fetch rows of their own, two
// at a time, whose terms go through shared memory to one thread per feature that adds them in edge order.  The other targets of a
// block are dealt out again, those without edges last, so that warps are whole where most hits are nobody's neighbours.
// us with every target in a group of lanes of its own / so, 200k hits, K = F = 64, one hit in 100 a neighbour: PushKnn 3075 / 1417,
// gradient of the accumulation 5078 / 2450; one neighbour of all hits: 56500 / 9060, 81600 / 17300; searched tables as before.
// R: rows in flight per target, eight where the targets are too few to fill the chip (gradient on 2000 hits, K = 16 27.7 / 25.1).
template <int LPT, int R, int MODE, bool SCALE, bool HVEC>
__global__ void __launch_bounds__(256, R == 2 ? 5 : 2)
edge_sum_kernel(const float *__restrict__ rows, int ldr, const float *__restrict__ maxima, int ldm,
                const float *__restrict__ weights, const unsigned *__restrict__ flags, const int *__restrict__ nidx,
                const int *__restrict__ bounds, const int *__restrict__ edges, WideLists wide, float *__restrict__ out,
                int n_vert, int K, int F, int f0, const int *__restrict__ order)
{
    pdl_begin();
    constexpr int T = 32 / LPT;  // targets of a warp
    __shared__ uint4 s_edge[256];  // source, weight, flags; terms of wide lists
    __shared__ int s_target[8 * T][3];  // hit, first edge, end; those with edges in front, for every 32
    constexpr int G = 256 / LPT;  // rows of a block
    const int lane = threadIdx.x & 31, hl = lane & (LPT - 1);
    const float inv = 1.f / (float)K;
    const int f = hl * VW;
    const bool have = f0 + f < F;
    const float *__restrict__ row0 = rows + (have ? f : 0);
    const float *__restrict__ max0 = MODE == kSumMeanMax ? maxima + (have ? f : 0) : nullptr;
    const unsigned flag_mask = f0 + f + VW <= F ? (1u << VW) - 1u : (1u << (have ? F - f0 - f : 0)) - 1u;

    if (threadIdx.x < 8 * T) {
        const int slot = blockIdx.x * (8 * T) + threadIdx.x;
        int m = -1, begin = 0, end = 0;
        if (slot < n_vert) {
            m = order ? order[slot] : slot;  // processing order only: every target is visited once
            begin = bounds[m];
            end = bounds[m + 1];
            if (end - begin > wide.limit) {
                m = -1;
                end = begin;
            }
        }
        constexpr unsigned kAll = 8 * T < 32 ? (1u << (8 * T)) - 1u : 0xffffffffu;
        const unsigned busy = __ballot_sync(kAll, end > begin), before = (1u << lane) - 1u;
        const int at = end > begin ? __popc(busy & before) : __popc(busy) + __popc(~busy & kAll & before);
        int *t = s_target[(threadIdx.x & ~31) + at];
        t[0] = m;
        t[1] = begin;
        t[2] = end;
    }
    __syncthreads();

    const int n_long = wide.counts[0], n_wide = n_long + wide.counts[1];
    for (int l = blockIdx.x; l < n_wide; l += gridDim.x) {
        const float *__restrict__ s_term = reinterpret_cast<const float *>(s_edge);
        const int m = wide.hits[l < n_long ? l : wide.room - 1 - (l - n_long)], end = bounds[m + 1], mine = threadIdx.x / LPT;
        int p = bounds[m];
        float acc = 0.f;
        int e[2];
#pragma unroll
        for (int q = 0; q < 2; q++) e[q] = p + q * G + mine < end ? edges[p + q * G + mine] : -1;
        for (; p < end; p += 2 * G) {
            EdgeVec g[2], h[2];
            float w[2];
            unsigned b[2];
#pragma unroll
            for (int q = 0; q < 2; q++) {
                w[q] = 0.f;
                b[q] = 0u;
                if (e[q] >= 0) {
                    const uint4 ed = edge_record<MODE>(e[q], m, K, weights, flags, nidx);
                    w[q] = __uint_as_float(ed.y);
                    g[q] = load_edge_vec(row0 + (size_t)ed.x * ldr);
                    if (MODE == kSumMeanMax) {
                        b[q] = ((LPT * VW > 32 && f >= 32 ? ed.w : ed.z) >> (f & 31)) & flag_mask;
                        h[q] = load_edge_vec_if<HVEC>(max0 + (size_t)ed.x * ldm, b[q]);
                    }
                }
                const int next = p + (2 + q) * G + mine;
                e[q] = next < end ? edges[next] : -1;
            }
#pragma unroll
            for (int q = 0; q < 2; q++) {
                const int n_here = min(G, end - p - q * G);
                if (mine < n_here) {
                    const EdgeVec t = edge_terms<MODE, SCALE>(g[q], h[q], w[q], b[q], inv);
                    s_edge[threadIdx.x] = make_uint4(__float_as_uint(t.v[0]), __float_as_uint(t.v[1]), __float_as_uint(t.v[2]), __float_as_uint(t.v[3]));
                }
                __syncthreads();
                if (threadIdx.x < LPT * VW) {
                    if (n_here == G) {
#pragma unroll 16
                        for (int k = 0; k < G; k++) acc = __fadd_rn(acc, s_term[k * (LPT * VW) + threadIdx.x]);
                    } else {
                        for (int k = 0; k < n_here; k++) acc = __fadd_rn(acc, s_term[k * (LPT * VW) + threadIdx.x]);
                    }
                }
                __syncthreads();
            }
        }
        if (threadIdx.x < LPT * VW && f0 + (int)threadIdx.x < F) out[(size_t)m * F + f0 + threadIdx.x] = acc;
    }

    uint4 *__restrict__ mine = s_edge + (threadIdx.x & ~(LPT - 1));
    const int *t = s_target[threadIdx.x / LPT];
    const int m = t[0], begin = t[1], end = t[2];
    float acc[VW];
#pragma unroll
    for (int v = 0; v < VW; v++) acc[v] = 0.f;
    for (int p = begin; __any_sync(0xffffffffu, p < end); p += LPT) {
        const int n_here = min(LPT, end - p);  // may be below zero where another target's list is longer
        __syncwarp();
        if (hl < n_here) mine[hl] = edge_record<MODE>(edges[p + hl], m, K, weights, flags, nidx);
        __syncwarp();
        // R rows at a time; while every target of the warp has as many more edges, without a test per target
        auto some = [&](int q0, auto tail) {
            EdgeVec g[R], h[R];
            float w[R];
            unsigned b[R];
#pragma unroll
            for (int q = 0; q < R; q++) {
                const uint4 ed = mine[q0 + q];
                w[q] = __uint_as_float(ed.y);
                b[q] = 0u;
                if (!tail.value || q0 + q < n_here) {
                    g[q] = load_edge_vec(row0 + (size_t)ed.x * ldr);
                    if (MODE == kSumMeanMax) {
                        b[q] = ((LPT * VW > 32 && f >= 32 ? ed.w : ed.z) >> (f & 31)) & flag_mask;
                        h[q] = load_edge_vec_if<HVEC>(max0 + (size_t)ed.x * ldm, b[q]);
                    }
                }
            }
#pragma unroll
            for (int q = 0; q < R; q++) {
                if (!tail.value || q0 + q < n_here) {
                    const EdgeVec t = edge_terms<MODE, SCALE>(g[q], h[q], w[q], b[q], inv);
#pragma unroll
                    for (int v = 0; v < VW; v++) acc[v] = __fadd_rn(acc[v], t.v[v]);
                }
            }
        };
        const int n_all = max(0, __reduce_min_sync(0xffffffffu, n_here)), n_max = __reduce_max_sync(0xffffffffu, n_here);
        int q0 = 0;
        for (; q0 + R <= n_all; q0 += R) some(q0, std::false_type());
        for (; q0 < n_max; q0 += R) some(q0, std::true_type());
    }
    if (have && m >= 0) {
        float *dst = out + (size_t)m * F + f0 + f;
#pragma unroll
        for (int v = 0; v < VW; v++)
            if (f0 + f + v < F) dst[v] = acc[v];
    }
}

// dst[i, 0 .. ld - 1] = x[i, 0 .. n - 1] / k, zeros behind: rows of whole vectors for edge_sum_kernel.  k == 1 copies.
// Dividing every row once instead of once per edge: both gradients of 200k hits, K = 40, F = 32 918 -> 718 us.
static __global__ void __launch_bounds__(256)
edge_rows_kernel(const float *__restrict__ x, int ldx, int n, float k, float *__restrict__ dst, int ld, int n_vert)
{
    pdl_begin();
    const long long t = (long long)blockIdx.x * 256 + threadIdx.x;
    const int i = (int)(t / ld), f = (int)(t - (long long)i * ld);
    if (i < n_vert) dst[t] = f < n ? __fdiv_rn(x[(size_t)i * ldx + f], k) : 0.f;
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
// VEC: rows are whole 16-byte vectors (F % 4 == 0, bases aligned), which cp.async puts into shared memory past the registers
// and L1.  12.8 M edges, F = 64: 0.85 ms with 4-byte loads and stores and a test of every feature for the maximum, bound by
// issue (80 % of the slots) and the L1 data stage (79 %); 0.62 with 16-byte loads and stores, packed products and the
// maxima taken from the bits; 0.50 with cp.async (cached in L1 as well 0.53; MAX without the bound on registers 0.56).
// MAX also writes the edge's bits for edge_sum_kernel (features 0 .. 63), which it compares for anyway.
template <bool GRAD, bool MAX, bool VEC>
__global__ void __launch_bounds__(256, MAX ? 5 : 6)
edge_dot_kernel(const float *__restrict__ own, int ld_own, const float *__restrict__ x, const int *__restrict__ arg,
                const int *__restrict__ nidx, float *__restrict__ out, long long n_edges, int n_vert, int K, int F,
                const int *__restrict__ order, unsigned *__restrict__ flags)
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
        const int row = n_edges <= 0xffffffffLL ? (int)((unsigned)t / (unsigned)K) : (int)(t / K);
        i = order ? order[row] : row;  // processing order only
        e = (long long)i * K + (t - (long long)row * K);
        m = nidx[e];
        if (m >= n_vert) m = -1;
    }
    const float *__restrict__ g = own + (size_t)i * ld_own;
    const int *__restrict__ am = MAX ? arg + (size_t)i * F : nullptr;
    const int arg_m = m >= 0 ? m : (int)0x80000000;  // no neighbour is nobody's maximum
    float mean_part = 0.f, max_part = 0.f;
    uint2 bits = make_uint2(0u, 0u);
    for (int f0 = 0; f0 < F; f0 += 32) {
        unsigned hit = 0u;
        __syncwarp();
        if (VEC) {
            const int c = (lane & 7) * 4;
            const bool in = f0 + c < F;
#pragma unroll
            for (int q = 0; q < 32; q += 4) {
                const int mq = __shfl_sync(0xffffffffu, m, q + (lane >> 3));
                const int bytes = in && mq >= 0 ? 16 : 0;  // the rest of the 16 bytes is filled with zeros
                const unsigned dst = (unsigned)__cvta_generic_to_shared(s + (q + (lane >> 3)) * kRow + c);
                const float *src = x + (bytes ? (size_t)mq * F + f0 + c : 0);
                asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" :: "r"(dst), "l"(src), "r"(bytes) : "memory");
            }
            asm volatile("cp.async.commit_group;\ncp.async.wait_group 0;" ::: "memory");
        } else {
            const bool in = f0 + lane < F;
#pragma unroll 8
            for (int q = 0; q < 32; q++) {
                const int mq = __shfl_sync(0xffffffffu, m, q);
                s[q * kRow + lane] = in && mq >= 0 ? __ldg(x + (size_t)mq * F + f0 + lane) : 0.f;
            }
        }
        __syncwarp();
#pragma unroll
        for (int c = 0; c < 32; c += 4) {
            if (f0 + c >= F) break;  // uniform
            const float4 xv = *reinterpret_cast<const float4 *>(s + lane * kRow + c);
            float4 gv = make_float4(0.f, 0.f, 0.f, 0.f);
            int4 av = make_int4(-1, -1, -1, -1);
            if (VEC) {
                gv = __ldg(reinterpret_cast<const float4 *>(g + f0 + c));
                if (MAX) av = __ldg(reinterpret_cast<const int4 *>(am + f0 + c));
            } else {
                const int left = F - f0 - c;
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
            const float2 p01 = mul2(gv.x, gv.y, xv.x, xv.y), p23 = mul2(gv.z, gv.w, xv.z, xv.w);
            mean_part = __fadd_rn(mean_part, p01.x);
            mean_part = __fadd_rn(mean_part, p01.y);
            mean_part = __fadd_rn(mean_part, p23.x);
            mean_part = __fadd_rn(mean_part, p23.y);
            if (MAX) {
                if (av.x == arg_m) hit |= 1u << c;
                if (av.y == arg_m) hit |= 2u << c;
                if (av.z == arg_m) hit |= 4u << c;
                if (av.w == arg_m) hit |= 8u << c;
            }
        }
        if (MAX) {
            // a feature's maximum lies in one slot, so a lane has F / K of them on average
            const float *__restrict__ gm = g + F + f0;
            // (two loads at a time: a table of few edges waits for them)
            for (unsigned left = hit; left != 0u;) {
                const int a = __ffs(left) - 1;
                left &= left - 1u;
                const int b = left != 0u ? __ffs(left) - 1 : a;
                const float ga = __ldg(gm + a), gb = __ldg(gm + b);
                max_part = __fadd_rn(max_part, __fmul_rn(ga, s[lane * kRow + a]));
                if (left != 0u) max_part = __fadd_rn(max_part, __fmul_rn(gb, s[lane * kRow + b]));
                left &= left - 1u;
            }
            if (f0 == 0) bits.x = hit;
            if (f0 == 32) bits.y = hit;
        }
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

// One slab of up to 64 features of edge_sum_kernel.  Lanes per target: as many as
// the width needs at four features each, so that narrow rows share a warp (200k hits, K = 16, F = 16: PushKnn 220 -> 146 us).
template <int MODE>
int launch_edge_sum_slab(const float *x, int ldx, const float *weights, const unsigned *flags, const int *nidx,
                         const Incoming &lists, float *out, int n_vert, int K, int F, int f0, const int *order,
                         cudaStream_t stream)
{
    float *const scratch = lists.rows;
    const int width = F - f0 < 64 ? F - f0 : 64;
    // rows are read where they lie if they are whole vectors and the division by K is an exact scaling
    const bool whole = copied_row(F, aligned16(x), false) == 0;
    const float *rows = x + f0;
    int ldr = ldx;
    if (copied_row(F, aligned16(x), MODE != kSumPlain && !power_of_two(K)) > 0) {
        ldr = (width + 3) / 4 * 4;
        HGC_CUDA_TRY(launch_overlapped(n_vert, edge_rows_kernel, div_up((long long)n_vert * ldr, 256), 256, 0, stream, x + f0, ldx, width,
                                       MODE == kSumPlain ? 1.f : (float)K, scratch, ldr, n_vert));
        HGC_LAUNCH_CHECK();
        rows = scratch;
    }
    const bool few = div_up(n_vert, 16) <= 2 * sm_count();
    const bool scale = MODE != kSumPlain && rows != scratch;  // only rows that are whole vectors are scaled
#define HGC_SUM(LPT, R, S, H) HGC_CUDA_TRY(launch_overlapped(n_vert, edge_sum_kernel<LPT, R, MODE, S, H>, div_up(n_vert, 8 * (32 / LPT)), 256, 0, stream, rows, ldr, x + F + f0, ldx, weights, flags, nidx, lists.bounds, lists.edges, lists.wide, out, n_vert, K, F, f0, order))
#define HGC_SUM_W(S, H) do { if (few) HGC_SUM(16, 8, S, H); else if (width > 32) HGC_SUM(16, 2, S, H); else if (width > 16) HGC_SUM(8, 2, S, H); else HGC_SUM(4, 2, S, H); } while (0)
    if constexpr (MODE == kSumPlain) HGC_SUM_W(false, false);
    else if constexpr (MODE == kSumMean) { if (scale) HGC_SUM_W(true, false); else HGC_SUM_W(false, false); }
    else { if (scale) HGC_SUM_W(true, true); else if (whole) HGC_SUM_W(false, true); else HGC_SUM_W(false, false); }
#undef HGC_SUM_W
#undef HGC_SUM
    HGC_LAUNCH_CHECK();
    return HGC_OK;
}

}  // namespace hgc
