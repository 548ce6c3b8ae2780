// Device side of the event layout, shared by the kernels that work tile by tile.
#pragma once
#include "common.cuh"
#include "hit_order.cuh"

namespace hgc {

constexpr int kOrderThreads = 256;

template <typename Op>
__device__ __forceinline__ int block_scan_inclusive(int v, Op op, int identity, int *s_warp)
{
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const int t = __shfl_up_sync(0xffffffffu, v, o);
        if (lane >= o) v = op(v, t);
    }
    __syncthreads();  // s_warp may still be read by the previous scan
    if (lane == 31) s_warp[warp] = v;
    __syncthreads();
    int before = identity;
    for (int w = 0; w < warp; w++) before = op(before, s_warp[w]);
    return op(before, v);
}

// First position, tile, chunk and super-chunk of every event, and of the run of hits that lie beyond the last
// event.  Row splits are clamped to an ascending sequence inside [0, n_vert], so the layout stays
// inside its arrays whatever they hold.  One block of kOrderThreads.
__device__ __forceinline__ void event_layout(const int *__restrict__ row_splits, int n_events, int n_vert, const HitOrder &o)
{
    if (n_events < 32) {  // a few events: one warp, no barriers
        if (threadIdx.x >= 32) return;
        const int e = threadIdx.x;
        int end = e < n_events ? min(max(row_splits[e + 1], 0), n_vert) : n_vert;
#pragma unroll
        for (int d = 1; d < 32; d <<= 1) {
            const int v = __shfl_up_sync(0xffffffffu, end, d);
            if (e >= d) end = max(end, v);
        }
        int begin = __shfl_up_sync(0xffffffffu, end, 1);
        if (e == 0) begin = 0;
        const int n = e <= n_events ? end - begin : 0;
        const int nt = (n + o.tile - 1) / o.tile, nc = (n + 31) / 32, ns = (nc + 31) / 32;
        int ti = nt, ci = nc, si = ns;
#pragma unroll
        for (int d = 1; d < 32; d <<= 1) {
            const int a = __shfl_up_sync(0xffffffffu, ti, d), b = __shfl_up_sync(0xffffffffu, ci, d);
            const int c = __shfl_up_sync(0xffffffffu, si, d);
            if (e >= d) { ti += a; ci += b; si += c; }
        }
        if (e <= n_events) {
            o.event_pos[e] = begin;
            o.event_tile[e] = ti - nt;
            o.event_chunk[e] = ci - nc;
            o.event_super[e] = si - ns;
            if (e == n_events) {
                o.event_pos[e + 1] = end;
                o.event_tile[e + 1] = ti;
                o.event_chunk[e + 1] = ci;
                o.event_super[e + 1] = si;
            }
        }
        return;
    }
    __shared__ int s_warp[kOrderThreads / kWarp];
    __shared__ int s_last[4];
    auto add = [](int a, int b) { return a + b; };
    auto mx = [](int a, int b) { return a > b ? a : b; };
    int pos = 0, tile = 0, chunk = 0, super = 0;  // carried over from the events before
    for (int base = 0; base <= n_events; base += kOrderThreads) {
        const int e = base + threadIdx.x;
        // end of event e; the last entry (the hits beyond the last event) ends with the batch
        int end = e < n_events ? min(max(row_splits[e + 1], 0), n_vert) : n_vert;
        end = mx(pos, block_scan_inclusive(end, mx, 0, s_warp));
        int begin = __shfl_up_sync(0xffffffffu, end, 1);
        __syncthreads();
        if ((threadIdx.x & 31) == 31) s_warp[threadIdx.x >> 5] = end;
        __syncthreads();
        if ((threadIdx.x & 31) == 0) begin = threadIdx.x == 0 ? pos : s_warp[(threadIdx.x >> 5) - 1];
        const int n = e <= n_events ? end - begin : 0;
        const int nt = (n + o.tile - 1) / o.tile, nc = (n + 31) / 32, ns = (nc + 31) / 32;
        const int ti = tile + block_scan_inclusive(nt, add, 0, s_warp);
        const int ci = chunk + block_scan_inclusive(nc, add, 0, s_warp);
        const int si = super + block_scan_inclusive(ns, add, 0, s_warp);
        if (e <= n_events) {
            o.event_pos[e] = begin;
            o.event_tile[e] = ti - nt;
            o.event_chunk[e] = ci - nc;
            o.event_super[e] = si - ns;
            if (e == n_events) {
                o.event_pos[e + 1] = end;
                o.event_tile[e + 1] = ti;
                o.event_chunk[e + 1] = ci;
                o.event_super[e + 1] = si;
            }
        }
        __syncthreads();
        if (threadIdx.x == kOrderThreads - 1) { s_last[0] = end; s_last[1] = ti; s_last[2] = ci; s_last[3] = si; }
        __syncthreads();
        pos = s_last[0]; tile = s_last[1]; chunk = s_last[2]; super = s_last[3];
    }
}

__device__ __forceinline__ int event_of_tile(const int *__restrict__ event_tile, int n_events, int tile)
{
    int lo = 0, hi = n_events;  // last event whose first tile is <= tile (events without hits share one)
    while (lo < hi) {
        const int mid = (lo + hi + 1) >> 1;
        if (event_tile[mid] <= tile) lo = mid; else hi = mid - 1;
    }
    return lo;
}

struct HitTile { int event, first, n; };  // positions [first, first + n)

__device__ __forceinline__ bool find_tile(const HitOrder &o, int n_events, int tile, HitTile *t)
{
    if (tile >= o.event_tile[n_events + 1]) return false;
    t->event = event_of_tile(o.event_tile, n_events, tile);
    t->first = o.event_pos[t->event] + (tile - o.event_tile[t->event]) * o.tile;
    t->n = min(o.event_pos[t->event + 1] - t->first, o.tile);
    return true;
}

}  // namespace hgc
