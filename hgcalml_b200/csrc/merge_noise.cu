// merge_noise_as_indiv_cp (modules/assign_condensate_op.py:16-44): noise hits become condensation points of their own.
// Noise hits and condensation points are counted per tile of an event, then every tile adds up what lies before it and
// writes its part of all outputs: three launches instead of some ninety tensor operations with six round trips
// to the host (16.5k hits: 0.75 ms -> 0.02 ms).
#include "common.cuh"
#include "hit_order.cuh"
#include "hit_order_device.cuh"

namespace hgc {
namespace {

constexpr int kThreads = kOrderThreads;

__global__ void __launch_bounds__(kThreads)
layout_kernel(const int *__restrict__ row_splits, int n_events, int n_vert, HitOrder o)
{
    pdl_begin();
    event_layout(row_splits, n_events, n_vert, o);
}

__global__ void __launch_bounds__(kThreads)
count_noise_kernel(const int *__restrict__ assignment, const int *__restrict__ association,
                   const unsigned char *__restrict__ is_cond, HitOrder o, int n_events, int2 *__restrict__ counts)
{
    pdl_begin();
    HitTile t;
    if (!find_tile(o, n_events, blockIdx.x, &t)) return;
    __shared__ int s_noise, s_points;
    if (threadIdx.x == 0) s_noise = s_points = 0;
    __syncthreads();
    int noise = 0, points = 0;
    if (t.event < n_events)
        for (int i = threadIdx.x; i < t.n; i += kThreads) {
            const int v = t.first + i;
            noise += assignment[v] < 0 ? 1 : 0;
            points += is_cond[v] || association[v] < 0 ? 1 : 0;
        }
    noise = __reduce_add_sync(0xffffffffu, noise);
    points = __reduce_add_sync(0xffffffffu, points);
    if ((threadIdx.x & 31) == 0) { atomicAdd(&s_noise, noise); atomicAdd(&s_points, points); }
    __syncthreads();
    if (threadIdx.x == 0) counts[blockIdx.x] = make_int2(s_noise, s_points);
}

__global__ void __launch_bounds__(kThreads)
merge_noise_kernel(const int *__restrict__ assignment, const int *__restrict__ association, const int *__restrict__ alpha,
                   const unsigned char *__restrict__ is_cond, const int *__restrict__ n_cond,
                   const int *__restrict__ row_splits, HitOrder o, int n_events, const int2 *__restrict__ counts,
                   int *__restrict__ new_assignment, int *__restrict__ new_association, int *__restrict__ new_alpha,
                   unsigned char *__restrict__ new_is_cond, int *__restrict__ new_n_cond, int *__restrict__ n_alpha)
{
    pdl_begin();
    __shared__ int s_warp[kThreads / kWarp];
    __shared__ int s_sum[3];  // noise hits before the event, before the tile, up to the end of the event
    __shared__ int s_base;
    auto add = [](int a, int b) { return a + b; };
    if (blockIdx.x == gridDim.x - 1) {
        // the last block has no tile: the counts of all events, and the total; -1 where the events are not all hits
        int carry = n_cond[0];
        bool bad = row_splits[0] != 0 || row_splits[n_events] != o.event_pos[n_events + 1];
        for (int e0 = 0; e0 < n_events; e0 += kThreads) {
            const int e = e0 + threadIdx.x;
            int points = 0;
            bad = bad || (e < n_events && row_splits[e + 1] < row_splits[e]);
            if (e < n_events)
                for (int q = o.event_tile[e]; q < o.event_tile[e + 1]; q++) points += counts[q].y;
            const int incl = carry + block_scan_inclusive(points, add, 0, s_warp);
            if (e < n_events) new_n_cond[e + 1] = incl;
            __syncthreads();
            if (threadIdx.x == kThreads - 1) s_base = incl;
            __syncthreads();
            carry = s_base;
        }
        int noise = 0;
        for (int q = threadIdx.x; q < o.event_tile[n_events]; q += kThreads) noise += counts[q].x;
        const int all = block_scan_inclusive(noise, add, 0, s_warp);
        bad = __syncthreads_or(bad ? 1 : 0) != 0;
        if (threadIdx.x == kThreads - 1) {
            new_n_cond[0] = n_cond[0];
            *n_alpha = bad ? -1 : all + n_cond[n_events] - n_cond[0];
        }
        return;
    }
    HitTile t;
    if (!find_tile(o, n_events, blockIdx.x, &t)) return;
    if (t.event >= n_events) {  // beyond the last event
        for (int i = threadIdx.x; i < t.n; i += kThreads) {
            const int v = t.first + i;
            new_assignment[v] = assignment[v];
            new_association[v] = association[v];
            new_is_cond[v] = is_cond[v];
        }
        return;
    }
    if (threadIdx.x < 3) s_sum[threadIdx.x] = 0;
    __syncthreads();
    const int tile0 = o.event_tile[t.event], tile1 = o.event_tile[t.event + 1];
    int a = 0, b = 0, c = 0;
    for (int q = threadIdx.x; q < tile1; q += kThreads) {
        const int n = counts[q].x;
        a += q < tile0 ? n : 0;
        b += q < (int)blockIdx.x ? n : 0;
        c += n;
    }
    a = __reduce_add_sync(0xffffffffu, a);
    b = __reduce_add_sync(0xffffffffu, b);
    c = __reduce_add_sync(0xffffffffu, c);
    if ((threadIdx.x & 31) == 0) { atomicAdd(&s_sum[0], a); atomicAdd(&s_sum[1], b); atomicAdd(&s_sum[2], c); }
    __syncthreads();
    const int before_event = s_sum[0], n_noise = s_sum[2] - s_sum[0];
    const int cond0 = n_cond[t.event] - n_cond[0], cond1 = n_cond[t.event + 1] - n_cond[0];
    int run = s_sum[1] - s_sum[0];  // noise hits of the event before this tile
    for (int i0 = 0; i0 < t.n; i0 += kThreads) {
        const int i = i0 + threadIdx.x, v = t.first + i;
        const bool in = i < t.n;
        const int as = in ? assignment[v] : 0;
        const bool noise = in && as < 0;
        const int incl = block_scan_inclusive(noise ? 1 : 0, add, 0, s_warp);
        if (in) {
            const int rank = run + incl - 1, asso = association[v];
            new_assignment[v] = noise ? rank : as + n_noise;
            new_association[v] = asso < 0 ? v : asso;
            new_is_cond[v] = is_cond[v] || asso < 0 ? 1 : 0;
            if (noise) new_alpha[before_event + cond0 + rank] = v;
        }
        __syncthreads();
        if (threadIdx.x == kThreads - 1) s_base = incl;
        __syncthreads();
        run += s_base;
    }
    // the event's condensates follow its noise hits; its tiles share the copying
    for (int k = cond0 + ((int)blockIdx.x - tile0) * kThreads + threadIdx.x; k < cond1; k += (tile1 - tile0) * kThreads)
        new_alpha[before_event + n_noise + k] = alpha[k];
}

struct Sized {
    Sizer s;
    template <typename T> T *take(size_t n) { s.take<T>(n); return nullptr; }
};

template <typename W>
void layout(W &ws, int n_vert, int n_rs, HitOrder *o, int2 **counts, int **n_alpha)
{
    const int n_events = n_rs > 1 ? n_rs - 1 : 0;
    const size_t e = (size_t)n_events + 2;
    *o = HitOrder();
    o->tile = order_tile(n_vert);
    o->event_pos = ws.template take<int>(e);
    o->event_tile = ws.template take<int>(e);
    o->event_chunk = ws.template take<int>(e);
    o->event_super = ws.template take<int>(e);
    *counts = ws.template take<int2>(order_tiles_cap(n_vert, n_events));
    *n_alpha = ws.template take<int>(1);
}

}  // namespace
}  // namespace hgc

using namespace hgc;

extern "C" size_t hgc_merge_noise_workspace_bytes(int n_vert, int n_rs)
{
    Sized w;
    HitOrder o;
    int2 *counts;
    int *n_alpha;
    layout(w, n_vert, n_rs, &o, &counts, &n_alpha);
    return w.s.used;
}

extern "C" int hgc_merge_noise(
        const int *d_assignment, const int *d_association, const int *d_alpha_idx, const unsigned char *d_is_cond,
        const int *d_n_condensates, const int *d_row_splits,
        int *d_new_assignment, int *d_new_association, int *d_new_alpha_idx, unsigned char *d_new_is_cond,
        int *d_new_n_condensates, int *h_n_alpha, int n_vert, int n_rs,
        void *workspace, size_t workspace_bytes, hgc_stream_t stream_)
{
    cudaStream_t stream = static_cast<cudaStream_t>(stream_);
    if (n_vert < 0 || n_rs < 1 || !d_n_condensates || !d_row_splits || !d_new_n_condensates) return HGC_ERR_INVALID_ARGUMENT;
    if (n_vert > 0 && (!d_assignment || !d_association || !d_alpha_idx || !d_is_cond || !d_new_assignment ||
                       !d_new_association || !d_new_alpha_idx || !d_new_is_cond))
        return HGC_ERR_INVALID_ARGUMENT;
    if (int rc = check_workspace(workspace, workspace_bytes, hgc_merge_noise_workspace_bytes(n_vert, n_rs))) return rc;
    Carver ws(workspace);
    HitOrder o;
    int2 *counts;
    int *n_alpha;
    layout(ws, n_vert, n_rs, &o, &counts, &n_alpha);
    const int n_events = n_rs - 1, tiles = (int)order_tiles_cap(n_vert, n_events);
    HGC_CUDA_TRY(cudaMemsetAsync(ws.status(), 0, kAlign, stream));
    HGC_CUDA_TRY(launch_pdl(layout_kernel, 1, kThreads, 0, stream, d_row_splits, n_events, n_vert, o));
    HGC_LAUNCH_CHECK();
    HGC_CUDA_TRY(launch_pdl(count_noise_kernel, tiles, kThreads, 0, stream, d_assignment, d_association, d_is_cond, o, n_events, counts));
    HGC_LAUNCH_CHECK();
    HGC_CUDA_TRY(launch_pdl(merge_noise_kernel, tiles + 1, kThreads, 0, stream, d_assignment, d_association, d_alpha_idx, d_is_cond,
                                                           d_n_condensates, d_row_splits, o, n_events, counts, d_new_assignment,
                                                           d_new_association, d_new_alpha_idx, d_new_is_cond,
                                                           d_new_n_condensates, n_alpha));
    HGC_LAUNCH_CHECK();
    if (h_n_alpha) {
        HGC_CUDA_TRY(cudaMemcpyAsync(h_n_alpha, n_alpha, sizeof(int), cudaMemcpyDeviceToHost, stream));
        HGC_CUDA_TRY(cudaStreamSynchronize(stream));
    }
    return HGC_OK;
}
