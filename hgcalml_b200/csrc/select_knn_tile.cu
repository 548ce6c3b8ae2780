// Host side of the tile search: layout of the sorted hits in padded chunks, boxes, dispatch.
#include "common.cuh"
#include "knn_device.cuh"
#include "select_knn_tile_api.cuh"

namespace hgc {
namespace {

// A block per super-chunk, a thread per hit: the 1024 hits of a super-chunk, consecutive on the curve, are
// split five times at the median of the coordinate in which the part is widest, which leaves parts of 32 hits:
// the chunks.  Their boxes do not overlap, and a ball of 64 hits in four dimensions meets a third fewer of
// them than of runs of 32 hits along the curve.  A part is split by sorting words of the quantised position
// in the part (22 bits) and the hit's number (10 bits), a network of shuffles and a few exchanges through
// shared memory; the split need not be exact.  Padding sorts last at every level, so the real hits
// stay in front.
constexpr int kPackThreads = 1024;
constexpr int kSplitDims = 8;  // coordinates that splits look at

__device__ __forceinline__ unsigned exchange_u32(unsigned v, unsigned *s_x, int partner, bool lower)
{
    __syncthreads();  // the previous exchange has been read
    s_x[threadIdx.x] = v;
    __syncthreads();
    const unsigned o = s_x[partner];
    return lower ? min(v, o) : max(v, o);
}

__global__ void __launch_bounds__(kPackThreads)
pack_tiles_kernel(const float *__restrict__ coords, int C, const int *__restrict__ perm,
                  const int *__restrict__ rank_of,
                  const int *__restrict__ direction, int n_events, HitOrder o, TileScratch s, int nv4, int nobody)
{
    pdl_begin();
    extern __shared__ float s_c[];  // [min(C, kSplitDims)][1024] coordinates in curve order
    __shared__ float s_lo[32][16], s_hi[32][16];
    __shared__ unsigned s_x[kPackThreads];
    const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
    const int sup = blockIdx.x;
    if (sup == 0 && warp == 31) {  // the chunk that holds no hits
        s.ranks[nobody + lane] = 0;
        for (int u = 0; u < nv4; u++)
            s.pts[(size_t)(nobody + lane) * nv4 + u] = make_float4(NAN, NAN, NAN, NAN);
    }
    if (sup >= o.event_super[n_events + 1]) return;
    int lo_e = 0, hi_e = n_events;  // last event whose first super-chunk is <= sup (events without hits share one)
    while (lo_e < hi_e) {
        const int mid = (lo_e + hi_e + 1) >> 1;
        if (o.event_super[mid] <= sup) lo_e = mid; else hi_e = mid - 1;
    }
    const int e = lo_e;
    const int chunk0 = o.event_chunk[e], chunk1 = o.event_chunk[e + 1];
    const int local0 = (sup - o.event_super[e]) * kPackThreads;
    const int pos0 = o.event_pos[e] + local0;
    const int n_here = min(o.event_pos[e + 1] - pos0, kPackThreads);
    const int cd = min(C, kSplitDims);
    {
        const int id = t < n_here ? perm[pos0 + t] : -1;
        for (int c = 0; c < cd; c++) s_c[c * kPackThreads + t] = id >= 0 ? coords[(size_t)id * C + c] : 0.f;
    }
    __syncthreads();
    int li = t;  // hit (in curve order) at this thread's place
    for (int size = kPackThreads; size > 32; size >>= 1) {
        if (n_here <= 32) break;
        // extents of the part this warp belongs to
        const bool real = li < n_here;
        for (int c = 0; c < cd; c++) {
            const float x = s_c[c * kPackThreads + li];
            const float lo = warp_min_f32(real ? x : INFINITY), hi = warp_max_f32(real ? x : -INFINITY);
            if (lane == 0) { s_lo[warp][c] = lo; s_hi[warp][c] = hi; }
        }
        __syncthreads();
        const int w0 = warp & ~(size / 32 - 1);
        float best_lo = 0.f, best_ext = -1.f;
        int dim = 0;
        for (int c = 0; c < cd; c++) {
            const bool in = lane < size / 32;
            const float lo = warp_min_f32(in ? s_lo[w0 + lane][c] : INFINITY);
            const float hi = warp_max_f32(in ? s_hi[w0 + lane][c] : -INFINITY);
            if (hi - lo > best_ext) { best_ext = hi - lo; best_lo = lo; dim = c; }
        }
        const float scale = best_ext > 0.f ? 4194302.f / best_ext : 0.f;
        unsigned w = 0x3fffffu;
        if (real) w = (unsigned)fminf(fmaxf((s_c[dim * kPackThreads + li] - best_lo) * scale, 0.f), 4194302.f);
        w = (w << 10) | (unsigned)li;
        // ascending sort of every part of `size` threads
        w = warp_sort_u32(w, lane);
        for (int k = 64; k <= size; k <<= 1) {
            w = exchange_u32(w, s_x, t ^ (k - 1), (t & (k >> 1)) == 0);
            for (int j = k >> 2; j >= 32; j >>= 1) w = exchange_u32(w, s_x, t ^ j, (t & j) == 0);
            w = warp_bitonic_merge_u32(w, lane);
        }
        li = (int)(w & 1023u);
    }

    const int chunk = chunk0 + local0 / 32 + warp;
    const bool have = chunk < chunk1;
    const int id = li < n_here ? perm[pos0 + li] : -1;
    if (have) {
        s.ids[(size_t)chunk * 32 + lane] = id;
        s.ranks[(size_t)chunk * 32 + lane] = id >= 0 ? rank_of[id] : 0;
        if (lane == 0) {
            // hits beyond the last event take part in nothing
            const bool none = e == n_events;
            s.chunk_info[chunk] = make_int4(chunk0, none ? chunk0 : chunk1, o.event_super[e], o.event_super[e + 1]);
        }
    }
    bool usable = id >= 0;
    if (direction != nullptr && usable) {
        const int d = direction[id];
        usable = !(d == 1 || d == 2);  // may not be anybody's neighbour
    }
    const float nan = __int_as_float(0x7fffffff);
    __syncthreads();  // s_lo, s_hi are used again
    for (int u = 0; u < nv4; u++) {
        float c[4], lo[4], hi[4];
#pragma unroll
        for (int k = 0; k < 4; k++) {
            const int d = u * 4 + k;
            c[k] = 0.f;
            if (d < C && usable) c[k] = coords[(size_t)id * C + d];
            lo[k] = warp_min_f32(usable ? c[k] : INFINITY);
            hi[k] = warp_max_f32(usable ? c[k] : -INFINITY);
            if (!usable) c[k] = nan;
        }
        if (have) {
            s.pts[((size_t)chunk * 32 + lane) * nv4 + u] = make_float4(c[0], c[1], c[2], c[3]);
            if (lane == 0) {
                s.chunk_box[((size_t)chunk * nv4 + u) * 2] = make_float4(lo[0], lo[1], lo[2], lo[3]);
                s.chunk_box[((size_t)chunk * nv4 + u) * 2 + 1] = make_float4(hi[0], hi[1], hi[2], hi[3]);
            }
        }
        if (lane == 0)
#pragma unroll
            for (int k = 0; k < 4; k++) { s_lo[warp][u * 4 + k] = lo[k]; s_hi[warp][u * 4 + k] = hi[k]; }
    }
    __syncthreads();
    if (warp < nv4) {
        float lo[4], hi[4];
#pragma unroll
        for (int k = 0; k < 4; k++) {
            lo[k] = warp_min_f32(s_lo[lane][warp * 4 + k]);
            hi[k] = warp_max_f32(s_hi[lane][warp * 4 + k]);
        }
        if (lane == 0) {
            s.super_box[((size_t)sup * nv4 + warp) * 2] = make_float4(lo[0], lo[1], lo[2], lo[3]);
            s.super_box[((size_t)sup * nv4 + warp) * 2 + 1] = make_float4(hi[0], hi[1], hi[2], hi[3]);
        }
    }
}

}  // namespace

int build_tiles(const float *coords, int n_coords, const int *curve_perm, const int *rank_of, const HitOrder &o,
                int n_events, const int *direction, const TileScratch &s, int n_vert, cudaStream_t stream)
{
    if (n_vert <= 0) return HGC_OK;
    const size_t smem = sizeof(float) * kPackThreads * (n_coords < kSplitDims ? n_coords : kSplitDims);
    HGC_CUDA_TRY(launch_overlapped(n_vert, pack_tiles_kernel, (int)tile_supers_cap(n_vert, n_events), kPackThreads, smem, stream, coords, n_coords, curve_perm, rank_of, direction, n_events, o, s, (n_coords + 3) / 4,
            (int)(tile_chunks_cap(n_vert, n_events) * 32)));
    HGC_LAUNCH_CHECK();
    return HGC_OK;
}

int search_tiles(const TileScratch &s, const HitOrder &o, const int *rank_to_id, const float *coords, int n_coords, const int *direction, int *out_idx,
                 float *out_dist, int n_vert, int n_events, int K, int tf_compat, cudaStream_t stream)
{
    if (n_vert <= 0) return HGC_OK;
    TileKnnArgs a;
    a.pts = s.pts; a.ids = s.ids; a.ranks = s.ranks; a.rank_to_id = rank_to_id; a.chunk_box = s.chunk_box; a.super_box = s.super_box; a.chunk_info = s.chunk_info;
    a.n_chunks = o.event_chunk + n_events + 1;
    a.coords = direction ? coords : nullptr;
    a.direction = direction;
    a.out_idx = out_idx; a.out_dist = out_dist;
    a.nobody = (int)(tile_chunks_cap(n_vert, n_events) * 32);
    a.n_coords = n_coords; a.K = K; a.tf_compat = tf_compat;
    a.expo = 2.f / (float)n_coords;
    a.guess = powf(1.6f, a.expo);  // 60 % more hits, at equal density: measured flat from 1.3 to 1.8
    // Queries per block: whole chunks share the list of one tile among most queries; small batches are cut
    // finer, so that every SM has work.
    const long long chunks = (long long)tile_chunks_cap(n_vert, n_events);
    const long long fill = (long long)sm_count() * 8;
    a.tile = 32;
    while (a.tile > 4 && chunks * (32 / a.tile) < fill) a.tile >>= 1;
    const long long tiles = chunks * (32 / a.tile);
    if (tiles > 0x7fffffffLL) return HGC_ERR_UNSUPPORTED;
    switch ((n_coords + 3) / 4) {
        case 1: return launch_tile_nv<1>(a, (int)tiles, stream);
        case 2: return launch_tile_nv<2>(a, (int)tiles, stream);
        case 3: return launch_tile_nv<3>(a, (int)tiles, stream);
        case 4: return launch_tile_nv<4>(a, (int)tiles, stream);
    }
    return HGC_ERR_UNSUPPORTED;
}

}  // namespace hgc
