// Host side of the tile search: layout of the sorted hits in padded chunks, boxes, dispatch.
#include "common.cuh"
#include "knn_device.cuh"
#include "select_knn_tile_api.cuh"

namespace hgc {
namespace {

// A block per super-chunk of 1024 hits that are consecutive on the curve, a warp per 32 W of them (128 or 256), which it splits two
// or three times at the median of the coordinate in which the part is widest: that leaves parts of 32 hits, the chunks.  The boxes of a
// warp's chunks overlap only where hits tie or differ by less than the quantisation (those of two warps may: nothing
// separates runs of the curve), and a ball of 64 hits in four dimensions meets fewer of them than of runs of 32 hits along the
// curve.  A part is split by sorting words of the quantised position in the part (25 bits for W = 4, 24 for W = 8) and the
// hit's place (7 or 8 bits), W words per lane, by a network of shuffles; the split need not be exact.  Padding sorts last, so
// the real hits stay in front.
// Five splits of the whole super-chunk, a thread per hit, took 18 us for one block and 57 us for 400k hits, most of it in
// shuffles and barriers, and gave chunks that are no better: search and packing, 400k hits in four dimensions, K = 64, from
// parts of 1024 1202 us, 512 1180, 256 1188, 128 1168, 32 (no split) 1192.  This kernel: 18 us for 400k hits, 10 for one block.
constexpr int kSuper = 1024;
constexpr int kSplitDims = 8;  // coordinates that splits look at

__device__ __forceinline__ void order_pair(unsigned &a, unsigned &b)
{
    const unsigned lo = min(a, b);
    b = max(a, b);
    a = lo;
}

// Ascending sort of every group of N words (N / W lanes, W consecutive words each).
template <int N, int W>
__device__ __forceinline__ void sort_parts(unsigned (&w)[W], int lane)
{
    // compares the words of a lane whose numbers differ in the bits of m
    auto inside = [&](int m) {
#pragma unroll
        for (int r = 0; r < W; r++)
            if ((r ^ m) > r) order_pair(w[r], w[r ^ m]);
    };
#pragma unroll
    for (int k = 2; k <= N; k <<= 1) {
        if (k <= W) {
            inside(k - 1);
        } else {
            unsigned o[W];
#pragma unroll
            for (int r = 0; r < W; r++) o[r] = __shfl_xor_sync(0xffffffffu, w[W - 1 - r], k / W - 1);
#pragma unroll
            for (int r = 0; r < W; r++) w[r] = (lane & (k / (2 * W))) == 0 ? min(w[r], o[r]) : max(w[r], o[r]);
        }
#pragma unroll
        for (int j = k / 4; j > 0; j >>= 1) {
            if (j < W) {
                inside(j);
            } else {
#pragma unroll
                for (int r = 0; r < W; r++) {
                    const unsigned v = __shfl_xor_sync(0xffffffffu, w[r], j / W);
                    w[r] = (lane & (j / W)) == 0 ? min(w[r], v) : max(w[r], v);
                }
            }
        }
    }
}

// One split: the places of a part of kPart >> LEVEL hits in the order of the coordinate in which it is widest.
template <int LEVEL, int W>
__device__ __forceinline__ void split_part(const float *__restrict__ s_w, int cd, int n_here, int lane, int (&li)[W])
{
    constexpr int kLanes = 32 >> LEVEL;  // that hold the part
    constexpr int kPlaceBits = W == 4 ? 7 : 8;
    constexpr unsigned kTop = (1u << (32 - kPlaceBits)) - 1u;
    const float span = W == 4 ? 33554426.f : 16777212.f;  // below kTop
    static_assert(W == 4 || W == 8, "parts of 128 or 256");
    float best_lo = 0.f, best_ext = -1.f;
    int dim = 0;
    for (int c = 0; c < cd; c++) {
        float lo = INFINITY, hi = -INFINITY;
#pragma unroll
        for (int r = 0; r < W; r++)
            if (li[r] < n_here) {
                const float x = s_w[c * kSuper + li[r]];
                lo = fminf(lo, x);
                hi = fmaxf(hi, x);
            }
        if (LEVEL == 0) {
            lo = warp_min_f32(lo);
            hi = warp_max_f32(hi);
        } else {
#pragma unroll
            for (int o = 1; o < kLanes; o <<= 1) {
                lo = fminf(lo, __shfl_xor_sync(0xffffffffu, lo, o));
                hi = fmaxf(hi, __shfl_xor_sync(0xffffffffu, hi, o));
            }
        }
        if (hi - lo > best_ext) { best_ext = hi - lo; best_lo = lo; dim = c; }
    }
    const float scale = best_ext > 0.f ? span / best_ext : 0.f;
    unsigned w[W];
#pragma unroll
    for (int r = 0; r < W; r++) {
        w[r] = kTop;
        if (li[r] < n_here) w[r] = (unsigned)fminf(fmaxf((s_w[dim * kSuper + li[r]] - best_lo) * scale, 0.f), span);
        w[r] = (w[r] << kPlaceBits) | (unsigned)li[r];
    }
    sort_parts<kLanes * W, W>(w, lane);
#pragma unroll
    for (int r = 0; r < W; r++) li[r] = (int)(w[r] & ((1u << kPlaceBits) - 1u));
}

template <int W>
__global__ void __launch_bounds__(kSuper / W)
pack_tiles_kernel(const float *__restrict__ coords, int C, const int *__restrict__ perm,
                  const int *__restrict__ rank_of,
                  const int *__restrict__ direction, int n_events, HitOrder o, TileScratch s, int nv4, int nobody)
{
    pdl_begin();
    constexpr int kPart = 32 * W, kWarpsHere = kSuper / kPart;
    extern __shared__ float s_c[];  // [min(C, kSplitDims)][1024] coordinates in curve order
    __shared__ float s_lo[kWarpsHere][16], s_hi[kWarpsHere][16];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int sup = blockIdx.x;
    if (sup == 0 && warp == kWarpsHere - 1) {  // the chunk that holds no hits
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
    const int local0 = (sup - o.event_super[e]) * kSuper + warp * kPart;
    const int pos0 = o.event_pos[e] + local0;
    const int n_here = min(o.event_pos[e + 1] - pos0, kPart);  // below one: nothing for this warp
    const int cd = min(C, kSplitDims);
    float *__restrict__ s_w = s_c + warp * kPart;
    int id[W], li[W];  // hit and place in the part, of the places lane * W ..
#pragma unroll
    for (int r = 0; r < W; r++) {
        li[r] = lane * W + r;
        id[r] = li[r] < n_here ? perm[pos0 + li[r]] : -1;
    }
#pragma unroll
    for (int r = 0; r < W; r++)
        for (int c = 0; c < cd; c++) s_w[c * kSuper + li[r]] = id[r] >= 0 ? coords[(size_t)id[r] * C + c] : 0.f;
    __syncwarp();
    if (n_here > 32) {
        split_part<0, W>(s_w, cd, n_here, lane, li);
        split_part<1, W>(s_w, cd, n_here, lane, li);
        if constexpr (W >= 8) split_part<2, W>(s_w, cd, n_here, lane, li);
#pragma unroll
        for (int r = 0; r < W; r++) id[r] = li[r] < n_here ? perm[pos0 + li[r]] : -1;
    }

    // 32 / W lanes hold a chunk now
    constexpr int kLanes = 32 / W;
    const int chunk = chunk0 + local0 / 32 + lane / kLanes;
    const bool have = chunk < chunk1;
    const size_t at = (size_t)chunk * 32 + (lane % kLanes) * W;
    bool usable[W];
#pragma unroll
    for (int r = 0; r < W; r++) {
        usable[r] = id[r] >= 0;
        if (direction != nullptr && usable[r]) {
            const int d = direction[id[r]];
            usable[r] = !(d == 1 || d == 2);  // may not be anybody's neighbour
        }
    }
    if (have) {
        int rank[W];
#pragma unroll
        for (int r = 0; r < W; r++) rank[r] = id[r] >= 0 ? rank_of[id[r]] : 0;
#pragma unroll
        for (int r = 0; r < W; r += 4) {
            *reinterpret_cast<int4 *>(s.ids + at + r) = make_int4(id[r], id[r + 1], id[r + 2], id[r + 3]);
            *reinterpret_cast<int4 *>(s.ranks + at + r) = make_int4(rank[r], rank[r + 1], rank[r + 2], rank[r + 3]);
        }
        if (lane % kLanes == 0) {
            // hits beyond the last event take part in nothing
            const bool none = e == n_events;
            s.chunk_info[chunk] = make_int4(chunk0, none ? chunk0 : chunk1, o.event_super[e], o.event_super[e + 1]);
        }
    }
    const float nan = __int_as_float(0x7fffffff);
    for (int u = 0; u < nv4; u++) {
        float p[W][4], lo[4], hi[4];
#pragma unroll
        for (int k = 0; k < 4; k++) {
            const int d = u * 4 + k;
            lo[k] = INFINITY;
            hi[k] = -INFINITY;
#pragma unroll
            for (int r = 0; r < W; r++) {
                p[r][k] = 0.f;
                if (d < C && id[r] >= 0) p[r][k] = d < cd ? s_w[d * kSuper + li[r]] : coords[(size_t)id[r] * C + d];
                if (usable[r]) {
                    lo[k] = fminf(lo[k], p[r][k]);
                    hi[k] = fmaxf(hi[k], p[r][k]);
                } else {
                    p[r][k] = nan;
                }
            }
#pragma unroll
            for (int j = 1; j < kLanes; j <<= 1) {
                lo[k] = fminf(lo[k], __shfl_xor_sync(0xffffffffu, lo[k], j));
                hi[k] = fmaxf(hi[k], __shfl_xor_sync(0xffffffffu, hi[k], j));
            }
        }
        if (have) {
#pragma unroll
            for (int r = 0; r < W; r++) s.pts[(at + r) * nv4 + u] = make_float4(p[r][0], p[r][1], p[r][2], p[r][3]);
            if (lane % kLanes == 0) {
                s.chunk_box[((size_t)chunk * nv4 + u) * 2] = make_float4(lo[0], lo[1], lo[2], lo[3]);
                s.chunk_box[((size_t)chunk * nv4 + u) * 2 + 1] = make_float4(hi[0], hi[1], hi[2], hi[3]);
            }
        }
#pragma unroll
        for (int k = 0; k < 4; k++) {
            const float l = warp_min_f32(lo[k]), h = warp_max_f32(hi[k]);
            if (lane == 0) { s_lo[warp][u * 4 + k] = l; s_hi[warp][u * 4 + k] = h; }
        }
    }
    __syncthreads();
    for (int u = warp; u < nv4; u += kWarpsHere) {
        float lo[4], hi[4];
#pragma unroll
        for (int k = 0; k < 4; k++) {
            lo[k] = warp_min_f32(s_lo[lane % kWarpsHere][u * 4 + k]);
            hi[k] = warp_max_f32(s_hi[lane % kWarpsHere][u * 4 + k]);
        }
        if (lane == 0) {
            s.super_box[((size_t)sup * nv4 + u) * 2] = make_float4(lo[0], lo[1], lo[2], lo[3]);
            s.super_box[((size_t)sup * nv4 + u) * 2 + 1] = make_float4(hi[0], hi[1], hi[2], hi[3]);
        }
    }
}

}  // namespace

int build_tiles(const float *coords, int n_coords, const int *curve_perm, const int *rank_of, const HitOrder &o,
                int n_events, const int *direction, const TileScratch &s, int n_vert, cudaStream_t stream)
{
    if (n_vert <= 0) return HGC_OK;
    const size_t smem = sizeof(float) * kSuper * (n_coords < kSplitDims ? n_coords : kSplitDims);
#define HGC_PACK(W) HGC_CUDA_TRY(launch_overlapped(n_vert, pack_tiles_kernel<W>, (int)tile_supers_cap(n_vert, n_events), kSuper / W, smem, stream, coords, n_coords, curve_perm, rank_of, direction, n_events, o, s, (n_coords + 3) / 4, (int)(tile_chunks_cap(n_vert, n_events) * 32)))
    // Parts of 256 where an event has many more hits than the curve has cells (6 bits per coordinate or fewer), which leaves runs
    // of 128 without an order of their own; elsewhere the longer chain per warp costs more.  Search and orders, us with parts of 128 /
    // 256: 300k hits 5 dimensions K = 12 1678 / 1633, 6 dimensions K = 64 3218 / 3181, 1 M 16138 / 15806; 100k 5 dimensions K = 12
    // 488 / 508; 300k 3 dimensions 499 / 499; 700 hits 36 / 43.
    if (n_coords >= 5 && n_vert / n_events >= 150000) HGC_PACK(8);
    else HGC_PACK(4);
#undef HGC_PACK
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
    // Queries per block: whole chunks share the list of one tile among most queries; smaller batches are cut finer, so that
    // every SM has work to the end.  A list costs little beside the queries in four dimensions and less in more, so the cut
    // goes on there while blocks are few rounds of what is resident (9 to 6 per SM).  us with 8 blocks per SM wanted everywhere /
    // with this rule, showers: 4 dimensions, K = 64, 25k hits 158 / 148, 50k 254 / 223, 80k 372 / 341, 130k 530 / 503; K = 32 50k 211 / 186; 5
    // dimensions, K = 48, 20k 180 / 162, 50k 387 / 328, 130k 861 / 817.  3 dimensions lose by it: 20k uniform hits 86 / 96.  4 dimensions, K < 24, 50k
    // showers in tiles of 32 / 16 (whole): K = 4 160 / 147, 16 178 / 165; 20k hits, K = 4 and 16, wanted 10 / 18: showers 96.8 / 95.4, 102.6 / 102.5,
    // uniform 98.4 / 97.9, 106.5 / 109.6, normal 115 / 108, 124 / 125.  K = 24 to 64, wanted 18 / 16: 20k K = 64 showers 132 / 126, uniform 146 /
    // 137, normal 170 / 165; 38k showers K = 24 to 64 154 / 161 to 188 / 191, uniform 160 / 152 to 211 / 199.  7 and more dimensions, of the time with 8
    // wanted (and chunks from parts of 1024): 8 dimensions, K = 16, 30k showers 0.63, uniform 0.85, normal 0.79; 50k 0.67, 0.95, 0.91; 70k 0.75,
    // 1.08, 1.05.
    const long long chunks = (long long)tile_chunks_cap(n_vert, n_events), sms = sm_count();
    const long long whole = sms * (n_coords <= 3 ? 8 : n_coords == 4 ? 30 : 40), cut = sms * (n_coords <= 3 ? 8 : n_coords == 4 ? (K < 24 ? 10 : 16) : 40);
    a.tile = 32;
    while (a.tile > 4 && chunks * (32 / a.tile) < (a.tile == 32 ? whole : cut)) a.tile >>= 1;
    // Tiles of 8 in large events of five and six dimensions (47k to 95k hits) do worse than both neighbours where hits lie evenly.
    // us for 70k hits in tiles of 32 with chunks cut from parts of 1024 / of 8 / 4 / 16: 5 dimensions, K = 16, showers 421 / 379 / 347 / 404, uniform 593 / 572 / 531 /
    // 550, normal 801 / 922 / 842 / 859; 6 dimensions, against the first, showers 0.84 / 0.77 / 0.89, uniform 1.16 / 1.00 / 1.04, normal 1.10 / 1.15 /
    // 1.04.  Five events of 14k, 5 dimensions, K = 48, showers: 8 360, 4 387.
    if (a.tile == 8 && n_vert / n_events >= 32768) a.tile = n_coords == 5 ? 4 : n_coords == 6 ? 16 : 8;
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
