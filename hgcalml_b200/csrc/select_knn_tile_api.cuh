// Interface of the tile search (select_knn_tile.cuh): the padded, boxed layout of the sorted hits and the
// calls that build and search it.
#pragma once
#include "common.cuh"
#include "hit_order.cuh"

namespace hgc {

struct TileKnnArgs {
    const float4 *pts;         // [chunks * 32][NV4]; NaN: padding, or a hit that may not be a neighbour
    const int *ids;            // [chunks * 32] hit number in the caller's order, -1 for padding
    const int *ranks;          // [chunks * 32] position in the bin-sorted order: ties fall to the lower one
    const int *rank_to_id;     // [n_vert] hit at a position of the bin-sorted order
    const float4 *chunk_box;   // [chunks][NV4][lo, hi]
    const float4 *super_box;   // [super-chunks][NV4][lo, hi]
    const int4 *chunk_info;    // [chunks]: the event's chunks [x, y) and super-chunks [z, w); x == y: no search
    const int *n_chunks;       // [1]
    const float *coords;       // the caller's coordinates when packed points may be NaN, else null
    const int *direction;      // [n_vert] in the caller's order, or null
    int *out_idx;              // [n_vert][K]
    float *out_dist;           // [n_vert][K]
    int n_coords, K, tf_compat;
    int nobody;                // first point of a chunk that holds no hits
    int tile;                  // queries per tile: 4, 8, 16 or 32
    float guess;               // factor on a neighbouring query's squared K-th distance
    float expo;                // 2 / coordinates (growth of the squared distance with the count)
};

template <int NV4>
int launch_tile_nv(const TileKnnArgs &a, int n_tiles, cudaStream_t stream);

// Upper bounds on the chunks and super-chunks of n_vert hits in n_events events plus one run of hits
// beyond the last event.
inline size_t tile_chunks_cap(int n_vert, int n_events) { return (size_t)(n_vert > 0 ? n_vert : 0) / 32 + n_events + 1; }
inline size_t tile_supers_cap(int n_vert, int n_events) { return tile_chunks_cap(n_vert, n_events) / 32 + n_events + 1; }

struct TileScratch {
    float4 *pts, *chunk_box, *super_box;
    int4 *chunk_info;
    int *ids, *ranks;
};

template <typename W>
inline TileScratch tile_scratch_layout(W &ws, int n_vert, int n_coords, int n_events)
{
    TileScratch s;
    const size_t nv4 = (n_coords + 3) / 4;
    const size_t chunks = tile_chunks_cap(n_vert, n_events), supers = tile_supers_cap(n_vert, n_events);
    s.pts = ws.template take<float4>((chunks + 1) * 32 * nv4);  // one chunk without hits at the end
    s.chunk_box = ws.template take<float4>(chunks * 2 * nv4);
    s.super_box = ws.template take<float4>(supers * 2 * nv4);
    s.chunk_info = ws.template take<int4>(chunks);
    s.ids = ws.template take<int>(chunks * 32);
    s.ranks = ws.template take<int>((chunks + 1) * 32);
    return s;
}

// Packs the hits (position p of the curve order is hit curve_perm[p], whose position in the bin-sorted order
// is rank_of[hit]) into chunks and computes the boxes.
int build_tiles(const float *coords, int n_coords, const int *curve_perm, const int *rank_of, const HitOrder &o,
                int n_events, const int *direction, const TileScratch &s, int n_vert, cudaStream_t stream);

// Searches: rows of d_indices / d_dist in the caller's order and numbering.
int search_tiles(const TileScratch &s, const HitOrder &o, const int *rank_to_id, const float *coords, int n_coords, const int *direction, int *out_idx,
                 float *out_dist, int n_vert, int n_events, int K, int tf_compat, cudaStream_t stream);

}  // namespace hgc
