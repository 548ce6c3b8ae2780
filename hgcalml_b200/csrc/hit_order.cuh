// The two orders of a ragged batch that the neighbour search works with, and the layout of its events.
#pragma once
#include "common.cuh"
#include "binning.cuh"

namespace hgc {

// Hits that a block of the sort works on: 256 threads times 2, 4 or 8; tiles never straddle events.  A pass over a few
// tiles is a chain of latencies that grows with the hits per thread; a pass over many is bound by throughput, and every
// block adds up the counts of the tiles before its own.  Keys and four passes at 20k hits: 48 us with 2048, 35 us with 512;
// at 200k 82 and 68 us with 2048 and 1024; at 400k the two are equal.
inline int order_tile(int n_vert) { return n_vert <= (1 << 15) ? 512 : n_vert <= (1 << 18) ? 1024 : 2048; }

struct HitOrder {
    int tile;             // order_tile
    GridParams *grid;
    float *partial;
    // [n_events + 2]: first position / sort tile / chunk of 32 / super-chunk of 1024 of every event; entry n_events
    // is the run of hits beyond the last event, entry n_events + 1 closes it
    int *event_pos, *event_tile, *event_chunk, *event_super;
    unsigned *key[2][2];  // [order][ping-pong] sort keys
    int *val[2][2];       // [order][ping-pong] hits
    int *tile_hist;       // [order][pass][tile][256] digit counts, zeroed
    int *event_hist;      // [order][pass][event][256], zeroed
};

constexpr int kOrderPasses = 4;  // 8-bit digits of a 32-bit key

inline size_t order_tiles_cap(int n_vert, int n_events) { return (size_t)(n_vert > 0 ? n_vert : 0) / order_tile(n_vert) + n_events + 1; }

template <typename W>
inline HitOrder hit_order_layout(W &ws, int n_vert, int n_events)
{
    HitOrder o;
    const size_t n = n_vert > 0 ? n_vert : 0, e = (size_t)n_events + 2;
    o.tile = order_tile(n_vert);
    // first, so that one memset clears them together with the status word
    o.tile_hist = ws.template take<int>(2 * kOrderPasses * order_tiles_cap(n_vert, n_events) * 256);
    o.event_hist = ws.template take<int>(2 * kOrderPasses * e * 256);
    o.grid = ws.template take<GridParams>(1);
    o.partial = ws.template take<float>((size_t)range_partial_blocks(n_vert) * 2 * kMaxBinDims);
    o.event_pos = ws.template take<int>(e);
    o.event_tile = ws.template take<int>(e);
    o.event_chunk = ws.template take<int>(e);
    o.event_super = ws.template take<int>(e);
    for (int s = 0; s < 2; s++)
        for (int b = 0; b < 2; b++) {
            o.key[s][b] = ws.template take<unsigned>(n);
            o.val[s][b] = ws.template take<int>(n);
        }
    return o;
}
inline size_t hit_order_zeroed_bytes(int n_vert, int n_events)
{
    Sizer s;
    s.take<int>(2 * kOrderPasses * order_tiles_cap(n_vert, n_events) * 256);
    s.take<int>(2 * kOrderPasses * ((size_t)n_events + 2) * 256);
    return s.used;
}

// Coordinate range and grid of the batch (o.grid, through o.partial) and the event layout (o.event_*).  status[8] counts
// the blocks that are done and must be zero.
int range_and_layout(const float *coords, int n_coords, int n_bin_dims, const int *row_splits, int n_rs, int n_bins,
                     int n_neigh, int n_vert, const HitOrder &o, unsigned *status, cudaStream_t stream);

// Event layout and both orders:
//   bin_perm[p]: hit at position p of the order by (event, bin, locality code, hit number); rank[hit] is its inverse
//   curve_perm[p]: hit at position p of the order by (event, position on a Hilbert curve, hit number)
// `o.grid` is of use afterwards only with bin_bits 0: the one kernel that orders small batches keeps the grid to itself.
// The sort clears nothing: `o`'s histograms and `status` must be zero.  bin_bits: bits of a bin number inside
// an event, at most 16; 0 for grids that need more, whose order by bin is left to the caller (bin_perm and rank are
// not written).
int order_hits(const float *coords, int n_coords, int n_bin_dims, const int *row_splits, int n_rs, int n_bins, int n_neigh,
               int n_vert, int bin_bits, const HitOrder &o, int *bin_perm, int *rank, int *curve_perm,
               unsigned *status, cudaStream_t stream);

}  // namespace hgc
