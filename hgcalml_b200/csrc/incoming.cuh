// Transposed neighbour lists: for every hit, the (hit, slot) edges that point at it, in ascending
// (hit, slot) order.  Used by the ops that push values from a hit to its neighbours (backward ops,
// PushKnn) so that they need no floating-point atomics and sum in a fixed order.
#pragma once
#include "common.cuh"

namespace hgc {

constexpr int kWarpList = 512;  // longest list that a warp sorts in registers

struct Incoming {
    int *bounds;          // [n_vert + 2] incoming edges of hit m are edges[bounds[m] .. bounds[m + 1])
    int *long_lists;      // [1 + n_edges / (kWarpList + 1) + 1] number of hits with more than kWarpList incoming edges, and the hits
    int *scan;            // scratch of the prefix sum
    int *edges;           // [n_edges] edge ids e = hit * n_neigh + slot
    int *place;           // [n_edges] place of an edge in its target's list; scratch of the long sort afterwards
    unsigned *flags;      // [n_edges][2] scratch of the op: one bit per feature of a slab of 64
    float *rows;          // [n_vert][64] scratch of the op: rows of a slab (edge_rows_kernel)
};

template <typename W>
Incoming incoming_layout(W &ws, int n_vert, int n_neigh)
{
    const size_t n = n_vert > 0 ? n_vert : 0, ne = n * (size_t)(n_neigh > 0 ? n_neigh : 0);
    Incoming b;
    b.bounds = ws.template take<int>(n + 2);  // first, with long_lists: one memset clears both and the status word
    b.long_lists = ws.template take<int>(ne / (kWarpList + 1) + 2);
    b.scan = ws.template take<int>(scan_scratch_ints((int)n + 1));
    b.edges = ws.template take<int>(ne);
    b.place = ws.template take<int>(ne);
    b.flags = ws.template take<unsigned>(2 * ne);
    b.rows = ws.template take<float>(64 * n);
    return b;
}

struct IncomingSizer {
    Sizer s;
    template <typename T> T *take(size_t n) { s.take<T>(n); return nullptr; }
};

// Builds the lists; also clears the workspace's status word.
int build_incoming(const int *nidx, int n_vert, int n_neigh, const Incoming &b, unsigned *status, cudaStream_t stream);

}  // namespace hgc
