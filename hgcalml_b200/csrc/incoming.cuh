// Transposed neighbour lists: for every hit, the (hit, slot) edges that point at it, in ascending
// (hit, slot) order.  Used by the ops that push values from a hit to its neighbours (backward ops,
// PushKnn) so that they need no floating-point atomics and sum in a fixed order.
#pragma once
#include "common.cuh"

namespace hgc {

constexpr int kWarpList = 512;  // longest list that a warp sorts in registers

// Lists longer than this are wide, and whole blocks of edge_sum_kernel work on them: five or six times what a hit receives on
// average, which hardly any does whose neighbours are looked for among all hits.  (Up to 32768 hits such a list is what the
// others wait for.)  us without / with wide lists, PushKnn: 200k hits, K = 16, F = 32, one hit in 25 a neighbour 512 / 232, one in 10
// 306 / 260 (only lists of more than 512 edges: 532, 298); one in 4, where three times K for a line took 302, 243 / 186.  9000 hits, 20 of
// them neighbours of all others 114 / 46.  200k hits, K = 64, F = 64, one hit in 8 a neighbour 1136 / 1230 with 6 K, 1188 with 512.
inline int wide_list(int n_vert, int n_neigh)
{
    if (n_neigh > (n_vert <= (1 << 15) ? 102 : 42)) return kWarpList;
    return n_vert <= (1 << 15) ? (n_neigh <= 16 ? 80 : 5 * n_neigh) : (n_neigh <= 21 ? 127 : 6 * n_neigh);
}

// The hits with wide lists: those of more than kWarpList edges from the front, the others from the back.
struct WideLists {
    int limit;    // wide_list
    int *counts;  // [2] of more than kWarpList, of the others
    int *hits;
    int room;
};

struct Incoming {
    int *bounds;          // [n_vert + 2] incoming edges of hit m are edges[bounds[m] .. bounds[m + 1])
    WideLists wide;
    int *scan;            // scratch of the prefix sum
    int *edges;           // [n_edges] edge ids e = hit * n_neigh + slot
    unsigned *flags;      // [n_edges][2] scratch of the op: one bit per feature of a slab of 64
    int *place;           // [n_edges] place of an edge in its target's list; scratch of the long sort afterwards
    float *rows;          // scratch of the op: rows of a slab (edge_rows_kernel)
};

// Floats per hit that an op copies its rows into, a slab of up to 64 features at a time: none where rows are whole 16-byte vectors
// that need no division.
inline int copied_row(int n_feat, bool aligned, bool divided)
{
    if (n_feat % 4 == 0 && aligned && !divided) return 0;
    return n_feat < 64 ? (n_feat + 3) / 4 * 4 : 64;
}
inline bool aligned16(const void *p) { return (reinterpret_cast<uintptr_t>(p) & 15u) == 0; }
inline bool power_of_two(int k) { return (k & (k - 1)) == 0; }

// `row`: floats per hit of the copied rows.  They take the place of `place`, which the finished lists do not need, that of `flags`
// in an op without flags, and what they are longer than that behind it.
template <typename W>
Incoming incoming_layout(W &ws, int n_vert, int n_neigh, int row = 0, bool with_flags = true)
{
    const size_t n = n_vert > 0 ? n_vert : 0, ne = n * (size_t)(n_neigh > 0 ? n_neigh : 0);
    Incoming b;
    b.bounds = ws.template take<int>(n + 2);  // first, with the counts: one memset clears both and the status word
    b.wide.limit = wide_list((int)n, n_neigh);
    b.wide.room = (int)(ne / ((size_t)b.wide.limit + 1)) + 1;
    b.wide.counts = ws.template take<int>(2 + (size_t)b.wide.room);
    b.wide.hits = b.wide.counts + 2;
    b.scan = ws.template take<int>(scan_scratch_ints((int)n + 1));
    b.edges = ws.template take<int>(ne);
    b.flags = ws.template take<unsigned>(2 * ne);
    b.place = ws.template take<int>(ne);
    b.rows = with_flags ? reinterpret_cast<float *>(b.place) : reinterpret_cast<float *>(b.flags);
    const size_t room = with_flags ? ne : 3 * ne, want = n * (size_t)row;
    if (want > room) ws.template take<float>(want - room);
    return b;
}

struct IncomingSizer {
    Sizer s;
    template <typename T> T *take(size_t n) { s.take<T>(n); return nullptr; }
};
inline size_t incoming_bytes(int n_vert, int n_neigh, int row = 0, bool with_flags = true)
{
    IncomingSizer w;
    incoming_layout(w, n_vert, n_neigh, row, with_flags);
    return w.s.used;
}

// Builds the lists; also clears the workspace's status word.
int build_incoming(const int *nidx, int n_vert, int n_neigh, const Incoming &b, unsigned *status, cudaStream_t stream);

}  // namespace hgc
