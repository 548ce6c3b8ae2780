// Wrapper-level BinnedSelectKnn: the whole Python function of modules/binned_select_knn_op.py:32-95
// (grid from the batch's coordinate range, BinByCoordinates, stable sort by bin, gathers, the
// neighbour search, index remap and scatter back to the caller's order) as one enqueue with no
// host round trip.  The search writes each row straight to the caller's row and numbering, which
// replaces IndexReplacer and the two scatter_nd calls.
#include "common.cuh"
#include "binning.cuh"
#include "hit_order.cuh"
#include "select_knn_tile_api.cuh"

namespace hgc {
namespace {

__global__ void gather_kernel(const int *__restrict__ src, const int *__restrict__ perm, int *__restrict__ dst, int n)
{
    pdl_begin();
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) dst[i] = src[perm[i]];
}

__global__ void invert_perm_kernel(const int *__restrict__ perm, int *__restrict__ inv, int n)
{
    pdl_begin();
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) inv[perm[i]] = i;
}

struct RaggedPlan {
    int cb;              // binned dimensions
    long long max_bins;  // upper bound on the number of bins of the device-derived grid
};

bool make_plan(int n_coords, int n_rs, int n_bins, int max_bin_dims, RaggedPlan *p)
{
    p->cb = max_bin_dims < n_coords ? max_bin_dims : n_coords;
    if (p->cb < 1 || p->cb > kMaxBinDims) return false;
    // bins per dimension = int(extent/width + 1) <= n_bins + 1; the default n_bins is at most 30
    const long long per_dim = (n_bins > 0 ? n_bins : 30) + 1;
    long long b = n_rs > 1 ? n_rs - 1 : 1;
    for (int d = 0; d < p->cb; d++) {
        b *= per_dim;
        if (b > (1LL << 30)) return false;
    }
    p->max_bins = b;
    return true;
}

}  // namespace
}  // namespace hgc

using namespace hgc;

namespace {

struct RaggedBuffers {
    HitOrder order;
    TileScratch tiles;
    int *bin_perm, *curve_perm, *rank;
    // orders by bin whose keys do not fit 32 bits (see wide_bins)
    int *keys, *subkeys, *k1, *v1, *tkeys, *tvals, *hist;
};

// A bin number inside an event and the 16-bit locality code make a 32-bit sort key up to 2^16 bins per event; finer
// grids (a bin count asked for by the caller, or four and five binned dimensions) are sorted in two steps.
bool wide_bins(const RaggedPlan &p, int n_events) { return p.max_bins / (n_events > 0 ? n_events : 1) > (1LL << 16); }

// One definition of the layout serves both the size query (Sizer) and the real carve (Carver).
template <typename W>
void layout(W &ws, int n_vert, int n_coords, int n_rs, const RaggedPlan &p, RaggedBuffers *b)
{
    const size_t n = n_vert > 0 ? n_vert : 0;
    const int n_events = n_rs > 1 ? n_rs - 1 : 0;
    RaggedBuffers t;
    t.order = hit_order_layout(ws, n_vert, n_events);
    t.tiles = tile_scratch_layout(ws, n_vert, n_coords, n_events);
    t.bin_perm = ws.template take<int>(n);
    t.curve_perm = ws.template take<int>(n);
    t.rank = ws.template take<int>(n);
    if (wide_bins(p, n_events)) {
        t.keys = ws.template take<int>(n);
        t.subkeys = ws.template take<int>(n);
        t.k1 = ws.template take<int>(n);
        t.v1 = ws.template take<int>(n);
        t.tkeys = ws.template take<int>(n);
        t.tvals = ws.template take<int>(n);
        t.hist = ws.template take<int>(sort_hist_ints(n_vert));
    }
    if (b) *b = t;
}

struct SizerW {
    Sizer s;
    template <typename T> T *take(size_t n) { s.take<T>(n); return nullptr; }
};

}  // namespace

extern "C" size_t hgc_binned_select_knn_ragged_workspace_bytes(int n_vert, int n_neigh, int n_coords,
                                                               int n_rs, int n_bins, int max_bin_dims)
{
    (void)n_neigh;
    RaggedPlan p;
    if (n_coords < 1 || !make_plan(n_coords, n_rs, n_bins, max_bin_dims, &p)) return 0;
    SizerW w;
    layout(w, n_vert, n_coords, n_rs, p, nullptr);
    return w.s.used;
}

extern "C" int hgc_binned_select_knn_ragged(
        const float *d_coords, const int *d_row_splits, const int *d_direction,
        int *d_indices, float *d_dist, int *d_sorting_out,
        int n_vert, int n_neigh, int n_coords, int n_rs,
        int n_bins, int max_bin_dims, int tf_compat, int use_direction,
        void *workspace, size_t workspace_bytes, hgc_stream_t stream_)
{
    cudaStream_t stream = static_cast<cudaStream_t>(stream_);
    if (n_vert < 0 || n_neigh < 1 || n_rs < 2 || n_coords < 2) return HGC_ERR_INVALID_ARGUMENT;
    RaggedPlan p;
    if (!make_plan(n_coords, n_rs, n_bins, max_bin_dims, &p)) return HGC_ERR_UNSUPPORTED;
    if (p.cb < 2) return HGC_ERR_INVALID_ARGUMENT;  // the op wants at least 2 binned dimensions
    if (p.cb > 5 || n_coords > 16 || n_neigh > 513) return HGC_ERR_UNSUPPORTED;
    if (n_vert == 0) return HGC_OK;
    if (!d_coords || !d_row_splits || !d_indices || !d_dist || (use_direction && !d_direction))
        return HGC_ERR_INVALID_ARGUMENT;
    const size_t need = hgc_binned_select_knn_ragged_workspace_bytes(n_vert, n_neigh, n_coords, n_rs,
                                                                     n_bins, max_bin_dims);
    if (int rc = check_workspace(workspace, workspace_bytes, need)) return rc;

    Carver ws(workspace);
    RaggedBuffers b;
    layout(ws, n_vert, n_coords, n_rs, p, &b);
    const int n_events = n_rs - 1;
    // the status word and the histograms of the sorts, which follow it
    HGC_CUDA_TRY(cudaMemsetAsync(ws.status(), 0, hit_order_zeroed_bytes(n_vert, n_events), stream));
    int *perm = d_sorting_out ? d_sorting_out : b.bin_perm;
    const bool wide = wide_bins(p, n_events);
    if (int rc = order_hits(d_coords, n_coords, p.cb, d_row_splits, n_rs, n_bins, n_neigh, n_vert,
                            wide ? 0 : bits_for(p.max_bins / (n_events > 0 ? n_events : 1) - 1), b.order, perm, b.rank,
                            b.curve_perm, ws.status(), stream))
        return rc;
    if (wide) {
        // two stable counting sorts, least significant key first
        const GridParams *g = b.order.grid;
        if (int rc = launch_bin_keys(d_coords, n_coords, p.cb, g->shift, d_row_splits, n_rs, &g->bin_width, g->n_bins,
                                     nullptr, nullptr, b.keys, n_vert, 0, &g->n_total_bins, ws.status(), stream, g,
                                     n_coords, b.subkeys))
            return rc;
        if (int rc = sort_pairs(b.subkeys, nullptr, b.k1, b.v1, b.tkeys, b.tvals, b.hist, n_vert, kSubBits, stream))
            return rc;
        HGC_CUDA_TRY(launch_pdl(gather_kernel, div_up(n_vert, 256), 256, 0, stream, b.keys, b.v1, b.k1, n_vert));
        HGC_LAUNCH_CHECK();
        if (int rc = sort_pairs(b.k1, b.v1, b.keys, perm, b.tkeys, b.tvals, b.hist, n_vert, bits_for(p.max_bins), stream))
            return rc;
        HGC_CUDA_TRY(launch_pdl(invert_perm_kernel, div_up(n_vert, 256), 256, 0, stream, perm, b.rank, n_vert));
        HGC_LAUNCH_CHECK();
    }
    const int *direction = use_direction ? d_direction : nullptr;
    if (int rc = build_tiles(d_coords, n_coords, b.curve_perm, b.rank, b.order, n_events, direction, b.tiles, n_vert, stream)) return rc;
    if (int rc = search_tiles(b.tiles, b.order, perm, d_coords, n_coords, direction, d_indices, d_dist, n_vert, n_rs - 1, n_neigh,
                              tf_compat, stream))
        return rc;
    return HGC_OK;
}
