// Wrapper-level BuildAndAssignCondensatesBinned: the Python function of modules/assign_condensate_op.py:245-310
// (threshold scaling, shift by the batch minimum, binning, sort by bin, high-beta filter, the op, mapping back,
// condensate flags) on the hits in the caller's order.
//
// The reference's loop takes the free high-beta hit with the largest beta, makes it a condensate and lets it claim
// what is inside its radius.  Only two things of the wrapper's preparation can be seen in the result: the shift of
// the coordinates (it rounds them), and the order by bin, which decides between hits of equal beta.  So no
// hit is moved: the high-beta hits alone are listed and sorted, by bin and then by beta, and every hit is tested
// where it is.
//
//   count_high, order_high   high-beta hits of every event, packed, with their sort keys
//   order_pass               stable sort by (event, beta descending, bin, hit), a launch per 8-bit digit
//   claim_grid               which of them are condensates, see there
//   list_condensates         their lists, in priority order and by grid cell
//   assign_hits              every hit against the condensates of the 27 cells around it
//
// The sort of all hits by bin, the gathers and the test of every hit against every condensate of its event
// are gone, and the claim pass settles some forty condensates per round instead of up to 32 per batch of a window.
#include <cooperative_groups.h>
#include "common.cuh"
#include "binning_device.cuh"
#include "condensates.cuh"
#include "hit_order.cuh"
#include "hit_order_device.cuh"
#include "../../include/hgcalml_b200.h"

namespace hgc {
namespace {

constexpr int kMaxCondDims = 8;
constexpr int kThreads = kOrderThreads;
constexpr int kWarps = kThreads / kWarp;
constexpr int kClusterBlocks = 8;
constexpr int kClaimThreads = 1024;
constexpr int kClaimStep = kClusterBlocks * kClaimThreads;
constexpr int kMaxCells = 13824;   // 24 per coordinate; a block keeps two words per cell in shared memory
constexpr int kMinCells = 64;      // the fewest that may be of use, see the two rules

// Claims by grid, or over windows of the priority order.  The grid spans three coordinates: fewer cells than 64 settle too
// few condensates per round, and with more coordinates than the grid has a cell holds hits that are far apart, of which
// only the first is settled.  4 x 200k hits, radius 1.0 on a range of 6 (216 cells): 3 coordinates 0.47 ms by grid; 4
// coordinates 1.74 ms and 1.56 over windows, 5 8.0 and 6.3, 8 69 and 48.  Radius 0.85 (512 cells): 4 2.0 by grid.
__device__ __forceinline__ bool claims_by_grid(int n_cells, int dims) { return n_cells >= (dims <= 3 ? kMinCells : 512); }
// Hits against the condensates of the 27 cells around them, or against all in priority order.  The distance fold walks the
// cells once for every condensate that covers the hit, more of them the more coordinates; all, only once.  4 x 200k hits,
// distance fold, 125 cells: 4 coordinates 1.47 ms by cell and 1.09 against all, 6 19.1 and 12.8; 216 cells: 4 2.22 and
// 2.20, 6 27.4 and 29.5.
__device__ __forceinline__ bool assigns_by_cell(int n_cells, int dims, bool by_max_beta)
{
    return n_cells >= (by_max_beta || dims <= 3 ? kMinCells : 150);
}

typedef unsigned long long u64;

// Grid over the condensates: cells at least as wide as the largest radius, over up to three coordinates.
struct CondGrid {
    int dims;        // gridded coordinates, 1 .. 3
    int n[3];        // cells per coordinate (1 beyond dims)
    float inv[3];    // cells per unit
};

struct Plan {
    int cb;             // binned dimensions
    int bin_passes;     // 8-bit digits of a bin number inside an event
    int n_bins_sc;
    int cells;          // upper bound on the grid cells per event
    int cells_per_dim;
    int max_settled;    // upper bound on cells of which no two touch
};

struct Buffers {
    // zeroed together with the status word
    int *tile_hist;       // [pass][tile][256]
    int *event_hist;      // [pass][event][256]
    int *count;           // [num_rows] condensates
    int *cell_count;      // [num_rows][cells + 1]
    unsigned *max_radius; // [1] bits of the largest radius
    // not zeroed
    HitOrder layout;      // only grid, partial and the event layout
    int *use_grid;        // [1]
    u64 *first_two;       // [2] smallest (bin, hit) keys of the high-beta hits
    int *tile_count, *row_splits_h;
    u64 *key[2];
    int *val[2];
    int *order;
    float *h_ccoords, *h_dist;
    int *h_mask, *h_orig, *status_h;
    float4 *p_rec;        // high-beta hits in priority order
    int *p_flag;          // their masks' signs (1: condensate that covers nothing, -1: cannot be covered), then their cells
    unsigned *open, *bitmap;
    CondList cl;
    int *alpha_h, *stage;
    float4 *c_rec;        // condensates by cell
    int *c_rank;
};

__device__ __forceinline__ CondGrid make_cond_grid(const GridParams *__restrict__ g, const unsigned *__restrict__ max_radius,
                                                   int dims, int cells_per_dim)
{
    // cells a little wider than the largest radius, so that what a condensate covers is at most one cell away whatever
    // the rounding
    const float width = __uint_as_float(*max_radius) * 1.001f;
    CondGrid c;
    c.dims = dims < 3 ? dims : 3;
#pragma unroll
    for (int d = 0; d < 3; d++) {
        c.n[d] = 1;
        c.inv[d] = 0.f;
        if (d < c.dims) {
            const float ext = g->range[d];
            const float w = fmaxf(width, ext / (float)cells_per_dim);
            if (ext > 0.f && w < ext) {
                c.inv[d] = 1.f / w;
                c.n[d] = min((int)(ext * c.inv[d]) + 1, cells_per_dim);
            }
        }
    }
    return c;
}

template <int NR>
__device__ __forceinline__ void cell_of(const CondGrid &c, const Rec<NR> &x, int (&at)[3])
{
#pragma unroll
    for (int d = 0; d < 3; d++)
        at[d] = d < rec_dims<NR>() ? min(max((int)(x.v[d] * c.inv[d]), 0), c.n[d] - 1) : 0;
}

// A hit is high if its beta is above the threshold or its mask is positive.
__device__ __forceinline__ bool is_high(const float *__restrict__ betas, const int *__restrict__ mask, int v, float threshold)
{
    return betas[v] > threshold || (mask && mask[v] > 0);
}

__device__ __forceinline__ unsigned bin_of(const float *__restrict__ ccoords, int dims, int cb, const GridParams *__restrict__ g,
                                           int v, unsigned *status)
{
    // as modules/compiled/bin_by_coordinates_kernel.cc:64-113
    unsigned flat = 0u;
    int stride = 1;
    for (int c = cb - 1; c >= 0; c--) {
        int ci = __float2int_rz(__fdiv_rn(__fsub_rn(ccoords[(size_t)v * dims + c], g->shift[c]), g->bin_width));
        const int nb = g->n_bins[c];
        if (ci < 0 || ci >= nb) {
            ci = 0;
            flag_status(status, HGC_STATUS_BIN_OUT_OF_RANGE);
        }
        flat += (unsigned)(ci * stride);
        stride *= nb;
    }
    return flat;
}

// High-beta hits of every tile; initial values of the outputs that later kernels fill in places.
__global__ void __launch_bounds__(kThreads)
count_high_kernel(const float *__restrict__ betas, const int *__restrict__ mask, float beta_threshold, HitOrder o,
                  int n_events, int *__restrict__ tile_count, int *__restrict__ alpha_out, unsigned char *__restrict__ is_cond,
                  u64 *__restrict__ first_two)
{
    pdl_begin();
    HitTile t;
    if (!find_tile(o, n_events, blockIdx.x, &t)) return;
    if (blockIdx.x == 0 && threadIdx.x < 2) first_two[threadIdx.x] = ~0ull;
    __shared__ int s_warp[kWarps];
    int n = 0;
    for (int i = threadIdx.x; i < t.n; i += kThreads) {
        const int v = t.first + i;
        n += t.event < n_events && is_high(betas, mask, v, beta_threshold) ? 1 : 0;
        alpha_out[v] = -1;
        is_cond[v] = 0;
    }
    n = __reduce_add_sync(0xffffffffu, n);
    if ((threadIdx.x & 31) == 0) s_warp[threadIdx.x >> 5] = n;
    __syncthreads();
    if (threadIdx.x == 0) {
        for (int w = 1; w < kWarps; w++) n += s_warp[w];
        tile_count[blockIdx.x] = n;
    }
}

// The first (SECOND: the second) high-beta hit of the batch in the order by bin.  Only run when there is a mask: the
// reference's pick loop tests no_condensation_mask_h at index 0 or 1 of that order instead of at the hit
// (binned_assign_to_condensates_kernel.cc:193).
template <bool SECOND>
__global__ void __launch_bounds__(kThreads)
first_high_kernel(const float *__restrict__ ccoords, const float *__restrict__ betas, const int *__restrict__ mask,
                  float beta_threshold, int dims, int cb, HitOrder o, int n_events, u64 *__restrict__ first_two)
{
    pdl_begin();
    HitTile t;
    if (!find_tile(o, n_events, blockIdx.x, &t) || t.event >= n_events) return;
    const u64 first = SECOND ? first_two[0] : 0ull;
    for (int i = threadIdx.x; i < t.n; i += kThreads) {
        const int v = t.first + i;
        if (!is_high(betas, mask, v, beta_threshold)) continue;
        const u64 flat = (u64)t.event * (unsigned)o.grid->bins_per_event + bin_of(ccoords, dims, cb, o.grid, v, nullptr);
        const u64 key = flat << 31 | (unsigned)v;
        if (!SECOND || key > first) atomicMin(first_two + (SECOND ? 1 : 0), key);
    }
}

// Packs the high-beta hits of every event (in the caller's order) with what the claim pass needs and their sort keys:
// beta in the high word, bin in the low one.
__global__ void __launch_bounds__(kThreads)
order_high_kernel(const float *__restrict__ ccoords, const float *__restrict__ betas, const float *__restrict__ dist,
                  const int *__restrict__ mask, float beta_threshold, float distance_threshold, int dims, int cb,
                  int bin_passes, int n_events, Buffers b, unsigned *status)
{
    pdl_begin();
    extern __shared__ int s_hist[];  // [passes][256]
    __shared__ int s_warp[kWarps];
    __shared__ int s_base;
    const HitOrder &o = b.layout;
    const int n_tiles = o.event_tile[n_events + 1], passes = bin_passes + 4;
    if (blockIdx.x == 0) {
        // row splits of the packed hits
        int carry = 0;
        for (int base = 0; base < n_tiles; base += kThreads) {
            const int q = base + threadIdx.x;
            const int n = q < n_tiles ? b.tile_count[q] : 0;
            const int incl = carry + block_scan_inclusive(n, [](int x, int y) { return x + y; }, 0, s_warp);
            if (q < n_tiles) b.stage[q] = incl;
            __syncthreads();
            if (threadIdx.x == kThreads - 1) s_base = incl;
            __syncthreads();
            carry = s_base;
        }
        __syncthreads();
        for (int e = threadIdx.x; e <= n_events; e += kThreads) {
            const int q = o.event_tile[e];
            b.row_splits_h[e] = q > 0 ? b.stage[q - 1] : 0;
        }
        __syncthreads();
    }
    HitTile t;
    if (!find_tile(o, n_events, blockIdx.x, &t) || t.event >= n_events) return;
    int before = 0, event_start = 0;
    const int tile0 = o.event_tile[t.event];
    for (int q = threadIdx.x; q < (int)blockIdx.x; q += kThreads) {
        const int n = b.tile_count[q];
        before += n;
        event_start += q < tile0 ? n : 0;
    }
    __shared__ int s_sum[2];
    if (threadIdx.x < 2) s_sum[threadIdx.x] = 0;
    for (int i = threadIdx.x; i < passes * 256; i += kThreads) s_hist[i] = 0;
    __syncthreads();
    before = __reduce_add_sync(0xffffffffu, before);
    event_start = __reduce_add_sync(0xffffffffu, event_start);
    if ((threadIdx.x & 31) == 0) { atomicAdd(&s_sum[0], before); atomicAdd(&s_sum[1], event_start); }
    __syncthreads();
    int run = s_sum[0];
    const int start = s_sum[1];
    float radius_max = 0.f;
    for (int i0 = 0; i0 < t.n; i0 += kThreads) {
        const int i = i0 + threadIdx.x, v = t.first + i;
        const bool high = i < t.n && is_high(betas, mask, v, beta_threshold);
        const int incl = block_scan_inclusive(high ? 1 : 0, [](int x, int y) { return x + y; }, 0, s_warp);
        if (high) {
            const int a = run + incl - 1;
            const int m = mask ? mask[v] : 0;
            const float radius = __fdiv_rn(dist[v], distance_threshold);
            for (int c = 0; c < dims; c++)
                b.h_ccoords[(size_t)a * dims + c] = __fsub_rn(ccoords[(size_t)v * dims + c], o.grid->all_min[c]);
            b.h_dist[a] = radius;
            b.h_mask[a] = m;
            b.h_orig[a] = v;
            b.status_h[a] = 0;
            if (m <= 0) radius_max = fmaxf(radius_max, fabsf(radius));
            bool flagged = false;
            if (mask) {
                const int id0 = (int)(b.first_two[0] & 0x7fffffffull), id1 = (int)(b.first_two[1] & 0x7fffffffull);
                flagged = mask[v == id0 ? id0 : id1] != 0;  // there is a second one when v is not the first
            }
            const u64 key = (u64)priority_key(betas[v], flagged) << 32 | bin_of(ccoords, dims, cb, o.grid, v, status);
            b.key[0][a] = key;
            for (int p = 0; p < passes; p++) {
                const int shift = p < bin_passes ? 8 * p : 32 + 8 * (p - bin_passes);
                atomicAdd(&s_hist[p * 256 + (int)((key >> shift) & 255u)], 1);
            }
            // the packed hits make tiles of their own
            atomicAdd(&b.tile_hist[(size_t)(tile0 + (a - start) / o.tile) * 256 + (int)(key & 255u)], 1);
        }
        __syncthreads();
        if (threadIdx.x == kThreads - 1) s_base = incl;
        __syncthreads();
        run += s_base;
    }
    radius_max = __uint_as_float(__reduce_max_sync(0xffffffffu, __float_as_uint(radius_max)));
    if ((threadIdx.x & 31) == 0 && radius_max > 0.f) atomicMax(b.max_radius, __float_as_uint(radius_max));
    __syncthreads();
    for (int p = 0; p < passes; p++) {
        const int c = s_hist[p * 256 + threadIdx.x];
        if (c) atomicAdd(&b.event_hist[((size_t)p * (n_events + 1) + t.event) * 256 + threadIdx.x], c);
    }
}

// One pass of the stable sort of the packed hits, event by event (see hit_order.cu).  The last pass (NR > 0) writes the
// order, and the hits' records in that order.
template <int kRounds, bool FIRST, int NR>
__global__ void __launch_bounds__(kThreads)
order_pass_kernel(Buffers b, int n_events, int tiles_cap, int pass, int shift, int next_shift, int dims)
{
    pdl_begin();
    constexpr int kTile = kRounds * kThreads;
    __shared__ int s_count[kWarps][256];
    __shared__ int s_warp[kWarps];
    const HitOrder &o = b.layout;
    if ((int)blockIdx.x >= o.event_tile[n_events]) return;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, d = threadIdx.x;
    const int e = event_of_tile(o.event_tile, n_events, blockIdx.x);
    const int off = b.row_splits_h[e], n_h = b.row_splits_h[e + 1] - off;
    const int local = ((int)blockIdx.x - o.event_tile[e]) * kTile;
    const int n = min(n_h - local, kTile);
    if (n <= 0) return;
    const u64 *__restrict__ key_in = b.key[pass & 1] + off + local;
    const int *__restrict__ val_in = b.val[pass & 1] + off + local;
    u64 key[kRounds];
    int val[kRounds];
    const int warp_base = warp * (kRounds * kWarp);
#pragma unroll
    for (int r = 0; r < kRounds; r++) {
        const int i = warp_base + r * kWarp + lane;
        key[r] = i < n ? key_in[i] : 0ull;
        val[r] = FIRST ? off + local + i : i < n ? val_in[i] : 0;
    }
    int start = off;
    {
        const int mine = b.event_hist[((size_t)pass * (n_events + 1) + e) * 256 + d];
        start += block_scan_inclusive(mine, [](int x, int y) { return x + y; }, 0, s_warp) - mine;
        const int *__restrict__ h = b.tile_hist + (size_t)pass * tiles_cap * 256 + d;
        int sum = 0;
#pragma unroll 16
        for (int q = o.event_tile[e]; q < (int)blockIdx.x; q++) sum += h[(size_t)q * 256];
        start += sum;
    }
#pragma unroll
    for (int w = 0; w < kWarps; w++) s_count[w][d] = 0;
    unsigned peers[kRounds];
#pragma unroll
    for (int r = 0; r < kRounds; r++) {
        const unsigned dg = warp_base + r * kWarp + lane < n ? (unsigned)(key[r] >> shift) & 255u : 256u;
        peers[r] = __match_any_sync(0xffffffffu, dg);
    }
    __syncthreads();
    int place[kRounds];
#pragma unroll
    for (int r = 0; r < kRounds; r++) {
        const bool ok = warp_base + r * kWarp + lane < n;
        const unsigned dg = (unsigned)(key[r] >> shift) & 255u, before = peers[r] & ((1u << lane) - 1u);
        const int seen = ok ? s_count[warp][dg] : 0;
        place[r] = seen + __popc(before);
        __syncwarp();
        if (ok && before == 0u) s_count[warp][dg] = seen + __popc(peers[r]);
        __syncwarp();
    }
    __syncthreads();
#pragma unroll
    for (int w = 0; w < kWarps; w++) {
        const int c = s_count[w][d];
        s_count[w][d] = start;
        start += c;
    }
    __syncthreads();
    int *__restrict__ next_hist = b.tile_hist + (size_t)(pass + 1) * tiles_cap * 256;
    const int tile0 = o.event_tile[e];
#pragma unroll
    for (int r = 0; r < kRounds; r++) {
        if (warp_base + r * kWarp + lane < n) {
            const int dst = s_count[warp][(unsigned)(key[r] >> shift) & 255u] + place[r];
            if constexpr (NR > 0) {
                const int a = val[r], m = b.h_mask[a];
                b.order[dst] = a;
                Rec<NR> x;
#pragma unroll
                for (int c = 0; c < NR * 4; c++) x.v[c] = 0.f;
#pragma unroll
                for (int c = 0; c < rec_dims<NR>(); c++)
                    if (c < dims) x.v[c] = b.h_ccoords[(size_t)a * dims + c];
                x.v[rec_r2_slot<NR>()] = __fmul_rn(b.h_dist[a], b.h_dist[a]);
                store_rec<NR>(b.p_rec + (size_t)dst * NR, x);
                b.p_flag[dst] = (m > 0) - (m < 0);
            } else {
                b.key[(pass + 1) & 1][dst] = key[r];
                b.val[(pass + 1) & 1][dst] = val[r];
                const int q = tile0 + (dst - off) / kTile;
                atomicAdd(&next_hist[(size_t)q * 256 + ((unsigned)(key[r] >> next_shift) & 255u)], 1);
            }
        }
    }
}

// Which of the high-beta hits are condensates: those that no condensate earlier in the priority order covers.  A cluster
// of 8 blocks per event (one block where there are many events), in rounds.  A hit that comes first among the open hits
// of its own cell and of the cells around it cannot be covered by an open one, so the first open hits of all cells that
// are first among their neighbours are settled together; then every open hit that one of them covers is closed.  500
// blobs on 2700 cells take about 13 rounds.  Masked hits (mask > 0) are condensates from the start: nothing covers them
// and they cover nothing; hits with a negative mask cover others but are not covered.
//
// Everything a round looks up is in shared memory: every block keeps the first open hit of every cell among its own hits,
// the blocks merge those tables (an eighth of the cells each) through distributed shared memory, and every block works
// out for itself which are settled and copies their records.  A round is two cluster barriers.  With the tables and
// records in L2 a round took 24 us, most of it in dependent loads, before (64k open hits per event).
// A round costs that much however many hits it settles, so grids that settle few are left to the windows of claim_kernel
// (claims_by_grid).
template <int NR, int CB>
__global__ void __cluster_dims__(CB, 1, 1) __launch_bounds__(kClaimThreads)
claim_grid_kernel(Buffers b, int dims, int cells_cap, int cells_per_dim, int max_settled)
{
    pdl_begin();
    constexpr int kStep = CB * kClaimThreads;  // hits of an event looked at together
    namespace cg = cooperative_groups;
    cg::cluster_group cluster = cg::this_cluster();
    extern __shared__ int s_dyn[];
    __shared__ int s_left[2][CB];
    __shared__ int s_count, s_sum, s_listed;
    int *s_best = s_dyn, *s_min = s_dyn + cells_cap;               // cells_cap is a multiple of 4
    float4 *s_rec = reinterpret_cast<float4 *>(s_min + cells_cap);  // [max_settled][NR]
    int *s_pos = reinterpret_cast<int *>(s_rec + (size_t)max_settled * NR), *s_at = s_pos + max_settled;
    const CondGrid grid = make_cond_grid(b.layout.grid, b.max_radius, dims, cells_per_dim);
    const int n_cells = grid.n[0] * grid.n[1] * grid.n[2];
    const bool use = claims_by_grid(n_cells, dims);
    if (blockIdx.x == 0 && threadIdx.x == 0) *b.use_grid = use ? 1 : 0;
    if (!use) return;  // the same in every block
    constexpr int U = NR == 1 ? 4 : NR == 2 ? 2 : 1;  // hits whose data is requested together
    constexpr int kFree = 0x7fffffff;
    const int e = blockIdx.x / CB, t = threadIdx.x, lane = t & 31;
    const int rank = (int)cluster.block_rank();
    const int g = rank * kClaimThreads + t;
    const int off = b.row_splits_h[e], n_h = b.row_splits_h[e + 1] - off;
    if (n_h == 0) return;  // all blocks of the cluster
    const int n_steps = (n_h + kStep - 1) / kStep;
    const int word0 = off / 32 + e;
    const float4 *__restrict__ recs = b.p_rec + (size_t)off * NR;
    int *__restrict__ cells = b.p_flag + off;
    unsigned *__restrict__ open_words = b.open + (size_t)word0 * 32 + g;  // word w of this thread: [w * kStep], w > 0

    for (int c = t; c < n_cells; c += kClaimThreads) s_best[c] = kFree;
    if (t == 0) s_count = s_sum = s_listed = 0;
    // this thread's hits are p = k * kStep + g; 32 of them share a word of open bits, kept in memory beyond the first
    unsigned open0 = 0u;
    int n_mine = 0;  // condensates among them
    for (int k = 0; k < n_steps; k++) {
        const int p = k * kStep + g;
        bool is_open = false, lonely = false;
        if (p < n_h) {
            const int flag = cells[p];
            const Rec<NR> x = load_rec<NR>(recs + (size_t)p * NR);
            int at[3];
            cell_of<NR>(grid, x, at);
            // cell coordinates in 8 bits each (7 for the first); the sign bit: cannot be covered
            cells[p] = at[0] << 16 | at[1] << 8 | at[2] | (flag != 0 ? (int)0x80000000 : 0);
            lonely = flag > 0;
            is_open = !lonely;
        }
        if ((k & 31) == 0 && k > 0) open_words[(size_t)(k / 32) * kStep] = 0u;
        if (is_open) {
            if (k < 32) open0 |= 1u << k;
            else open_words[(size_t)(k / 32) * kStep] |= 1u << (k & 31);
        }
        n_mine += lonely ? 1 : 0;
        const unsigned bits = __ballot_sync(0xffffffffu, lonely);
        if (lane == 0 && p < n_h) b.bitmap[word0 + p / 32] = bits;
    }
    __syncthreads();
    auto flat = [&grid](int at) { return (((at >> 16) & 127) * grid.n[1] + ((at >> 8) & 255)) * grid.n[2] + (at & 255); };
    const int slice = (n_cells + CB - 1) / CB;

    for (int round = 0;; round++) {
        // first open hit of every cell, among this block's
        for (int w = 0; w * 32 < n_steps; w++) {
            unsigned u = w == 0 ? open0 : open_words[(size_t)w * kStep];
            while (u) {
                int p[U], at[U];
#pragma unroll
                for (int q = 0; q < U; q++) {
                    p[q] = u ? (w * 32 + __ffs(u) - 1) * kStep + g : -1;
                    u &= u - 1u;
                }
#pragma unroll
                for (int q = 0; q < U; q++) at[q] = p[q] >= 0 ? cells[p[q]] : 0;
#pragma unroll
                for (int q = 0; q < U; q++)
                    if (p[q] >= 0) {
                        const int c = flat(at[q]);
                        if (s_best[c] > p[q]) atomicMin(s_best + c, p[q]);
                    }
            }
        }
        cluster.sync();
        if (round > 0) {
            int total = 0;
#pragma unroll
            for (int r = 0; r < CB; r++) total += s_left[(round - 1) & 1][r];
            // the same in every block of the cluster, and nobody looks at another block from here on: a block that leaves
            // while others may still write to its shared memory faults them.  (A round settles a hit at least.)
            if (total == 0 || round > n_h) break;
        }
        // merged, for all blocks
        for (int c = rank * slice + t; c < min((rank + 1) * slice, n_cells); c += kClaimThreads) {
            int v[CB], m = kFree;
#pragma unroll
            for (int r = 0; r < CB; r++) v[r] = *cluster.map_shared_rank(s_best + c, r);
#pragma unroll
            for (int r = 0; r < CB; r++) m = min(m, v[r]);
#pragma unroll
            for (int r = 0; r < CB; r++) *cluster.map_shared_rank(s_min + c, r) = m;
        }
        cluster.sync();
        // which of them are first among the cells around: occupied cells are listed first, since later rounds have few
        for (int c0 = t - lane; c0 < n_cells; c0 += kClaimThreads) {
            const int c = c0 + lane;
            const bool occupied = c < n_cells && s_min[c] != kFree;
            const unsigned m = __ballot_sync(0xffffffffu, occupied);
            int base = 0;
            if (lane == 0 && m) base = atomicAdd(&s_listed, __popc(m));
            base = __shfl_sync(0xffffffffu, base, 0);
            if (occupied) s_best[base + __popc(m & ((1u << lane) - 1u))] = c;  // the merged table has its place
        }
        __syncthreads();
        const int n_listed = s_listed;
        for (int i0 = t; i0 < n_listed; i0 += kClaimThreads) {
            const int c = s_best[i0], p = s_min[c];
            const int z = c % grid.n[2], y = c / grid.n[2] % grid.n[1], x = c / (grid.n[2] * grid.n[1]);
            bool first = true;
            for (int i = max(x - 1, 0); first && i <= min(x + 1, grid.n[0] - 1); i++)
                for (int j = max(y - 1, 0); first && j <= min(y + 1, grid.n[1] - 1); j++) {
                    const int *row = s_min + (i * grid.n[1] + j) * grid.n[2];
                    first = row[max(z - 1, 0)] >= p && row[z] >= p && row[min(z + 1, grid.n[2] - 1)] >= p;
                }
            if (first) {
                const int s = atomicAdd(&s_count, 1);  // in any order
                s_pos[s] = p;
                s_at[s] = x << 16 | y << 8 | z;
                store_rec<NR>(s_rec + (size_t)s * NR, load_rec<NR>(recs + (size_t)p * NR));
            }
        }
        __syncthreads();
        // and, for every cell, which of the 27 cells around it hold one (no two next to each other do): s_min takes
        // those bits, s_best of a cell that holds one its number
        for (int c = t; c < n_cells; c += kClaimThreads) s_min[c] = 0;
        __syncthreads();
        for (int i = t; i < s_count * 27; i += kClaimThreads) {
            const int s = i / 27, k = i % 27, at = s_at[s];
            const int x = (at >> 16) + k / 9 - 1, y = ((at >> 8) & 255) + k / 3 % 3 - 1, z = (at & 255) + k % 3 - 1;
            if (x < 0 || x >= grid.n[0] || y < 0 || y >= grid.n[1] || z < 0 || z >= grid.n[2]) continue;
            const int c = (x * grid.n[1] + y) * grid.n[2] + z;
            atomicOr(s_min + c, 1 << (26 - k));  // seen from there, the cell is on the opposite side
            if (k == 13) s_best[c] = s;
        }
        __syncthreads();
        // close them and what they cover
        int left = 0;
        for (int w = 0; w * 32 < n_steps; w++) {
            unsigned word = w == 0 ? open0 : open_words[(size_t)w * kStep], u = word;
            while (u) {
                int bit[U], at[U], near_[U];
                Rec<NR> mine[U];
#pragma unroll
                for (int q = 0; q < U; q++) {
                    bit[q] = u ? __ffs(u) - 1 : -1;
                    u &= u - 1u;
                }
#pragma unroll
                for (int q = 0; q < U; q++) at[q] = bit[q] >= 0 ? cells[(w * 32 + bit[q]) * kStep + g] : 0;
#pragma unroll
                for (int q = 0; q < U; q++) {
                    near_[q] = bit[q] >= 0 ? s_min[flat(at[q])] : 0;
                    if (near_[q]) mine[q] = load_rec<NR>(recs + (size_t)((w * 32 + bit[q]) * kStep + g) * NR);
                }
#pragma unroll
                for (int q = 0; q < U; q++) {
                    if (near_[q] == 0) continue;
                    const int p = (w * 32 + bit[q]) * kStep + g;
                    const int x = (at[q] >> 16) & 127, y = (at[q] >> 8) & 255, z = at[q] & 255;
                    bool stays = true;
                    if ((near_[q] >> 13) & 1) {  // one in its own cell
                        if (s_pos[s_best[flat(at[q])]] == p) {
                            atomicOr(b.bitmap + word0 + p / 32, 1u << (p & 31));
                            n_mine++;
                            stays = false;
                        }
                    }
                    if (at[q] >= 0)
                        for (int m = near_[q]; m && stays; m &= m - 1) {
                            const int k = __ffs(m) - 1;
                            const int s = s_best[((x + k / 9 - 1) * grid.n[1] + y + k / 3 % 3 - 1) * grid.n[2] + z + k % 3 - 1];
                            const Rec<NR> c = load_rec<NR>(s_rec + (size_t)s * NR);
                            if (rec_distsq<NR>(c, mine[q], dims) <= c.v[rec_r2_slot<NR>()]) stays = false;
                        }
                    if (!stays) word &= ~(1u << bit[q]);
                }
            }
            if (w == 0) open0 = word;
            else open_words[(size_t)w * kStep] = word;
            left += __popc(word);
        }
        left = __reduce_add_sync(0xffffffffu, left);
        if (lane == 0 && left) atomicAdd(&s_sum, left);
        __syncthreads();
        if (t < CB) *cluster.map_shared_rank(&s_left[round & 1][rank], t) = s_sum;
        for (int c = t; c < n_cells; c += kClaimThreads) s_best[c] = kFree;
        if (t == 0) s_count = s_listed = 0;
        __syncthreads();
        if (t == 0) s_sum = 0;  // added to again only after the next cluster barriers
    }
    n_mine = __reduce_add_sync(0xffffffffu, n_mine);
    if (lane == 0 && n_mine) atomicAdd(b.count + e, n_mine);
}

// Lists of an event's condensates: in priority order (alpha_idx, flags, the rank of masked ones) and by grid cell.
template <int NR>
__global__ void __launch_bounds__(1024)
list_condensates_kernel(Buffers b, int dims, int cells_cap, int cells_per_dim, bool by_max_beta, int *__restrict__ n_condensates,
                        int *__restrict__ alpha_out, unsigned char *__restrict__ is_cond, int *__restrict__ assignment)
{
    pdl_begin();
    __shared__ int s_warp[32];
    __shared__ int s_base, s_before;
    const int e = blockIdx.x, t = threadIdx.x, lane = t & 31, warp = t >> 5;
    const CondGrid grid = make_cond_grid(b.layout.grid, b.max_radius, dims, cells_per_dim);
    const int n_cells = grid.n[0] * grid.n[1] * grid.n[2];
    const bool by_grid = *b.use_grid != 0, by_cell = assigns_by_cell(n_cells, dims, by_max_beta);
    const int off = b.row_splits_h[e], n_h = b.row_splits_h[e + 1] - off;
    const int word0 = off / 32 + e;
    int *__restrict__ cell_start = b.cell_count + (size_t)e * (cells_cap + 1);
    auto block_scan = [&](int v) {  // inclusive, over 1024 threads
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int x = __shfl_up_sync(0xffffffffu, v, o);
            if (lane >= o) v += x;
        }
        __syncthreads();
        if (lane == 31) s_warp[warp] = v;
        __syncthreads();
        int w = s_warp[lane];
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int x = __shfl_up_sync(0xffffffffu, w, o);
            if (lane >= o) w += x;
        }
        const int before = __shfl_sync(0xffffffffu, w, warp > 0 ? warp - 1 : 0);
        return v + (warp > 0 ? before : 0);
    };
    // condensates of the events before
    int before = 0;
    for (int q = t; q < e; q += 1024) before += b.count[q];
    before = __reduce_add_sync(0xffffffffu, before);
    if (t == 0) s_before = 0;
    __syncthreads();
    if (lane == 0) atomicAdd(&s_before, before);
    __syncthreads();
    before = s_before;

    auto cell_at = [&](int a, Rec<NR> *x) {  // -1: covers nothing
#pragma unroll
        for (int d = 0; d < NR * 4; d++) x->v[d] = 0.f;
#pragma unroll
        for (int d = 0; d < rec_dims<NR>(); d++)
            if (d < dims) x->v[d] = b.h_ccoords[(size_t)a * dims + d];
        x->v[rec_r2_slot<NR>()] = __fmul_rn(b.h_dist[a], b.h_dist[a]);
        int at[3];
        cell_of<NR>(grid, *x, at);
        return b.h_mask[a] > 0 ? -1 : (at[0] * grid.n[1] + at[1]) * grid.n[2] + at[2];
    };
    int carry = 0;
    const int n_words = (n_h + 31) / 32;
    for (int base = 0; base < n_words; base += 1024) {
        const int w = base + t;
        unsigned bits = 0u;
        if (w < n_words) {
            if (by_grid) {
                bits = b.bitmap[word0 + w];
            } else {
                for (int i = 0; i < 32; i++)
                    if (w * 32 + i < n_h && b.status_h[b.order[off + w * 32 + i]]) bits |= 1u << i;
            }
        }
        const int incl = block_scan(__popc(bits));
        int r = carry + incl - __popc(bits);
        for (; bits; bits &= bits - 1u, r++) b.cl.subset_pos[off + r] = b.order[off + w * 32 + __ffs(bits) - 1];
        __syncthreads();
        if (t == 1023) s_base = carry + incl;
        __syncthreads();
        carry = s_base;
    }
    const int n_cond = carry;
    if (t == 0) {
        if (e == 0) n_condensates[0] = 0;
        n_condensates[e + 1] = before + n_cond;
    }
    for (int r = t; r < n_cond; r += 1024) {
        const int a = b.cl.subset_pos[off + r], id = b.h_orig[a];
        alpha_out[before + r] = id;
        is_cond[id] = 1;
        Rec<NR> x;
        const int cell = cell_at(a, &x);
        if (cell < 0) assignment[id] = r;  // a masked hit is assigned to itself: picked up by assign_hits_kernel
        else if (by_cell) atomicAdd(cell_start + cell, 1);
    }
    __syncthreads();
    carry = 0;
    if (!by_cell) {  // those that cover others, in priority order
        for (int base = 0; base < n_cond; base += 1024) {
            const int r = base + t;
            Rec<NR> x;
            const bool covers = r < n_cond && cell_at(b.cl.subset_pos[off + r], &x) >= 0;
            const int incl = block_scan(covers ? 1 : 0);
            if (covers) {
                store_rec<NR>(b.c_rec + (size_t)(off + carry + incl - 1) * NR, x);
                b.c_rank[off + carry + incl - 1] = r;
            }
            __syncthreads();
            if (t == 1023) s_base = carry + incl;
            __syncthreads();
            carry = s_base;
        }
        if (t == 0) cell_start[0] = carry;
        return;
    }
    for (int base = 0; base <= n_cells; base += 1024) {
        const int c = base + t;
        const int n = c < n_cells ? __ldcg(cell_start + c) : 0;
        const int incl = block_scan(n);
        if (c <= n_cells) cell_start[c] = carry + incl;  // end of the cell: filling counts down to its start
        __syncthreads();
        if (t == 1023) s_base = carry + incl;
        __syncthreads();
        carry = s_base;
    }
    for (int r = t; r < n_cond; r += 1024) {
        Rec<NR> x;
        const int cell = cell_at(b.cl.subset_pos[off + r], &x);
        if (cell < 0) continue;
        const int at = atomicSub(cell_start + cell, 1) - 1;
        store_rec<NR>(b.c_rec + (size_t)(off + at) * NR, x);
        b.c_rank[off + at] = r;
    }
}

// Every hit against the condensates of the cells around it.  Of those that cover it the first in priority order wins
// (by_max_beta), or the reference's distance fold is applied to them in priority order
// (binned_assign_to_condensates_kernel.cc:80-125).  A masked hit is only ever assigned to itself.
// Where the cells around a hit hold most condensates, the hits of a block walk all of them in priority order instead,
// through shared memory (assigns_by_cell): one walk does the fold, and by beta the first that covers the hit ends it.
template <int NR>
__global__ void __launch_bounds__(kThreads)
assign_hits_kernel(Buffers b, const float *__restrict__ ccoords, const int *__restrict__ mask, int dims, int n_events,
                   int cells_cap, int cells_per_dim, bool by_max_beta, int *assignment, int *__restrict__ association,
                   const unsigned char *__restrict__ is_cond, const int *__restrict__ n_condensates,
                   const int *__restrict__ alpha)
{
    pdl_begin();
    HitTile t;
    if (!find_tile(b.layout, n_events, blockIdx.x / (b.layout.tile / kThreads), &t)) return;
    const int i = (blockIdx.x % (b.layout.tile / kThreads)) * kThreads + threadIdx.x;
    const CondGrid grid = make_cond_grid(b.layout.grid, b.max_radius, dims, cells_per_dim);
    if (!assigns_by_cell(grid.n[0] * grid.n[1] * grid.n[2], dims, by_max_beta) && t.event < n_events) {
        __shared__ float4 s_rec[kThreads][NR];
        const int off = b.row_splits_h[t.event], first = n_condensates[t.event];
        const int n_cover = b.cell_count[(size_t)t.event * (cells_cap + 1)];
        const bool live = i < t.n;
        const int v = t.first + i, m = live && mask ? mask[v] : 0;
        int found = live && m > 0 && is_cond[v] ? assignment[v] : -1;  // its own rank
        Rec<NR> x;
#pragma unroll
        for (int d = 0; d < NR * 4; d++) x.v[d] = 0.f;
#pragma unroll
        for (int d = 0; d < rec_dims<NR>(); d++)
            if (live && d < dims) x.v[d] = __fsub_rn(ccoords[(size_t)v * dims + d], b.layout.grid->all_min[d]);
        bool done = !live || m != 0;
        float min_distance = 10e20f;
        for (int c0 = 0; c0 < n_cover; c0 += kThreads) {
            if (__syncthreads_and(done ? 1 : 0)) break;
            if (c0 + (int)threadIdx.x < n_cover)
#pragma unroll
                for (int u = 0; u < NR; u++) s_rec[threadIdx.x][u] = b.c_rec[(size_t)(off + c0 + threadIdx.x) * NR + u];
            __syncthreads();
            const int here = min(kThreads, n_cover - c0);
            for (int c = 0; c < here && !done; c++) {
                const Rec<NR> r = load_rec<NR>(s_rec[c]);
                const float dsq = rec_distsq<NR>(r, x, dims), r2 = r.v[rec_r2_slot<NR>()];
                if (!(dsq <= r2)) continue;
                if (by_max_beta || __fmul_rn(min_distance, r2) >= dsq) {
                    found = c0 + c;
                    min_distance = dsq;
                    done = by_max_beta;
                }
            }
        }
        if (m == 0 && found >= 0) found = b.c_rank[off + found];
        if (live) {
            assignment[v] = found;
            association[v] = found >= 0 ? alpha[first + found] : -1;
        }
        return;
    }
    if (i >= t.n) return;
    const bool real = t.event < n_events;
    const int off = real ? b.row_splits_h[t.event] : 0, first_alpha = real ? n_condensates[t.event] : 0;
    const int n_cond = real ? n_condensates[t.event + 1] - first_alpha : 0;
    const int *__restrict__ cell_start = b.cell_count + (size_t)(real ? t.event : 0) * (cells_cap + 1);
    const int v = t.first + i;
    int found = -1;
    if (n_cond > 0) {
        const int m = mask ? mask[v] : 0;
        if (m != 0) {
            if (m > 0 && is_cond[v]) found = assignment[v];  // its own rank
        } else {
            Rec<NR> x;
#pragma unroll
            for (int d = 0; d < NR * 4; d++) x.v[d] = 0.f;
#pragma unroll
            for (int d = 0; d < rec_dims<NR>(); d++)
                if (d < dims) x.v[d] = __fsub_rn(ccoords[(size_t)v * dims + d], b.layout.grid->all_min[d]);
            int at[3];
            cell_of<NR>(grid, x, at);
            const int lo2 = max(at[2] - 1, 0), hi2 = min(at[2] + 1, grid.n[2] - 1);
            // cells along the last coordinate follow each other: nine ranges of the list, requested together
            int begin[9], end[9];
#pragma unroll
            for (int k = 0; k < 9; k++) {
                const int p = at[0] + k / 3 - 1, q = at[1] + k % 3 - 1;
                begin[k] = end[k] = 0;
                if (p >= 0 && p < grid.n[0] && q >= 0 && q < grid.n[1]) {
                    const int *row = cell_start + (p * grid.n[1] + q) * grid.n[2];
                    begin[k] = __ldg(row + lo2);
                    end[k] = __ldg(row + hi2 + 1);
                }
            }
            float min_distance = 10e20f;
            int last = -1;
            for (;;) {
                // first condensate after `last` that covers the hit, and whether there are more
                int next = 0x7fffffff, n_after = 0;
                float next_dsq = 0.f, next_r2 = 0.f;
#pragma unroll
                for (int w = 0; w < 9; w++)
                    for (int k = begin[w]; k < end[w]; k++) {
                        const Rec<NR> c = load_rec<NR>(b.c_rec + (size_t)(off + k) * NR);
                        const float dsq = rec_distsq<NR>(c, x, dims), r2 = c.v[rec_r2_slot<NR>()];
                        if (!(dsq <= r2)) continue;
                        const int rank = __ldg(b.c_rank + off + k);
                        if (rank <= last) continue;
                        n_after++;
                        if (rank < next) { next = rank; next_dsq = dsq; next_r2 = r2; }
                    }
                if (n_after == 0) break;
                if (by_max_beta) { found = next; break; }
                if (__fmul_rn(min_distance, next_r2) >= next_dsq) { found = next; min_distance = next_dsq; }
                if (n_after == 1) break;
                last = next;
            }
        }
    }
    assignment[v] = found;
    association[v] = found >= 0 ? alpha[first_alpha + found] : -1;
}

// n_bins_sc of the wrapper (assign_condensate_op.py:265-266), sort passes and grid size.
bool make_plan(int n_vert, int dims, int nbin_dims, int n_rs, Plan *p)
{
    p->cb = dims < nbin_dims ? dims : nbin_dims;
    if (p->cb < 1 || p->cb > kMaxBinDims) return false;
    int nb = (int)ceil(pow((double)n_vert / 5., 1. / 3.));
    nb = nb > 25 ? 25 : nb;
    nb = nb < 4 ? 4 : nb;
    p->n_bins_sc = nb;
    long long b = 1;
    for (int d = 0; d < p->cb; d++) b *= nb + 1;
    if (b * (n_rs > 1 ? n_rs - 1 : 1) > (1LL << 30)) return false;
    p->bin_passes = (bits_for(b - 1) + 7) / 8;
    // as many cells as an average event has hits, within limits
    long long cells = n_rs > 1 ? n_vert / (n_rs - 1) : n_vert;
    cells = cells < 4 * kMinCells ? 4 * kMinCells : cells > kMaxCells ? kMaxCells : cells;
    const int gd = dims < 3 ? dims : 3;
    auto power = [gd](long long x) { return gd == 1 ? x : gd == 2 ? x * x : x * x * x; };
    int per = 1;
    while (per < 120 && power(per + 1) <= cells) per++;  // cell numbers along a coordinate are kept in 7 or 8 bits
    p->cells_per_dim = per;
    p->cells = ((int)power(per) + 3) / 4 * 4;
    p->max_settled = (int)power((per + 1) / 2);
    return true;
}

// Tiles as for a quarter of the hits: the sort passes work on the high-beta hits only (4 x 200k hits, a third of them high:
// 476 -> 452 us a call).
int cond_tile(int n_vert) { return order_tile(n_vert / 4); }
size_t cond_tiles_cap(int n_vert, int n_events) { return (size_t)(n_vert > 0 ? n_vert : 0) / cond_tile(n_vert) + n_events + 1; }

template <typename W>
void layout(W &ws, int n_vert, int dims, int num_rows, const Plan &p, Buffers *out, size_t *zeroed)
{
    const size_t n = n_vert > 0 ? n_vert : 0, rows = num_rows > 0 ? num_rows : 0;
    const size_t d = dims > 0 ? dims : 1, nr = rec_size((int)d), e = rows + 2;
    const size_t tiles = cond_tiles_cap(n_vert, (int)rows), passes = p.bin_passes + 4;
    const size_t words = n / 32 + rows + 1;
    Buffers b;
    b.tile_hist = ws.template take<int>((passes + 1) * tiles * 256);
    b.event_hist = ws.template take<int>(passes * (rows + 1) * 256);
    b.count = ws.template take<int>(rows);
    b.cell_count = ws.template take<int>(rows * (p.cells + 1));
    b.max_radius = ws.template take<unsigned>(1);
    if (zeroed) *zeroed = ws.used_bytes();
    b.layout = HitOrder();
    b.layout.tile = cond_tile(n_vert);
    b.layout.grid = ws.template take<GridParams>(1);
    b.layout.partial = ws.template take<float>((size_t)range_partial_blocks(n_vert) * 2 * kMaxBinDims);
    b.layout.event_pos = ws.template take<int>(e);
    b.layout.event_tile = ws.template take<int>(e);
    b.layout.event_chunk = ws.template take<int>(e);
    b.layout.event_super = ws.template take<int>(e);
    b.use_grid = ws.template take<int>(1);
    b.first_two = ws.template take<u64>(2);
    b.tile_count = ws.template take<int>(tiles);
    b.row_splits_h = ws.template take<int>(rows + 1);
    for (int i = 0; i < 2; i++) {
        b.key[i] = ws.template take<u64>(n);
        b.val[i] = ws.template take<int>(n);
    }
    b.order = ws.template take<int>(n);
    b.h_ccoords = ws.template take<float>(n * d);
    b.h_dist = ws.template take<float>(n);
    b.h_mask = ws.template take<int>(n);
    b.h_orig = ws.template take<int>(n);
    b.status_h = ws.template take<int>(n);
    b.p_rec = ws.template take<float4>(n * nr);
    b.p_flag = ws.template take<int>(n);
    b.open = ws.template take<unsigned>(words * 32 + kClaimStep);
    b.bitmap = ws.template take<unsigned>(words);
    b.cl.centre = ws.template take<float>(n * d);
    b.cl.radius_sq = ws.template take<float>(n);
    b.cl.subset_pos = ws.template take<int>(n);
    b.cl.lonely = ws.template take<int>(n);
    b.cl.count = b.count;
    b.alpha_h = ws.template take<int>(n);
    const size_t stage = claim_stage_ints(num_rows);
    b.stage = ws.template take<int>(stage > tiles ? stage : tiles);
    b.c_rec = ws.template take<float4>(n * nr);
    b.c_rank = ws.template take<int>(n);
    if (out) *out = b;
}

struct SizerW {
    Sizer s;
    template <typename T> T *take(size_t n) { s.take<T>(n); return nullptr; }
    size_t used_bytes() const { return s.used; }
};
struct CarverW {
    Carver c;
    template <typename T> T *take(size_t n) { return c.take<T>(n); }
    size_t used_bytes() const { return c.used; }
};

template <bool FIRST, int NR>
int launch_pass(const Buffers &b, int num_rows, int tiles, int pass, int shift, int next_shift, int dims, cudaStream_t stream)
{
    switch (b.layout.tile) {
        case 512: HGC_CUDA_TRY(launch_pdl(order_pass_kernel<2, FIRST, NR>, tiles, kThreads, 0, stream, b, num_rows, tiles, pass, shift, next_shift, dims)); break;
        case 1024: HGC_CUDA_TRY(launch_pdl(order_pass_kernel<4, FIRST, NR>, tiles, kThreads, 0, stream, b, num_rows, tiles, pass, shift, next_shift, dims)); break;
        default: HGC_CUDA_TRY(launch_pdl(order_pass_kernel<8, FIRST, NR>, tiles, kThreads, 0, stream, b, num_rows, tiles, pass, shift, next_shift, dims));
    }
    HGC_LAUNCH_CHECK();
    return HGC_OK;
}

// The last sort pass, the claims, the lists and the assignment, for records of NR float4.
template <int NR>
int run_claims(const Buffers &b, const Plan &p, int dims, int num_rows, int tiles, const float *ccoords, const int *mask,
               bool by_max_beta, int *assignment, int *association, int *alpha_idx, unsigned char *is_cond,
               int *n_condensates, cudaStream_t stream)
{
    const int last = p.bin_passes + 3;
    if (int rc = launch_pass<false, NR>(b, num_rows, tiles, last, 32 + 24, 0, dims, stream)) return rc;
    const size_t smem = 2 * sizeof(int) * (size_t)p.cells + (size_t)p.max_settled * (NR * sizeof(float4) + 2 * sizeof(int));
    // An SM holds one block, so the chip 18 clusters of eight: more events than that wait for each other, and a block of its
    // own for every event is faster whatever their size (without barriers across SMs, and without the registers that merging
    // eight tables takes).  600 events of 100 hits 1.39 -> 0.29 ms, 40 of 5000 0.49 -> 0.26, 64 of 60k 1.71 -> 0.92.
    const bool one_block = num_rows > sm_count() / kClusterBlocks;
    const auto claim = one_block ? claim_grid_kernel<NR, 1> : claim_grid_kernel<NR, kClusterBlocks>;
    // (set on every call: the setting belongs to the current device)
    HGC_CUDA_TRY(cudaFuncSetAttribute(claim, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    HGC_CUDA_TRY(launch_pdl(claim, num_rows * (one_block ? 1 : kClusterBlocks), kClaimThreads, smem, stream, b, dims, p.cells, p.cells_per_dim,
                            p.max_settled));
    HGC_LAUNCH_CHECK();
    if (int rc = launch_claim_windows(dims, b.h_ccoords, b.h_dist, b.h_mask, b.h_orig, b.row_splits_h, b.order, b.status_h,
                                      b.alpha_h, b.stage, b.cl, num_rows, b.use_grid, stream))
        return rc;
    HGC_CUDA_TRY(launch_pdl(list_condensates_kernel<NR>, num_rows, 1024, 0, stream, b, dims, p.cells, p.cells_per_dim, by_max_beta, n_condensates, alpha_idx,
                                                               is_cond, assignment));
    HGC_LAUNCH_CHECK();
    HGC_CUDA_TRY(launch_pdl(assign_hits_kernel<NR>, tiles * (b.layout.tile / kThreads), kThreads, 0, stream, b, ccoords, mask, dims, num_rows, p.cells,
                                                                     p.cells_per_dim, by_max_beta, assignment, association,
                                                                     is_cond, n_condensates, alpha_idx));
    HGC_LAUNCH_CHECK();
    return HGC_OK;
}

}  // namespace
}  // namespace hgc

using namespace hgc;

extern "C" size_t hgc_build_and_assign_condensates_workspace_bytes(int n_vert, int dimensions, int n_rs,
                                                                   int nbin_dims)
{
    Plan p;
    if (dimensions < 1 || dimensions > kMaxCondDims || n_rs < 1 || !make_plan(n_vert, dimensions, nbin_dims, n_rs, &p))
        return 0;
    SizerW w;
    layout(w, n_vert, dimensions, n_rs - 1, p, nullptr, nullptr);
    return w.s.used;
}

extern "C" int hgc_build_and_assign_condensates(
        const float *d_ccoords, const float *d_betas, const float *d_dist, const int *d_no_condensation_mask,
        const int *d_row_splits,
        int *d_assignment, int *d_association, int *d_alpha_idx, unsigned char *d_is_cond,
        int *d_n_condensates, int *h_n_alpha,
        int n_vert, int dimensions, int n_rs, float beta_threshold, float distance_threshold,
        int assign_by_max_beta, int nbin_dims,
        void *workspace, size_t workspace_bytes, hgc_stream_t stream_)
{
    cudaStream_t stream = static_cast<cudaStream_t>(stream_);
    // argument rules of the wrapper (assign_condensate_op.py:245-247)
    if (n_vert < 0 || n_rs < 1 || dimensions < 1 || nbin_dims < 1 || nbin_dims > 6) return HGC_ERR_INVALID_ARGUMENT;
    if (!(beta_threshold >= 0.f && beta_threshold <= 1.f) || !(distance_threshold > 0.f)) return HGC_ERR_INVALID_ARGUMENT;
    if (dimensions > kMaxCondDims) return HGC_ERR_UNSUPPORTED;
    Plan p;
    if (!make_plan(n_vert, dimensions, nbin_dims, n_rs, &p)) return HGC_ERR_UNSUPPORTED;
    const int num_rows = n_rs - 1;
    if (!d_n_condensates || !d_row_splits) return HGC_ERR_INVALID_ARGUMENT;
    if (n_vert > 0 && (!d_ccoords || !d_betas || !d_dist || !d_assignment || !d_association || !d_alpha_idx || !d_is_cond))
        return HGC_ERR_INVALID_ARGUMENT;
    const size_t need = hgc_build_and_assign_condensates_workspace_bytes(n_vert, dimensions, n_rs, nbin_dims);
    if (int rc = check_workspace(workspace, workspace_bytes, need)) return rc;
    if (h_n_alpha) *h_n_alpha = 0;
    if (n_vert == 0 || num_rows == 0) {
        HGC_CUDA_TRY(cudaMemsetAsync(workspace, 0, kAlign, stream));
        HGC_CUDA_TRY(cudaMemsetAsync(d_n_condensates, 0, sizeof(int) * (size_t)n_rs, stream));
        if (n_vert > 0) {
            const size_t bytes = sizeof(int) * (size_t)n_vert;
            HGC_CUDA_TRY(cudaMemsetAsync(d_assignment, 0xff, bytes, stream));
            HGC_CUDA_TRY(cudaMemsetAsync(d_association, 0xff, bytes, stream));
            HGC_CUDA_TRY(cudaMemsetAsync(d_alpha_idx, 0xff, bytes, stream));
            HGC_CUDA_TRY(cudaMemsetAsync(d_is_cond, 0, (size_t)n_vert, stream));
        }
        return HGC_OK;
    }
    CarverW ws{Carver(workspace)};
    unsigned *status = ws.c.status();
    Buffers b;
    size_t zeroed = 0;
    layout(ws, n_vert, dimensions, num_rows, p, &b, &zeroed);
    HGC_CUDA_TRY(cudaMemsetAsync(workspace, 0, zeroed, stream));

    // grid of BinByCoordinates(ccoords[:, :nbin_dims] - min, n_bins=n_bins_sc, pre_normalized=True)
    if (int rc = range_and_layout(d_ccoords, dimensions, p.cb, d_row_splits, n_rs, p.n_bins_sc, 32, n_vert, b.layout, status,
                                  stream))
        return rc;
    const int tiles = (int)cond_tiles_cap(n_vert, num_rows);
    HGC_CUDA_TRY(launch_pdl(count_high_kernel, tiles, kThreads, 0, stream, d_betas, d_no_condensation_mask, beta_threshold, b.layout, num_rows,
                                                      b.tile_count, d_alpha_idx, d_is_cond, b.first_two));
    HGC_LAUNCH_CHECK();
    if (d_no_condensation_mask) {
        HGC_CUDA_TRY(launch_pdl(first_high_kernel<false>, tiles, kThreads, 0, stream, d_ccoords, d_betas, d_no_condensation_mask, beta_threshold,
                                                                 dimensions, p.cb, b.layout, num_rows, b.first_two));
        HGC_LAUNCH_CHECK();
        HGC_CUDA_TRY(launch_pdl(first_high_kernel<true>, tiles, kThreads, 0, stream, d_ccoords, d_betas, d_no_condensation_mask, beta_threshold,
                                                                dimensions, p.cb, b.layout, num_rows, b.first_two));
        HGC_LAUNCH_CHECK();
    }
    const int passes = p.bin_passes + 4;
    HGC_CUDA_TRY(launch_pdl(order_high_kernel, tiles, kThreads, sizeof(int) * 256 * passes, stream, d_ccoords, d_betas, d_dist, d_no_condensation_mask, beta_threshold, distance_threshold, dimensions, p.cb,
            p.bin_passes, num_rows, b, status));
    HGC_LAUNCH_CHECK();
    auto shift_of = [&p](int pass) { return pass < p.bin_passes ? 8 * pass : 32 + 8 * (pass - p.bin_passes); };
    for (int i = 0; i + 1 < passes; i++) {  // the last one belongs to run_claims
        if (int rc = i == 0 ? launch_pass<true, 0>(b, num_rows, tiles, i, shift_of(i), shift_of(i + 1), dimensions, stream)
                            : launch_pass<false, 0>(b, num_rows, tiles, i, shift_of(i), shift_of(i + 1), dimensions, stream))
            return rc;
    }
    int rc = HGC_ERR_UNSUPPORTED;
#define HGC_RUN(NR)                                                                                                  \
    rc = run_claims<NR>(b, p, dimensions, num_rows, tiles, d_ccoords, d_no_condensation_mask, assign_by_max_beta != 0, \
                        d_assignment, d_association, d_alpha_idx, d_is_cond, d_n_condensates, stream)
    if (rec_size(dimensions) == 1) HGC_RUN(1);
    else if (rec_size(dimensions) == 2) HGC_RUN(2);
    else HGC_RUN(3);
#undef HGC_RUN
    if (rc) return rc;
    if (h_n_alpha) {
        HGC_CUDA_TRY(cudaMemcpyAsync(h_n_alpha, d_n_condensates + num_rows, sizeof(int), cudaMemcpyDeviceToHost, stream));
        HGC_CUDA_TRY(cudaStreamSynchronize(stream));
    }
    return HGC_OK;
}
