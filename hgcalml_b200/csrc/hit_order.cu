// Ordering of a ragged batch for the neighbour search: by grid bin (the reference's argsort) and along a Hilbert
// curve, both inside every event.
//
// Events are contiguous in the input, so both sorts run event by event: a block works on a tile of up to 2048
// hits of one event and the event needs no key bits.  Both are stable sorts of 32-bit keys, least significant
// digit first, four passes of 8 bits, and every pass does both orders in one launch (blockIdx.y).  A pass is
// one kernel: the digits of every tile have been counted by the kernel before it (the keys kernel for
// the first pass; a scattering block adds the next digit of every hit to the count of the tile the hit lands in),
// the digits of the whole event by the keys kernel for all passes at once.  A block adds up the counts of
// the tiles before its own, which takes no waiting for other blocks.  Counts are sums of integers, so the
// result does not depend on the order of the atomic additions.
//
// At 200k hits a pass is bound by latency (about 100 blocks): what counts is the number of launches, seven
// here for grid, keys and both orders, against 43 with separate count, scan and scatter kernels per digit and
// order.
#include "common.cuh"
#include "binning_device.cuh"
#include "hit_order.cuh"
#include "hit_order_device.cuh"

namespace hgc {
namespace {

constexpr int kThreads = kOrderThreads;
constexpr int kWarps = kThreads / kWarp;

// Range of the coordinates over the batch; the first block also lays out the events, the last one to
// finish derives the grid.
__global__ void __launch_bounds__(kThreads)
range_and_layout_kernel(const float *__restrict__ coords, int C, int n_dims, int n_all, int n_vert,
                        const int *__restrict__ row_splits, int n_rs, int n_bins, int n_neigh, HitOrder o,
                        unsigned *arrived)
{
    pdl_begin();
    __shared__ bool s_last;
    range_of_block(coords, C, n_all, n_vert, o.partial);
    __syncthreads();
    if (threadIdx.x == 0) {
        __threadfence();
        s_last = atomicAdd(arrived, 1u) == gridDim.x - 1;
    }
    if (blockIdx.x == 0) event_layout(row_splits, n_rs - 1, n_vert, o);
    __syncthreads();
    if (!s_last) return;
    __threadfence();
    grid_from_partials(o.partial, gridDim.x, n_dims, n_all, row_splits, n_rs, n_bins, n_neigh, 0, o.grid);
}

// Bin number inside the event (as modules/compiled/bin_by_coordinates_kernel.cc:64-113: truncating float division, last
// dimension fastest, out-of-range bins forced to 0), then the 16-bit locality code.  frac: scratch, a column per thread.
template <int D, int T>
__device__ __forceinline__ unsigned bin_key(const float (&x)[D], int n_dims, const GridParams *__restrict__ g,
                                            unsigned short (*frac)[T], unsigned *status)
{
    const float bw = g->bin_width;
    unsigned flat = 0u;
    int stride = 1;
#pragma unroll
    for (int c = D - 1; c >= 0; c--) {
        unsigned f;
        if (c < n_dims) {
            const float u = __fdiv_rn(__fsub_rn(x[c], g->shift[c]), bw);
            int ci = __float2int_rz(u);
            f = (unsigned)fminf(fmaxf((u - (float)ci) * 65536.f, 0.f), 65535.f);
            const int nb = g->n_bins[c];
            if (ci < 0 || ci >= nb) {
                ci = 0;
                flag_status(status, HGC_STATUS_BIN_OUT_OF_RANGE);
            }
            flat += (unsigned)(ci * stride);
            stride *= nb;
        } else {
            const float ext = g->all_ext[c];
            const float u = ext > 0.f ? (x[c] - g->all_min[c]) / ext : 0.f;
            f = (unsigned)fminf(fmaxf(u * 65536.f, 0.f), 65535.f);
        }
        frac[c][threadIdx.x] = (unsigned short)f;
    }
    unsigned code = 0u;
#pragma unroll
    for (int k = 0; k < kSubBits; k++) {
        const int c = g->sub_seq[k];  // the same for all threads
        code = (code << 1) | ((unsigned)(frac[c][threadIdx.x] >> g->sub_bit[k]) & 1u);
    }
    return (flat << kSubBits) | code;
}

// Position on a Hilbert curve of B bits per coordinate.
template <int D, int B>
__device__ __forceinline__ unsigned curve_key(const float (&x)[D], const GridParams *__restrict__ g)
{
    const float scale = g->curve_scale * (float)(1u << B);
    unsigned at[D];
#pragma unroll
    for (int c = 0; c < D; c++) at[c] = (unsigned)fminf(fmaxf((x[c] - g->all_min[c]) * scale, 0.f), (float)((1u << B) - 1u));
    return hilbert_code<D, B>(at);
}

// Keys of both orders, digit counts of the tile (first pass) and of the event (all passes).
//   order 0: bin_key, order 1: curve_key
template <int D, int B>
__global__ void __launch_bounds__(kThreads)
order_keys_kernel(const float *__restrict__ coords, int C, int n_dims, HitOrder o, int n_events, int tiles_cap,
                  unsigned *status)
{
    pdl_begin();
    __shared__ int s_hist[2][kOrderPasses][256];
    __shared__ unsigned short s_frac[kMaxBinDims][kThreads];
    HitTile t;
    if (!find_tile(o, n_events, blockIdx.x, &t)) return;
    for (int i = threadIdx.x; i < 2 * kOrderPasses * 256; i += kThreads) (&s_hist[0][0][0])[i] = 0;
    __syncthreads();
    if (t.event == n_events && threadIdx.x == 0) flag_status(status, HGC_STATUS_FLAT_BIN_OVERFLOW);
    const GridParams *__restrict__ g = o.grid;
    for (int i = threadIdx.x; i < t.n; i += kThreads) {
        const int v = t.first + i;
        float x[D];
#pragma unroll
        for (int c = 0; c < D; c++) x[c] = coords[(size_t)v * C + c];
        const unsigned key[2] = {bin_key<D>(x, n_dims, g, s_frac, status), curve_key<D, B>(x, g)};
#pragma unroll
        for (int s = 0; s < 2; s++) {
            o.key[s][0][v] = key[s];
#pragma unroll
            for (int p = 0; p < kOrderPasses; p++) atomicAdd(&s_hist[s][p][(key[s] >> (8 * p)) & 255u], 1);
        }
    }
    __syncthreads();
    const int d = threadIdx.x;  // kThreads == 256 digits
#pragma unroll
    for (int s = 0; s < 2; s++) {
        o.tile_hist[((size_t)(s * kOrderPasses) * tiles_cap + blockIdx.x) * 256 + d] = s_hist[s][0][d];
#pragma unroll
        for (int p = 0; p < kOrderPasses; p++) {
            const int c = s_hist[s][p][d];
            if (c) atomicAdd(&o.event_hist[((size_t)(s * kOrderPasses + p) * (n_events + 2) + t.event) * 256 + d], c);
        }
    }
}

// One pass of both sorts, or of that along the curve alone (first_order 1).  LAST: the permutation (and, for order 0,
// its inverse) is written instead of keys and values.
template <int kRounds, bool FIRST, bool LAST>
__global__ void __launch_bounds__(kThreads)
order_pass_kernel(HitOrder o, int n_events, int tiles_cap, int pass, int first_order, int *__restrict__ bin_perm,
                  int *__restrict__ rank, int *__restrict__ curve_perm)
{
    pdl_begin();
    __shared__ int s_count[kWarps][256];
    __shared__ int s_warp[kWarps];
    const int order = first_order + blockIdx.y, lane = threadIdx.x & 31, warp = threadIdx.x >> 5, d = threadIdx.x;
    HitTile t;
    if (!find_tile(o, n_events, blockIdx.x, &t)) return;
    const unsigned *__restrict__ key_in = o.key[order][pass & 1];
    const int *__restrict__ val_in = o.val[order][pass & 1];
    const int shift = 8 * pass;

    // this tile's items: a warp owns 32 * kRounds consecutive ones, so that equal digits keep their order
    unsigned key[kRounds];
    int val[kRounds];
    const int warp_base = warp * (kRounds * kWarp);
#pragma unroll
    for (int r = 0; r < kRounds; r++) {
        const int i = warp_base + r * kWarp + lane;
        key[r] = 0u;
        val[r] = 0;
        if (i < t.n) {
            key[r] = key_in[t.first + i];
            val[r] = FIRST ? t.first + i : val_in[t.first + i];
        }
    }
    // where the digit starts: smaller digits of the event, and the same digit in the tiles before
    int start = o.event_pos[t.event];
    {
        const int mine = o.event_hist[((size_t)(order * kOrderPasses + pass) * (n_events + 2) + t.event) * 256 + d];
        start += block_scan_inclusive(mine, [](int a, int b) { return a + b; }, 0, s_warp) - mine;
        const int *__restrict__ h = o.tile_hist + (size_t)(order * kOrderPasses + pass) * tiles_cap * 256 + d;
        int sum = 0;
#pragma unroll 16
        for (int q = o.event_tile[t.event]; q < (int)blockIdx.x; q++) sum += h[(size_t)q * 256];
        start += sum;
    }
#pragma unroll
    for (int w = 0; w < kWarps; w++) s_count[w][d] = 0;
    unsigned peers[kRounds];
#pragma unroll
    for (int r = 0; r < kRounds; r++) {
        // places beyond the tile take a digit of their own
        const unsigned dg = warp_base + r * kWarp + lane < t.n ? (key[r] >> shift) & 255u : 256u;
        peers[r] = __match_any_sync(0xffffffffu, dg);
    }
    __syncthreads();
    int place[kRounds];  // inside the run of this digit in this warp
#pragma unroll
    for (int r = 0; r < kRounds; r++) {
        const bool ok = warp_base + r * kWarp + lane < t.n;
        const unsigned dg = (key[r] >> shift) & 255u, before = peers[r] & ((1u << lane) - 1u);
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
    int *__restrict__ next_hist = o.tile_hist + (size_t)(order * kOrderPasses + pass + 1) * tiles_cap * 256;
    const int pos0 = o.event_pos[t.event], tile0 = o.event_tile[t.event];
#pragma unroll
    for (int r = 0; r < kRounds; r++) {
        if (warp_base + r * kWarp + lane < t.n) {
            const int dst = s_count[warp][(key[r] >> shift) & 255u] + place[r];
            if (LAST) {
                if (order == 0) {
                    bin_perm[dst] = val[r];
                    rank[val[r]] = dst;
                } else {
                    curve_perm[dst] = val[r];
                }
            } else {
                o.key[order][(pass + 1) & 1][dst] = key[r];
                o.val[order][(pass + 1) & 1][dst] = val[r];
                const int q = tile0 + (dst - pos0) / (kRounds * kThreads);
                atomicAdd(&next_hist[(size_t)q * 256 + ((key[r] >> (shift + 8)) & 255u)], 1);
            }
        }
    }
}

// Lanes whose digit of BITS bits equals this lane's, among those that are `ok` (the answer of others is of no use).
// match.any takes about 64 cycles of the SM for every warp; a ballot per bit takes 3 to 4 instructions.
template <int BITS>
__device__ __forceinline__ unsigned equal_digits(unsigned digit, bool ok)
{
    unsigned peers = __ballot_sync(0xffffffffu, ok);
#pragma unroll
    for (int b = 0; b < BITS; b++) {
        const bool set = (digit >> b) & 1u;
        const unsigned m = __ballot_sync(0xffffffffu, set);
        peers &= set ? m : ~m;
    }
    return peers;
}

// Small batches: range, grid, event layout and both orders in one launch, a block per event and order, the sort inside its
// shared memory.  Each block finds the range of the whole batch for itself, which is a few loads per thread.
// A chain of six launches is mostly launches and first touches here; search with both orders, us with the chain / with this
// kernel: 700 hits 53 / 34, 2048 55 / 43, 4096 59 / 54, 31 events of 100 50 / 34, 30 of 200 52 / 39, three of 2000 to 3000 66 / 60.  One
// block per event of any size because the host does not know the sizes, so that more than 4096 hits (512 threads, eight hits each)
// take it, with 1024 threads, only where the events are small on average: one event of 8192 hits 82 / 88.  No more events than a
// warp lays out.
constexpr int kSmallHits = 8192, kSmallMean = 2800, kSmallEvents = 31, kSmallItems = 8;
constexpr int kSmallBits = 9, kSmallDigits = 1 << kSmallBits;

template <int D, int B, int kSmallThreads>
__global__ void __launch_bounds__(kSmallThreads)
order_small_kernel(const float *__restrict__ coords, int C, int n_dims, int n_vert, const int *__restrict__ row_splits, int n_rs,
                   int n_bins, int n_neigh, HitOrder o, int *__restrict__ bin_perm, int *__restrict__ rank,
                   int *__restrict__ curve_perm, unsigned *status)
{
    pdl_begin();
    constexpr int kSmallWarps = kSmallThreads / kWarp, kHits = kSmallThreads * kSmallItems;
    __shared__ GridParams s_grid;
    __shared__ float s_mn[kSmallWarps][D], s_mx[kSmallWarps][D];
    __shared__ int s_first, s_end, s_warp[kSmallDigits / 64];
    extern __shared__ unsigned s_small[];
    unsigned (*s_count)[kSmallDigits / 2] = reinterpret_cast<unsigned (*)[kSmallDigits / 2]>(s_small);  // two digits per word: places of a digit in the warps before
    __shared__ int s_start[kSmallDigits];
    unsigned *s_key = s_small + kSmallWarps * (kSmallDigits / 2);
    unsigned short *s_hit = reinterpret_cast<unsigned short *>(s_key + kHits);
    const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
    const int order = blockIdx.x & 1, e = blockIdx.x >> 1, n_events = n_rs - 1;
    float mn[D], mx[D];
#pragma unroll
    for (int c = 0; c < D; c++) { mn[c] = INFINITY; mx[c] = -INFINITY; }
#pragma unroll
    for (int r = 0; r < kSmallItems; r++) {
        const int v = r * kSmallThreads + t;
        if (v < n_vert)
#pragma unroll
            for (int c = 0; c < D; c++) {
                const float x = coords[(size_t)v * C + c];
                mn[c] = fminf(mn[c], x);
                mx[c] = fmaxf(mx[c], x);
            }
    }
#pragma unroll
    for (int c = 0; c < D; c++) {
        const float a = warp_min_f32(mn[c]), b = warp_max_f32(mx[c]);
        if (lane == 0) { s_mn[warp][c] = a; s_mx[warp][c] = b; }
    }
    if (blockIdx.x == 0) event_layout(row_splits, n_events, n_vert, o);  // one warp's work for so few events
    __syncthreads();
    if (warp == 0) {
        float a = 0.f, b = 0.f;
#pragma unroll
        for (int c = 0; c < D; c++) {
            const float lo = warp_min_f32(s_mn[lane % kSmallWarps][c]), hi = warp_max_f32(s_mx[lane % kSmallWarps][c]);
            if (lane == c) { a = lo; b = hi; }
        }
        grid_from_range(a, b, n_dims, D, row_splits, n_rs, n_bins, n_neigh, 0, &s_grid);
    } else if (warp == 1) {  // as event_layout
        int end = lane < n_events ? min(max(row_splits[lane + 1], 0), n_vert) : n_vert;
#pragma unroll
        for (int d = 1; d < 32; d <<= 1) {
            const int v = __shfl_up_sync(0xffffffffu, end, d);
            if (lane >= d) end = max(end, v);
        }
        if (lane == e) s_end = end;
        if (lane == e - 1) s_first = end;
        if (lane == 0 && e == 0) s_first = 0;
    }
    __syncthreads();
    const int pos0 = s_first, n = s_end - pos0;
    if (n <= 0) return;
    if (e == n_events && t == 0) flag_status(status, HGC_STATUS_FLAT_BIN_OVERFLOW);
    // keys: scratch of the locality code lies where the counts will be
    unsigned short (*frac)[kSmallThreads] = reinterpret_cast<unsigned short (*)[kSmallThreads]>(&s_count[0][0]);
    static_assert(sizeof(unsigned) * kSmallWarps * (kSmallDigits / 2) >= sizeof(unsigned short) * kMaxBinDims * kSmallThreads, "");
    for (int i = t; i < n; i += kSmallThreads) {
        float x[D];
#pragma unroll
        for (int c = 0; c < D; c++) x[c] = coords[(size_t)(pos0 + i) * C + c];
        s_key[i] = order == 0 ? bin_key<D>(x, n_dims, &s_grid, frac, status) : curve_key<D, B>(x, &s_grid);
        s_hit[i] = (unsigned short)i;
    }
    const int bits = order == 0 ? kSubBits + 32 - __clz(max(s_grid.bins_per_event - 1, 1)) : D * B;
    const int passes = (bits + kSmallBits - 1) / kSmallBits, width = (bits + passes - 1) / passes, digits = 1 << width;
    // a warp owns 32 * rounds consecutive places, so that equal digits keep their order
    const int rounds = (n + kSmallThreads - 1) / kSmallThreads, first = warp * (32 * rounds) + lane;
    for (int p = 0; p < passes; p++) {
        const int shift = p * width;
        unsigned key[kSmallItems], digit[kSmallItems];
        int hit[kSmallItems], place[kSmallItems];
        __syncthreads();
#pragma unroll
        for (int i = 0; i < kSmallDigits / 64; i++) if (64 * i < digits) s_count[warp][lane + 32 * i] = 0u;
        __syncwarp();
        unsigned short *mine = reinterpret_cast<unsigned short *>(s_count[warp]);
#pragma unroll
        for (int r = 0; r < kSmallItems; r++) {
            if (r >= rounds || first - lane + 32 * r >= n) break;  // the same for the warp
            const int i = first + 32 * r;
            const bool ok = i < n;
            key[r] = ok ? s_key[i] : 0u;
            hit[r] = ok ? s_hit[i] : 0;
            digit[r] = (key[r] >> shift) & (unsigned)(digits - 1);
            const unsigned peers = equal_digits<kSmallBits>(digit[r], ok), before = peers & ((1u << lane) - 1u);
            const int seen = ok ? mine[digit[r]] : 0;
            place[r] = seen + __popc(before);
            __syncwarp();
            if (ok && before == 0u) mine[digit[r]] = (unsigned short)(seen + __popc(peers));
            __syncwarp();
        }
        __syncthreads();
        // first place of every digit: the smaller digits, and per warp this digit in the warps before
        unsigned both = 0u;
        if (t < digits / 2)
#pragma unroll
            for (int w = 0; w < kSmallWarps; w++) {
                const unsigned c = s_count[w][t];
                s_count[w][t] = both;
                both += c;
            }
        const int low = (int)(both & 0xffffu), sum = low + (int)(both >> 16);
        int incl = sum;
#pragma unroll
        for (int d = 1; d < 32; d <<= 1) {
            const int v = __shfl_up_sync(0xffffffffu, incl, d);
            if (lane >= d) incl += v;
        }
        if (lane == 31 && warp < kSmallDigits / 64) s_warp[warp] = incl;
        __syncthreads();
        if (t < digits / 2) {
            int start = incl - sum;
            for (int w = 0; w < warp; w++) start += s_warp[w];
            s_start[2 * t] = start;
            s_start[2 * t + 1] = start + low;
        }
        __syncthreads();
#pragma unroll
        for (int r = 0; r < kSmallItems; r++)
            if (r < rounds && first + 32 * r < n) {
                const int dst = s_start[digit[r]] + mine[digit[r]] + place[r];
                if (p + 1 < passes) {
                    s_key[dst] = key[r];
                    s_hit[dst] = (unsigned short)hit[r];
                } else if (order == 0) {
                    bin_perm[pos0 + dst] = pos0 + hit[r];
                    rank[pos0 + hit[r]] = pos0 + dst;
                } else {
                    curve_perm[pos0 + dst] = pos0 + hit[r];
                }
            }
    }
}

template <int D, int B, int T>
int launch_small(const float *coords, int n_coords, int n_bin_dims, int n_vert, const int *row_splits, int n_rs, int n_bins, int n_neigh,
                 const HitOrder &o, int *bin_perm, int *rank, int *curve_perm, unsigned *status, cudaStream_t stream)
{
    const auto kernel = order_small_kernel<D, B, T>;
    const size_t smem = sizeof(unsigned) * (T / kWarp) * (kSmallDigits / 2) + (sizeof(unsigned) + sizeof(unsigned short)) * T * kSmallItems;
    // (set on every call: the setting belongs to the current device)
    if (T > 512) HGC_CUDA_TRY(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    HGC_CUDA_TRY(launch_pdl(kernel, 2 * n_rs, T, smem, stream, coords, n_coords, n_bin_dims, n_vert, row_splits, n_rs, n_bins, n_neigh, o,
                            bin_perm, rank, curve_perm, status));
    HGC_LAUNCH_CHECK();
    return HGC_OK;
}

}  // namespace

int range_and_layout(const float *coords, int n_coords, int n_bin_dims, const int *row_splits, int n_rs, int n_bins,
                     int n_neigh, int n_vert, const HitOrder &o, unsigned *status, cudaStream_t stream)
{
    HGC_CUDA_TRY(launch_overlapped(n_vert, range_and_layout_kernel, range_partial_blocks(n_vert), kThreads, 0, stream, coords, n_coords, n_bin_dims, n_coords < kMaxBinDims ? n_coords : kMaxBinDims, n_vert, row_splits, n_rs, n_bins,
            n_neigh, o, status + 8));
    HGC_LAUNCH_CHECK();
    return HGC_OK;
}

int order_hits(const float *coords, int n_coords, int n_bin_dims, const int *row_splits, int n_rs, int n_bins, int n_neigh,
               int n_vert, int bin_bits, const HitOrder &o, int *bin_perm, int *rank, int *curve_perm,
               unsigned *status, cudaStream_t stream)
{
    if (n_vert <= 0) return HGC_OK;
    if (bin_bits + kSubBits > 32) return HGC_ERR_UNSUPPORTED;
    const int n_events = n_rs - 1;
    const int n_all = n_coords < kMaxBinDims ? n_coords : kMaxBinDims;
    if (n_vert <= (n_vert / n_events <= kSmallMean ? kSmallHits : kSmallHits / 2) && n_events <= kSmallEvents && bin_bits > 0) {
#define HGC_SMALL(D, B)                                                                                            \
    case D: if (int rc = n_vert <= 512 * kSmallItems ? launch_small<D, B, 512>(coords, n_coords, n_bin_dims, n_vert, row_splits, n_rs, n_bins, n_neigh, o, bin_perm, rank, curve_perm, status, stream) \
                                                     : launch_small<D, B, 1024>(coords, n_coords, n_bin_dims, n_vert, row_splits, n_rs, n_bins, n_neigh, o, bin_perm, rank, curve_perm, status, stream)) return rc; break
        switch (n_all) {
            HGC_SMALL(2, 13);
            HGC_SMALL(3, 9);
            HGC_SMALL(4, 6);
            HGC_SMALL(5, 5);
            HGC_SMALL(6, 4);
            HGC_SMALL(7, 3);
            HGC_SMALL(8, 3);
            default: return HGC_ERR_UNSUPPORTED;
        }
#undef HGC_SMALL
        return HGC_OK;
    }
    if (int rc = range_and_layout(coords, n_coords, n_bin_dims, row_splits, n_rs, n_bins, n_neigh, n_vert, o, status, stream))
        return rc;
    const int tiles = (int)order_tiles_cap(n_vert, n_events);
#define HGC_KEYS(D, B)                                                                                            \
    case D: HGC_CUDA_TRY(launch_overlapped(n_vert, order_keys_kernel<D, B>, tiles, kThreads, 0, stream, coords, n_coords, n_bin_dims, o, n_events, tiles, status)); break
    switch (n_all) {
        HGC_KEYS(2, 16);
        HGC_KEYS(3, 10);
        HGC_KEYS(4, 8);
        HGC_KEYS(5, 6);
        HGC_KEYS(6, 5);
        HGC_KEYS(7, 4);
        HGC_KEYS(8, 4);
        default: return HGC_ERR_UNSUPPORTED;
    }
#undef HGC_KEYS
    HGC_LAUNCH_CHECK();
    const int first_order = bin_bits > 0 ? 0 : 1;
    const dim3 grid(tiles, 2 - first_order);
    for (int p = 0; p < kOrderPasses; p++) {
#define HGC_PASS(R)                                                                                                  \
    case R * kThreads:                                                                                               \
        if (p == 0)                                                                                                  \
            HGC_CUDA_TRY(launch_overlapped(n_vert, order_pass_kernel<R, true, false>, grid, kThreads, 0, stream, o, n_events, tiles, p, first_order, bin_perm, rank, curve_perm)); \
        else if (p + 1 < kOrderPasses)                                                                               \
            HGC_CUDA_TRY(launch_overlapped(n_vert, order_pass_kernel<R, false, false>, grid, kThreads, 0, stream, o, n_events, tiles, p, first_order, bin_perm, rank, curve_perm)); \
        else                                                                                                         \
            HGC_CUDA_TRY(launch_overlapped(n_vert, order_pass_kernel<R, false, true>, grid, kThreads, 0, stream, o, n_events, tiles, p, first_order, bin_perm, rank, curve_perm)); \
        break
        switch (o.tile) {
            HGC_PASS(2);
            HGC_PASS(4);
            HGC_PASS(8);
        }
#undef HGC_PASS
        HGC_LAUNCH_CHECK();
    }
    return HGC_OK;
}

}  // namespace hgc
