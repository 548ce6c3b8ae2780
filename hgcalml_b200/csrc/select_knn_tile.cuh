// Exact nearest-neighbour search of the wrapper-level entry, one block per tile of neighbouring queries (device
// code; instantiated per coordinate width in select_knn_tile_nv*.cu).
//
// Layout (hit_order.cu, pack_tiles_kernel).  The hits of an event follow a Hilbert curve through all their
// coordinates; parts of 128 or 256 are cut by medians into chunks of 32 hits, 1024 make a super-chunk.  A chunk never
// straddles events (the last one of an event is padded with NaN points, which no comparison accepts).  Chunks and
// super-chunks have bounding boxes over all coordinates.
//
// A block of four warps answers the queries of one tile (up to 32 hits of one chunk):
//  1. Bounds.  Four representatives of the tile, one per warp, look at the chunks next to their own on the
//     curve; the K-th smallest distance among those hits bounds their K-th nearest distance from above, and by
//     the triangle inequality |q - rep| + bound(rep) bounds that of every query q.
//  2. List.  Super-chunk boxes, then chunk boxes, are tested against the box of the tile: only chunks within
//     the largest of the tile's bounds can matter to any of its queries.  The list is put in order of the
//     distance from the tile's centre (32 classes), so that a query reads only as far as its own bound reaches.
//  3. Queries.  Each warp takes the tile's queries one after another.  A query starts from the K-th distance
//     of the nearest query already answered, half as many hits again: the chunks within it are noted, 32 box
//     tests at a time, then their hits are compared 32 at a time, four chunks in flight, and hits inside
//     are parked in shared memory.  With K - 1 of them the answer is among them; otherwise (a quarter of the
//     queries of the shower events) the radius grows.  A full buffer is pruned by counting: a bound that
//     keeps at least K - 1 of the distances and few more is found by interpolation, without sorting.  The row is
//     sorted once, at the end, as 32-bit words.
//
// What it replaced on this path: one warp per query over the bins around the query's, with a list that was
// kept sorted all along (select_knn_kernel.cuh, still the kernel of the op-level entry, whose callers bring their own
// bins).  64 events of 200k hits, K = 64, 4 coordinates: 68.0 -> 32.5 ms; 200k hits with coordinates N(0,1)-like in four
// dimensions: 1.77 -> 0.88 ms.  5.7k -> 2.0k warp instructions per query: 18 chunk visits instead of 36 candidate steps,
// one word sort instead of seven merges of 64-bit keys, and what finds the chunks is shared by a tile.
// The kernel is bound by the latency of gathers that miss L1 (64 % hit) and by issue (74 % of the slots) together.
// It is therefore sensitive to everything that takes L1 away: spilled registers (a 144-byte frame: +35 %), shared
// memory, more resident blocks (10 instead of 9 per SM: +7 %).  What depends on the tile only is kept in
// shared memory rather than in registers for that reason.
//
// Exactness.  Distances are summed with separately rounded operations in coordinate order, so they
// are bit-identical to the CPU op (modules/compiled/binned_select_knn_kernel.cc:19-29).  Box distances use
// the same operations on the gaps between boxes; rounding is monotone, so they never exceed the computed
// distance of any two points inside.  Bounds from the triangle inequality are widened by 1e-5 (and
// 1e-37 for squares that underflow), far above the rounding of the operations behind them.  Hits are
// compared by (distance, position in the bin-sorted order), so ties fall to the lower position.
#pragma once
#include "common.cuh"
#include "knn_device.cuh"
#include "select_knn_tile_api.cuh"

namespace hgc {

constexpr int kTileWarps = 4;
constexpr int kTileThreads = kTileWarps * kWarp;
// Chunks in a tile's list; tiles that need more walk the boxes per query.  What the list takes of shared memory, L1 lacks:
// 200k hits N(0,1)-like in four dimensions, four searches: 512 4.34, 1024 3.61, 1280 3.53, 2048 3.72 ms.
constexpr int kTileListCap = 1280;
constexpr int kTileBuckets = 32;      // classes of distance from the tile's centre
constexpr int kTileClassBits = 5;

// L: registers of 32 sorted neighbours, K - 1 <= 32 * L
template <int L> struct TileShape {
    static constexpr int kPruneAt = L == 1 ? 64 : L == 2 ? 96 : 32 * L + 16 * L;  // parked hits that trigger a prune
    static constexpr int kCap = kPruneAt + 64;                                    // two chunks may be appended on top
    static constexpr int kWindow = L <= 2 ? 8 : 4 * L;                             // slack a prune may leave above K - 1
    static constexpr int kRep = 2 * L + 3;                                        // chunks a representative looks at
};
constexpr int kTileNear = 68;   // chunks within reach that a warp collects before it looks at their hits

__device__ __forceinline__ unsigned redux_max_u32(unsigned v) { return __reduce_max_sync(0xffffffffu, v); }
__device__ __forceinline__ int redux_add_i32(int v) { return __reduce_add_sync(0xffffffffu, v); }
// Approximate square root (relative error below 2^-22); only for bounds that are widened by more than that.
__device__ __forceinline__ float sqrt_fast(float v)
{
    float r;
    asm("sqrt.approx.f32 %0, %1;" : "=f"(r) : "f"(v));
    return r;
}

// A bound T with count(v <= T) >= target and, unless values tie or the iterations run out, at most
// target + window.  On entry count(v <= hi) == chi >= target; on return chi belongs to the result.
// Interpolates between counts; the first guess takes hits as uniform in space (count ~ distsq^(1/expo)).
template <int N>
__device__ __forceinline__ float count_bound(const float (&v)[N], int target, int window, float hi, int &chi,
                                             float expo)
{
    float lo = 0.f;
    int clo = 0;
    const float aim = (float)target + 0.5f * (float)window;
    float frac = exp2f(expo * __log2f(__fdividef(aim, (float)chi)));
    for (int it = 0; it < 14 && chi > target + window; it++) {
        const float t = fmaf(hi - lo, frac, lo);
        int c = 0;
#pragma unroll
        for (int i = 0; i < N; i++) c += v[i] <= t ? 1 : 0;
        c = redux_add_i32(c);
        if (c < target) { lo = t; clo = c; } else { hi = t; chi = c; }
        frac = it < 8 ? fminf(fmaxf(__fdividef(aim - (float)clo, (float)(chi - clo)), 0.03f), 0.97f) : 0.5f;
    }
    return hi;
}

struct Pruned { knn_key thr; int cnt; };

// Sorts the parked hits and keeps exactly the `keep` smallest, in order; returns the largest of them.  For rows
// whose distances tie so that counting cannot part them; rare.  Out of line for the long lists, whose networks are most of the
// kernel's code otherwise (200k hits, K = 100: 1020 -> 975 us); a call costs the short ones more in spills than it saves (K = 64
// +2 %).
template <int L>
__device__ __forceinline__ knn_key keep_smallest_inline(knn_key *buf, int cnt, int keep, int lane)
{
    knn_key list[L];
#pragma unroll
    for (int r = 0; r < L; r++) list[r] = HGC_KNN_INF_KEY;
    for (int i = lane; i - lane < cnt; i += 32)
        merge_into_list<L>(list, warp_sort(i < cnt ? buf[i] : HGC_KNN_INF_KEY, lane), lane);
    __syncwarp();
#pragma unroll
    for (int r = 0; r < L; r++)
        if (r * 32 + lane < keep) buf[r * 32 + lane] = list[r];
    __syncwarp();
    return shfl_key(list_reg<L>(list, (keep - 1) / 32), (keep - 1) & 31);
}

template <int L>
__device__ __noinline__ knn_key keep_smallest_call(knn_key *buf, int cnt, int keep, int lane)
{
    return keep_smallest_inline<L>(buf, cnt, keep, lane);
}
template <int L>
__device__ __forceinline__ knn_key keep_smallest(knn_key *buf, int cnt, int keep, int lane)
{
    if constexpr (L > 2) return keep_smallest_call<L>(buf, cnt, keep, lane);
    else return keep_smallest_inline<L>(buf, cnt, keep, lane);
}

// Reduces the parked hits to at most `limit` (>= want) of the smallest and tightens the bound.
template <int L>
__device__ __forceinline__ Pruned prune_parked(knn_key *buf, int cnt, int want, int window, int limit, knn_key thr,
                                            float expo, int lane)
{
    constexpr int N = TileShape<L>::kCap / 32;
    knn_key k[N];
    float v[N];
    __syncwarp();
    float hi = 0.f;
#pragma unroll
    for (int i = 0; i < N; i++) {
        const int e = lane + 32 * i;
        k[i] = e < cnt ? buf[e] : HGC_KNN_INF_KEY;
        v[i] = e < cnt ? key_distsq(k[i]) : __int_as_float(0x7fffffff);
        hi = fmaxf(hi, v[i]);
    }
    hi = __uint_as_float(redux_max_u32(__float_as_uint(hi)));
    int chi = cnt;
    const float t = count_bound<N>(v, want, window, hi, chi, expo);
    __syncwarp();
    Pruned out;
    out.thr = thr;
    if (chi <= limit) {
        int n = 0;
#pragma unroll
        for (int i = 0; i < N; i++) {
            const bool keep = v[i] <= t;
            const unsigned m = __ballot_sync(0xffffffffu, keep);
            if (keep) buf[n + __popc(m & ((1u << lane) - 1u))] = k[i];
            n += __popc(m);
        }
        out.cnt = n;
        const knn_key nt = make_key(t, 0x7fffffff);
        if (nt < thr) out.thr = nt;
        __syncwarp();
    } else {
        out.thr = keep_smallest<L>(buf, cnt, want, lane);
        out.cnt = want;
    }
    return out;
}

// The 32 * L smallest of the parked hits in ascending order, striped; places beyond cnt hold INF.  `bound` is an
// upper bound of the parked distances.
//
// For K <= 64 words of 32 bits are sorted instead of keys: the distance as a fraction of the bound (24 bits or
// more) and the slot.  The first 32 * L words are sorted, every further block of 32 is sorted and merged
// into the front.  Only where two words that end up next to each other agree in their fraction (one row in a
// thousand) are the full keys sorted.  K - 1 < 32 * L, so that the word after the last one needed is seen too.
template <int L>
__device__ __forceinline__ void load_sorted(knn_key *buf, int cnt, float bound, knn_key (&list)[L], int lane)
{
    static_assert(L <= 2, "longer lists are pruned to 32 * L keys and sorted in full");
    constexpr int kSlotBits = TileShape<L>::kCap <= 128 ? 7 : 8;
    constexpr unsigned kSlots = 1u << kSlotBits;
    static_assert(TileShape<L>::kCap <= 256, "slot numbers of eight bits");
    const float scale = bound > 1e-30f && bound < 1e30f ? __fdividef((float)((1u << (32 - kSlotBits)) - 2u), bound) : 0.f;
    auto word = [&](int e) -> unsigned {
        if (e >= cnt) return 0xffffffffu;
        const unsigned f = min((unsigned)(key_distsq(buf[e]) * scale), (1u << (32 - kSlotBits)) - 2u);
        return (f << kSlotBits) | (unsigned)e;
    };
    unsigned w[L];
#pragma unroll
    for (int r = 0; r < L; r++) w[r] = warp_sort_u32(word(r * 32 + lane), lane);
    if (L == 2) {
        const unsigned o = __shfl_xor_sync(0xffffffffu, w[L - 1], 31);
        const unsigned lo = min(w[0], o), hi = max(w[0], o);
        w[0] = warp_bitonic_merge_u32(lo, lane);
        w[L - 1] = warp_bitonic_merge_u32(hi, lane);
    }
    for (int base = 32 * L; base < cnt; base += 32) {
        const unsigned o = __shfl_xor_sync(0xffffffffu, warp_sort_u32(word(base + lane), lane), 31);
        if (L == 2) {
            // the 64 smallest of 64 + 32: the block only competes with the upper register
            const unsigned up = min(w[L - 1], o);
            const unsigned lo = min(w[0], up), hi = max(w[0], up);
            w[0] = warp_bitonic_merge_u32(lo, lane);
            w[L - 1] = warp_bitonic_merge_u32(hi, lane);
        } else {
            w[0] = warp_bitonic_merge_u32(min(w[0], o), lane);
        }
    }
    bool tie = false;
#pragma unroll
    for (int r = 0; r < L; r++) {
        unsigned next = __shfl_down_sync(0xffffffffu, w[r], 1);
        if (r + 1 < L) {
            const unsigned over = __shfl_sync(0xffffffffu, w[r + 1 < L ? r + 1 : r], 0);
            if (lane == 31) next = over;
        } else if (lane == 31) {
            next = ~w[r];
        }
        tie = tie || (w[r] != 0xffffffffu && (w[r] ^ next) < kSlots);
        list[r] = w[r] != 0xffffffffu ? buf[w[r] & (kSlots - 1u)] : HGC_KNN_INF_KEY;
    }
    if (__any_sync(0xffffffffu, tie)) {
        const int keep = min(cnt, 32 * L);
        keep_smallest<L>(buf, cnt, keep, lane);
#pragma unroll
        for (int r = 0; r < L; r++) list[r] = r * 32 + lane < keep ? buf[r * 32 + lane] : HGC_KNN_INF_KEY;
    }
}

template <int NV4, int L>
struct TileQuery {
    using S = TileShape<L>;
    Point<NV4> q;
    knn_key thr;      // (bound, position): hits up to and including it are kept
    knn_key *buf;     // this warp's parked hits
    int *near_;       // this warp's chunks within reach (first hit of each)
    int cnt, n_near, lane;
    const TileKnnArgs *a;

    // Parks the hits (one per lane, at position j of the packed points) that are within the bound.
    __device__ __forceinline__ void append(float ds, int rank, bool ok)
    {
        const knn_key key = make_key(ds, rank);
        const bool pass = ok && key <= thr;
        const unsigned m = __ballot_sync(0xffffffffu, pass);  // (leaving early where it is empty: 400k hits +1 %)
        if (pass) buf[cnt + __popc(m & ((1u << lane) - 1u))] = key;
        cnt += __popc(m);
    }

    // Notes the chunk of every lane whose box is within the bound.
    __device__ __forceinline__ void note(bool ok, int cid)
    {
        const unsigned m = __ballot_sync(0xffffffffu, ok);
        if (ok) near_[n_near + __popc(m & ((1u << lane) - 1u))] = cid * 32;
        n_near += __popc(m);
    }

    // Looks at the hits of the noted chunks; the loads of four chunks are in flight together (two for the last one or
    // two: filling them up to four cost 5 %).
    __device__ __forceinline__ void look()
    {
        const float4 *__restrict__ pts = a->pts;
        const int *__restrict__ ranks = a->ranks;
        constexpr int U = NV4 == 1 ? 4 : 2;
        if (lane < U) near_[n_near + lane] = a->nobody;  // a chunk without hits fills up the last step
        __syncwarp();
        for (int i = 0; i < n_near; i += U) {
            Point<NV4> p[U];
            int j[U];
            if (U == 4) {
                const int4 c = *reinterpret_cast<const int4 *>(near_ + i);
                j[0] = c.x + lane; j[1] = c.y + lane; j[U - 2] = c.z + lane; j[U - 1] = c.w + lane;
            } else {
                const int2 c = *reinterpret_cast<const int2 *>(near_ + i);
                j[0] = c.x + lane; j[1] = c.y + lane;
            }
#pragma unroll
            for (int u = 0; u < U; u++) {
                if (u >= 2 && i + 2 >= n_near) break;  // uniform
                p[u] = load_point<NV4>(pts, (size_t)j[u]);
                j[u] = __ldg(ranks + j[u]);
            }
#pragma unroll
            for (int u = 0; u < U; u += 2) {
                if (u >= 2 && i + 2 >= n_near) break;
                append(distsq<NV4>(q, p[u]), j[u], true);
                append(distsq<NV4>(q, p[u + 1]), j[u + 1], true);
                if (cnt > S::kPruneAt) {
                    const Pruned pr = prune_parked<L>(buf, cnt, a->K - 1, S::kWindow, S::kPruneAt, thr, a->expo, lane);
                    thr = pr.thr;
                    cnt = pr.cnt;
                }
            }
        }
        n_near = 0;
        __syncwarp();
    }
};

// Squared distance between the boxes [qlo, qhi] and box (lo, hi), with the operation sequence of distsq.
template <int NV4>
__device__ __forceinline__ float box_gap_distsq(const Point<NV4> &qlo, const Point<NV4> &qhi,
                                                const float4 *__restrict__ box)
{
    float s = 0.f;
#pragma unroll
    for (int u = 0; u < NV4; u++) {
        const float4 l = __ldg(box + 2 * u), h = __ldg(box + 2 * u + 1);
        const float2 a01 = sub2(l.x, l.y, qhi.v[u].x, qhi.v[u].y), a23 = sub2(l.z, l.w, qhi.v[u].z, qhi.v[u].w);
        const float2 b01 = sub2(qlo.v[u].x, qlo.v[u].y, h.x, h.y), b23 = sub2(qlo.v[u].z, qlo.v[u].w, h.z, h.w);
        const float2 q01 = sqr2(make_float2(fmaxf(fmaxf(a01.x, b01.x), 0.f), fmaxf(fmaxf(a01.y, b01.y), 0.f)));
        const float2 q23 = sqr2(make_float2(fmaxf(fmaxf(a23.x, b23.x), 0.f), fmaxf(fmaxf(a23.y, b23.y), 0.f)));
        s = u == 0 ? q01.x : __fadd_rn(s, q01.x);
        s = __fadd_rn(s, q01.y);
        s = __fadd_rn(s, q23.x);
        s = __fadd_rn(s, q23.y);
    }
    return s;
}

// (8 blocks per SM for 5 to 8 coordinates: 114k hits, K = 41 411 us, 6 blocks 427 us)
template <int NV4, int L>
__global__ void __launch_bounds__(kTileThreads, L <= 2 && NV4 == 1 ? 9 : (L <= 2 && NV4 == 2 ? 8 : L <= 4 ? 6 : 3))
select_knn_tile_kernel(const TileKnnArgs a)
{
    pdl_begin();
    using S = TileShape<L>;
    __shared__ knn_key s_buf[kTileWarps][S::kCap];
    __shared__ unsigned s_list[kTileListCap];  // chunk id << 5 | distance class
    __shared__ float4 s_rep[kTileWarps][NV4];
    __shared__ float s_bound[kTileWarps];
    __shared__ __align__(16) int s_near[kTileWarps][kTileNear];
    __shared__ int s_hist[kTileBuckets], s_end[kTileBuckets];  // chunks of a class; end of the class in the list
    __shared__ float s_sure[32], s_first[32], s_scale;  // bounds of the queries; classes per squared distance
    __shared__ float4 s_mid[NV4];                      // centre of the tile's box
    __shared__ int s_id[32];
    __shared__ float4 s_mine[NV4][32];
    __shared__ float s_radius[32];  // K-th distance of the tile's queries that are answered, else INF
    __shared__ int s_count, s_next;

    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int T = a.tile;
    const int chunk = blockIdx.x / (32 / T), first = (blockIdx.x % (32 / T)) * T;  // 32 is a multiple of T
    if (chunk >= a.n_chunks[0]) return;
    const int4 ev = __ldg(a.chunk_info + chunk);  // chunks [x, y), super-chunks [z, w) of the event
    const int my_id = a.ids[chunk * 32 + lane];
    const bool in_tile = my_id >= 0 && lane >= first && lane < first + T;
    const int n_q = __popc(__ballot_sync(0xffffffffu, in_tile));
    if (n_q == 0) return;

    if (threadIdx.x == 0) { s_count = 0; s_next = 0; }
    if (threadIdx.x < kTileBuckets) s_hist[threadIdx.x] = 0;
    if (threadIdx.x < 32) s_radius[threadIdx.x] = INFINITY;

    // this lane's query point (the packed points hold NaN for hits that may not be neighbours)
    Point<NV4> mine;
    if (a.coords != nullptr && my_id >= 0) {
        const float *src = a.coords + (size_t)my_id * a.n_coords;
#pragma unroll
        for (int u = 0; u < NV4; u++) {
            mine.v[u].x = u * 4 + 0 < a.n_coords ? src[u * 4 + 0] : 0.f;
            mine.v[u].y = u * 4 + 1 < a.n_coords ? src[u * 4 + 1] : 0.f;
            mine.v[u].z = u * 4 + 2 < a.n_coords ? src[u * 4 + 2] : 0.f;
            mine.v[u].w = u * 4 + 3 < a.n_coords ? src[u * 4 + 3] : 0.f;
        }
    } else {
        mine = load_point<NV4>(a.pts, (size_t)chunk * 32 + lane);
    }
    const int K = a.K, want = K - 1;
    const bool search = want > 0 && ev.y > ev.x;

    float my_guess = INFINITY;  // squared: the nearest representative's own bound
    if (search) {
        // ---- 1. bounds ----
        {
            const int rep = first + (warp * n_q) / kTileWarps;
            Point<NV4> rq;
#pragma unroll
            for (int u = 0; u < NV4; u++) {
                rq.v[u].x = __shfl_sync(0xffffffffu, mine.v[u].x, rep);
                rq.v[u].y = __shfl_sync(0xffffffffu, mine.v[u].y, rep);
                rq.v[u].z = __shfl_sync(0xffffffffu, mine.v[u].z, rep);
                rq.v[u].w = __shfl_sync(0xffffffffu, mine.v[u].w, rep);
            }
            int c0 = chunk - S::kRep / 2;
            if (c0 + S::kRep > ev.y) c0 = ev.y - S::kRep;
            if (c0 < ev.x) c0 = ev.x;
            float v[S::kRep], hi = 0.f;
            int have = 0;
#pragma unroll
            for (int i = 0; i < S::kRep; i++) {
                v[i] = __int_as_float(0x7fffffff);
                if (c0 + i < ev.y) v[i] = distsq<NV4>(rq, load_point<NV4>(a.pts, (size_t)(c0 + i) * 32 + lane));
                if (!(v[i] < INFINITY)) v[i] = __int_as_float(0x7fffffff);  // pads, and overflowed distances
                have += v[i] < INFINITY ? 1 : 0;
                hi = fmaxf(hi, v[i]);
            }
            have = redux_add_i32(have);
            hi = __uint_as_float(redux_max_u32(__float_as_uint(hi)));
            float bound = INFINITY;
            // the representative itself may be among them: K of them hold K - 1 others
            if (have >= K) bound = count_bound<S::kRep>(v, K, S::kWindow, hi, have, a.expo);
            if (lane == 0) {
                s_bound[warp] = sqrt_fast(bound);
#pragma unroll
                for (int u = 0; u < NV4; u++) s_rep[warp][u] = rq.v[u];
            }
        }
        __syncthreads();
        float b = INFINITY, near_rep = INFINITY;
#pragma unroll
        for (int w = 0; w < kTileWarps; w++) {
            Point<NV4> rq;
#pragma unroll
            for (int u = 0; u < NV4; u++) rq.v[u] = s_rep[w][u];
            const float away = sqrt_fast(distsq<NV4>(mine, rq)), bound = s_bound[w];
            b = fminf(b, bound + away);
            if (away < near_rep) { near_rep = away; my_guess = bound * bound; }
        }
        const float my_bound = b * b * 1.00001f + 1e-37f;  // squared: holds for certain
        if (warp == 0) { s_sure[lane] = my_bound; s_first[lane] = my_guess; s_id[lane] = my_id; }
        if (warp == 1)
#pragma unroll
            for (int u = 0; u < NV4; u++) s_mine[u][lane] = mine.v[u];
        const float reach = warp_max_f32(in_tile ? my_bound : 0.f);

        // ---- 2. list ----
        Point<NV4> lo, hi, mid;
#pragma unroll
        for (int u = 0; u < NV4; u++) {
            lo.v[u].x = warp_min_f32(in_tile ? mine.v[u].x : INFINITY); hi.v[u].x = warp_max_f32(in_tile ? mine.v[u].x : -INFINITY);
            lo.v[u].y = warp_min_f32(in_tile ? mine.v[u].y : INFINITY); hi.v[u].y = warp_max_f32(in_tile ? mine.v[u].y : -INFINITY);
            lo.v[u].z = warp_min_f32(in_tile ? mine.v[u].z : INFINITY); hi.v[u].z = warp_max_f32(in_tile ? mine.v[u].z : -INFINITY);
            lo.v[u].w = warp_min_f32(in_tile ? mine.v[u].w : INFINITY); hi.v[u].w = warp_max_f32(in_tile ? mine.v[u].w : -INFINITY);
            mid.v[u] = make_float4(0.5f * (lo.v[u].x + hi.v[u].x), 0.5f * (lo.v[u].y + hi.v[u].y),
                                   0.5f * (lo.v[u].z + hi.v[u].z), 0.5f * (lo.v[u].w + hi.v[u].w));
        }
        const float class_scale = reach < INFINITY ? (float)kTileBuckets / reach : 0.f;
        // neighbouring super-chunks go to different warps
        for (int s0 = ev.z; s0 < ev.w; s0 += kTileThreads) {
            const int s = s0 + lane * kTileWarps + warp;
            bool near_ = false;
            if (s < ev.w) near_ = box_gap_distsq<NV4>(lo, hi, a.super_box + (size_t)s * 2 * NV4) <= reach;
            unsigned m = __ballot_sync(0xffffffffu, near_);
            while (m) {
                const int src = __ffs(m) - 1;
                m &= m - 1u;
                const int c = ev.x + (s0 + src * kTileWarps + warp - ev.z) * 32 + lane;
                bool take = false;
                unsigned cls = 0;
                if (c < ev.y && c != chunk) {
                    const float4 *box = a.chunk_box + (size_t)c * 2 * NV4;
                    take = box_gap_distsq<NV4>(lo, hi, box) <= reach;
                    if (take) cls = (unsigned)fminf(box_gap_distsq<NV4>(mid, mid, box) * class_scale, (float)(kTileBuckets - 1));
                }
                const unsigned tm = __ballot_sync(0xffffffffu, take);
                if (tm) {
                    int base = 0;
                    if (lane == 0) base = atomicAdd(&s_count, __popc(tm));
                    base = __shfl_sync(0xffffffffu, base, 0) + __popc(tm & ((1u << lane) - 1u));
                    if (take && base < kTileListCap) s_list[base] = ((unsigned)c << kTileClassBits) | cls;
                }
            }
        }
        __syncthreads();
        const int n_list = s_count;
        if (threadIdx.x == 0) {
            s_scale = class_scale;
#pragma unroll
            for (int u = 0; u < NV4; u++) s_mid[u] = mid.v[u];
        }
        if (n_list <= kTileListCap) {
            // counting sort by class; inside a class in any order (results do not depend on it)
            constexpr int kPerThread = kTileListCap / kTileThreads;
            unsigned e[kPerThread];
            int r[kPerThread];
#pragma unroll
            for (int i = 0; i < kPerThread; i++) {
                const int p = i * kTileThreads + threadIdx.x;
                if (p < n_list) {
                    e[i] = s_list[p];
                    r[i] = atomicAdd(&s_hist[e[i] & (kTileBuckets - 1)], 1);
                }
            }
            __syncthreads();
            int h = lane < kTileBuckets ? s_hist[lane] : 0, incl = h;
#pragma unroll
            for (int o = 1; o < kTileBuckets; o <<= 1) {
                const int t = __shfl_up_sync(0xffffffffu, incl, o);
                if (lane >= o) incl += t;
            }
            const int excl = incl - h;
            if (threadIdx.x < kTileBuckets) s_end[threadIdx.x] = incl;
#pragma unroll
            for (int i = 0; i < kPerThread; i++) {
                const int p = i * kTileThreads + threadIdx.x;
                if (i * kTileThreads >= n_list) break;  // uniform
                const int base = __shfl_sync(0xffffffffu, excl, p < n_list ? (int)(e[i] & (kTileBuckets - 1)) : 0);
                if (p < n_list) s_list[base + r[i]] = e[i];
            }
        }
    }

    __syncthreads();
    // ---- 3. queries ----
    TileQuery<NV4, L> Q;
    Q.buf = s_buf[warp];
    Q.near_ = s_near[warp];
    Q.lane = lane;
    Q.a = &a;
    for (;;) {
        int qi = 0;
        if (lane == 0) qi = atomicAdd(&s_next, 1);
        qi = first + __shfl_sync(0xffffffffu, qi, 0);
        if (qi >= first + n_q) break;
        const int self_id = a.ids[chunk * 32 + qi];
        Q.cnt = 0;
        Q.n_near = 0;
        bool searching = search;
        if (a.direction != nullptr) {
            const int dir = a.direction[self_id];
            if (dir == 0 || dir == 2) searching = false;  // may not have neighbours: defaults only
        }
        if (searching) {
#pragma unroll
            for (int u = 0; u < NV4; u++) Q.q.v[u] = s_mine[u][qi];
            // Queries of a tile are neighbours, so their K-th distances are alike.  Those answered already bound
            // this one's through the triangle inequality (`sure`); the search first keeps to a little more than
            // the nearest one's own, and with K - 1 hits inside these hold the answer.  Otherwise the radius
            // grows by what the count suggests, up to the bound that holds for certain.
            float sure = s_sure[qi], limit;
            {
                const float r = *(volatile float *)&s_radius[lane];
                Point<NV4> other;
#pragma unroll
                for (int u = 0; u < NV4; u++) other.v[u] = s_mine[u][lane];
                const float away = sqrt_fast(distsq<NV4>(Q.q, other));
                const bool known = r < INFINITY;
                const float b = warp_min_f32(known ? r + away : INFINITY);
                sure = fminf(sure, b * b * 1.00001f + 1e-37f);
                const unsigned pick = __reduce_min_sync(0xffffffffu, known ? (__float_as_uint(away) & ~31u) | (unsigned)lane
                                                                           : 0xffffffffu);
                limit = s_first[qi];
                const float rn = __shfl_sync(0xffffffffu, r, (int)(pick & 31u));
                if (pick != 0xffffffffu) limit = rn * rn * a.guess;
                limit = fminf(limit, sure);
            }
            Point<NV4> mid;
#pragma unroll
            for (int u = 0; u < NV4; u++) mid.v[u] = s_mid[u];
            const float from_mid = sqrt_fast(distsq<NV4>(Q.q, mid));
            for (int tries = 1;; tries++) {
                Q.thr = make_key(limit, 0x7fffffff);
                Q.cnt = 0;
                {   // its own chunk first, without itself
                    const int j = chunk * 32 + lane;
                    Q.append(distsq<NV4>(Q.q, load_point<NV4>(a.pts, (size_t)j)), __ldg(a.ranks + j), lane != qi);
                }
                // |centre - box| <= |centre - q| + |q - box|: classes beyond that are out of reach
                const float far_ = from_mid + sqrt_fast(limit);
                const float far_class = far_ * far_ * s_scale * 1.0001f + 0.001f;
                const int n_list = s_count;
                const bool listed = n_list <= kTileListCap;
                const int n_here = far_class < (float)(kTileBuckets - 1) ? s_end[(int)far_class] : n_list;
                unsigned m = 0u;  // super-chunks within reach that are not done (tiles without a list)
                int next = 0, s = 0;
                bool more = true;
                do {
                    int cid = chunk;
                    bool ok = false;
                    if (listed) {
                        ok = next + lane < n_here;
                        if (ok) cid = (int)(s_list[next + lane] >> kTileClassBits);
                        next += 32;
                        more = next < n_here;
                    } else {
                        // too many chunks for a list: walk the boxes of the event, from the query's own super-chunk on
                        const int4 ev = __ldg(a.chunk_info + chunk);
                        const int n_super = ev.w - ev.z;
                        if (m == 0u) {
                            s = ((chunk - ev.x) >> 5) + next + lane;
                            if (s >= n_super) s -= n_super;
                            m = __ballot_sync(0xffffffffu, next + lane < n_super && box_gap_distsq<NV4>(Q.q, Q.q,
                                    a.super_box + (size_t)(ev.z + s) * 2 * NV4) <= key_distsq(Q.thr));
                            next += 32;
                        }
                        if (m != 0u) {
                            const int c = ev.x + __shfl_sync(0xffffffffu, s, __ffs(m) - 1) * 32 + lane;
                            m &= m - 1u;
                            ok = c < ev.y && c != chunk;
                            if (ok) cid = c;
                        }
                        more = m != 0u || next < n_super;
                    }
                    const float lb = box_gap_distsq<NV4>(Q.q, Q.q, a.chunk_box + (size_t)cid * 2 * NV4);
                    Q.note(ok && lb <= key_distsq(Q.thr), cid);
                    if (Q.n_near > (more ? kTileNear - 36 : 0)) Q.look();
                } while (more);
                if (Q.cnt >= want || limit == sure) break;
                limit = tries >= 3 ? sure : fminf(sure, fmaxf(limit, 1e-37f) * exp2f(a.expo * __log2f(__fdividef(1.4f * (float)(want + 1), (float)(Q.cnt + 1)))));
            }
            // want == 32 * L leaves no word behind the last one needed, see load_sorted
            if (Q.cnt > 32 * L && (L > 2 || want == 32 * L))
                Q.cnt = prune_parked<L>(Q.buf, Q.cnt, want, 32 * L - want, 32 * L, Q.thr, a.expo, lane).cnt;
            __syncwarp();
        }
        // the row: slot 0 = the query, slots 1.. ascending by (distance, position)
        knn_key list[L];
        if constexpr (L <= 2) {
            load_sorted<L>(Q.buf, Q.cnt, key_distsq(Q.thr), list, lane);
        } else {
#pragma unroll
            for (int r = 0; r < L; r++) list[r] = r * 32 + lane < Q.cnt ? Q.buf[r * 32 + lane] : HGC_KNN_INF_KEY;
            sort_striped<L>(list, lane);
        }
        __syncwarp();  // the buffer is free again
        if (want > 0) {
            const knn_key kth = shfl_key(list_reg<L>(list, (want - 1) / 32), (want - 1) & 31);
            if (lane == 0 && kth != HGC_KNN_INF_KEY) *(volatile float *)&s_radius[qi] = sqrt_fast(key_distsq(kth));
        }
        int *row_idx = a.out_idx + (size_t)self_id * K;
        float *row_dist = a.out_dist + (size_t)self_id * K;
        const int pad = a.tf_compat ? self_id : -1;
        if (lane == 0) { row_idx[0] = self_id; row_dist[0] = 0.f; }
#pragma unroll
        for (int r = 0; r < L; r++) {
            const int slot = 1 + r * 32 + lane;
            if (slot < K) {
                int id = pad;
                float ds = 0.f;
                if (list[r] != HGC_KNN_INF_KEY) {
                    id = __ldg(a.rank_to_id + key_index(list[r]));
                    ds = key_distsq(list[r]);
                }
                row_idx[slot] = id;
                row_dist[slot] = ds;
            }
        }
    }
}

template <int NV4, int L>
int launch_tile_l(const TileKnnArgs &a, int n_tiles, cudaStream_t stream)
{
    HGC_CUDA_TRY(launch_overlapped(a.nobody, select_knn_tile_kernel<NV4, L>, n_tiles, kTileThreads, 0, stream, a));
    HGC_LAUNCH_CHECK();
    return HGC_OK;
}

template <int NV4>
int launch_tile_nv(const TileKnnArgs &a, int n_tiles, cudaStream_t stream)
{
    const int want = a.K - 1;
    if (want <= 32) return launch_tile_l<NV4, 1>(a, n_tiles, stream);
    if (want <= 64) return launch_tile_l<NV4, 2>(a, n_tiles, stream);
    if (want <= 128) return launch_tile_l<NV4, 4>(a, n_tiles, stream);
    if (want <= 256) return launch_tile_l<NV4, 8>(a, n_tiles, stream);
    if (want <= 512) return launch_tile_l<NV4, 16>(a, n_tiles, stream);
    return HGC_ERR_UNSUPPORTED;
}

}  // namespace hgc
