// Transposition of the neighbour table: a counting sort of the edges by target.
//
// Targets are counted with integer atomics, which also hand every edge a place in its target's list; a prefix sum
// gives the lists their room, the edges are written to their places, and every list is then sorted by edge id,
// which takes out the order in which the atomics happened: the result is the same on every run.  Lists hold about
// as many edges as a hit has neighbours, up to three times as many where hits lie densely, so a warp sorts one in
// registers; longer lists than that (kWarpList) go to a block of their own.
//
// Bound by the scattered accesses to L2 (one atomic and one 4-byte write per edge) while lists fit a warp.
// 200k hits, lists built in: K = 16 0.095 ms, K = 64 0.32 ms, K = 128 0.68 ms, K = 256 1.6 ms.  The whole of
// SelectKnnGrad: 0.52 ms at K = 64, 1.09 at 128, 2.7 at 256, against 1.05, 2.1 and 5.0 ms with three passes of the
// stable radix sort over (target, edge) pairs and a search for the list bounds, which also took 17 launches instead
// of 7.
#include "incoming.cuh"
#include "knn_device.cuh"

namespace hgc {
namespace {

__global__ void __launch_bounds__(256)
count_targets_kernel(const int *__restrict__ nidx, long long n_edges, int n_vert, int *__restrict__ count,
                     int *__restrict__ place)
{
    pdl_begin();
    const long long e = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (e >= n_edges) return;
    const int m = nidx[e];
    if (m >= 0 && m < n_vert) place[e] = atomicAdd(count + m, 1);  // others belong to no list
}

__global__ void __launch_bounds__(256)
place_edges_kernel(const int *__restrict__ nidx, const int *__restrict__ place, long long n_edges, int n_vert,
                   const int *__restrict__ bounds, int *__restrict__ edges)
{
    pdl_begin();
    const long long e = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (e >= n_edges) return;
    const int m = nidx[e];
    if (m >= 0 && m < n_vert) edges[bounds[m] + place[e]] = (int)e;
}

// Merges neighbouring ascending runs of M registers: compare with the mirrored run, then clean both bitonic halves.
// A template parameter for the run, because the compiler stops unrolling a loop over it at 16 registers.
template <int R, int M>
__device__ __forceinline__ void merge_runs(unsigned (&v)[R], int lane)
{
#pragma unroll
    for (int g = 0; g < R; g += 2 * M) {
#pragma unroll
        for (int i = 0; i < M; i++) {
            const unsigned lo = v[g + i], hi = __shfl_xor_sync(0xffffffffu, v[g + 2 * M - 1 - i], 31);
            v[g + i] = min(lo, hi);
            v[g + 2 * M - 1 - i] = __shfl_xor_sync(0xffffffffu, max(lo, hi), 31);
        }
#pragma unroll
        for (int h = M >> 1; h > 0; h >>= 1)
#pragma unroll
            for (int i = 0; i < 2 * M; i++)
                if (!(i & h)) {
                    const unsigned lo = v[g + i], hi = v[g + i + h];
                    v[g + i] = min(lo, hi);
                    v[g + i + h] = max(lo, hi);
                }
#pragma unroll
        for (int i = 0; i < 2 * M; i++) v[g + i] = warp_bitonic_merge_u32(v[g + i], lane);
    }
    if constexpr (2 * M < R) merge_runs<R, 2 * M>(v, lane);
}

// Sorts 32 * R ids held by a warp (striped) and writes back the first n.
template <int R>
__device__ __forceinline__ void sort_list(int *list, int n, int lane)
{
    unsigned v[R];
#pragma unroll
    for (int r = 0; r < R; r++)
        v[r] = warp_sort_u32(r * 32 + lane < n ? (unsigned)list[r * 32 + lane] : 0xffffffffu, lane);
    if constexpr (R > 1) merge_runs<R, 1>(v, lane);
#pragma unroll
    for (int r = 0; r < R; r++)
        if (r * 32 + lane < n) list[r * 32 + lane] = (int)v[r];
}

// A warp per list.  32 registers, so that all 64 warps of an SM have a list: sixteen ids per lane then cost a few spills,
// but with the 48 registers that they would take the short lists wait longer (K = 16, 200k hits: 95 -> 104 us).
// Lists of 129 to 512 edges, a block each before: K = 96, 200k hits 4.4 -> 0.8 ms, K = 128 8.1 -> 1.1 ms for SelectKnnGrad.
__global__ void __launch_bounds__(256, 8)
sort_lists_kernel(const int *__restrict__ bounds, int *__restrict__ edges, int n_vert, WideLists wide)
{
    pdl_begin();
    const int m = blockIdx.x * 8 + (threadIdx.x >> 5), lane = threadIdx.x & 31;
    if (m >= n_vert) return;
    const int begin = bounds[m], n = bounds[m + 1] - begin;
    if (n <= 1) return;
    if (n <= 32) sort_list<1>(edges + begin, n, lane);
    else if (n <= 64) sort_list<2>(edges + begin, n, lane);
    else if (n <= 128) sort_list<4>(edges + begin, n, lane);
    else if (n <= 256) sort_list<8>(edges + begin, n, lane);
    else if (n <= kWarpList) sort_list<16>(edges + begin, n, lane);
    if (n > wide.limit && lane == 0) {
        if (n > kWarpList) wide.hits[atomicAdd(wide.counts, 1)] = m;
        else wide.hits[wide.room - 1 - atomicAdd(wide.counts + 1, 1)] = m;
    }
}

// Lists of more than kWarpList edges: a block per list, radix sort of 8-bit digits through global memory.
__global__ void __launch_bounds__(256)
sort_long_lists_kernel(const int *__restrict__ bounds, int *edges, int *tmp, WideLists wide, int n_passes)
{
    pdl_begin();
    __shared__ int s_run[256], s_count[8][256], s_warp[8];
    const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
    const int n_long = wide.counts[0];
    for (int l = blockIdx.x; l < n_long; l += gridDim.x) {
        const int m = wide.hits[l], begin = bounds[m], n = bounds[m + 1] - begin;
        int *src = edges + begin, *dst = tmp + begin;
        for (int p = 0; p < n_passes; p++) {
            const int shift = 8 * p;
            __syncthreads();
            s_run[t] = 0;
            __syncthreads();
            for (int i = t; i < n; i += 256) atomicAdd(&s_run[(src[i] >> shift) & 255], 1);
            __syncthreads();
            const int c = s_run[t];
            int incl = c;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const int v = __shfl_up_sync(0xffffffffu, incl, o);
                if (lane >= o) incl += v;
            }
            if (lane == 31) s_warp[warp] = incl;
            __syncthreads();
            for (int w = 0; w < warp; w++) incl += s_warp[w];
            s_run[t] = incl - c;
            // 256 ids at a time, warp by warp in order
            for (int base = 0; base < n; base += 256) {
                for (int w = 0; w < 8; w++) s_count[w][t] = 0;
                __syncthreads();
                const bool ok = base + t < n;
                const int id = ok ? src[base + t] : 0;
                const unsigned dg = ok ? (unsigned)(id >> shift) & 255u : 256u;
                const unsigned peers = __match_any_sync(0xffffffffu, dg), before = peers & ((1u << lane) - 1u);
                if (ok && before == 0u) s_count[warp][dg] = __popc(peers);
                __syncthreads();
                int run = s_run[t];
                for (int w = 0; w < 8; w++) {
                    const int k = s_count[w][t];
                    s_count[w][t] = run;
                    run += k;
                }
                s_run[t] = run;
                __syncthreads();
                if (ok) dst[s_count[warp][dg] + __popc(before)] = id;
                __syncthreads();
            }
            int *x = src; src = dst; dst = x;
        }
        if (n_passes & 1)
            for (int i = t; i < n; i += 256) edges[begin + i] = tmp[begin + i];
    }
}

}  // namespace

int build_incoming(const int *nidx, int n_vert, int n_neigh, const Incoming &b, unsigned *status, cudaStream_t stream)
{
    const long long ne = (long long)n_vert * n_neigh;
    // the status word, the counts (bounds) and those of wide lists lie one after another
    HGC_CUDA_TRY(cudaMemsetAsync(status, 0, (size_t)(reinterpret_cast<char *>(b.wide.counts + 2) - reinterpret_cast<char *>(status)), stream));
    HGC_CUDA_TRY(launch_overlapped(n_vert, count_targets_kernel, div_up(ne, 256), 256, 0, stream, nidx, ne, n_vert, b.bounds, b.place));
    HGC_LAUNCH_CHECK();
    if (int rc = exclusive_scan_ints(b.bounds, n_vert + 1, b.scan, stream)) return rc;
    HGC_CUDA_TRY(launch_overlapped(n_vert, place_edges_kernel, div_up(ne, 256), 256, 0, stream, nidx, b.place, ne, n_vert, b.bounds, b.edges));
    HGC_LAUNCH_CHECK();
    HGC_CUDA_TRY(launch_overlapped(n_vert, sort_lists_kernel, div_up(n_vert, 8), 256, 0, stream, b.bounds, b.edges, n_vert, b.wide));
    HGC_LAUNCH_CHECK();
    if (ne > kWarpList) {
        // Eight blocks per SM where there are edges enough: 60k hits, K = 500, 44 % of the lists longer than this:
        // 6.5 ms with one block per SM, 2.7 with four, 2.0 with eight.  Idle blocks cost 2 us per 1000, which a small
        // table would notice (1 M edges: 38 -> 40 us), so no more than one for every four of the longest warp lists.
        const long long want = ne / (4 * kWarpList), resident = 8 * sm_count();
        const int blocks = (int)(want < 1 ? 1 : want < resident ? want : resident);
        HGC_CUDA_TRY(launch_pdl(sort_long_lists_kernel, blocks, 256, 0, stream, b.bounds, b.edges, b.place, b.wide, (bits_for(ne) + 7) / 8));
        HGC_LAUNCH_CHECK();
    }
    return HGC_OK;
}

}  // namespace hgc
