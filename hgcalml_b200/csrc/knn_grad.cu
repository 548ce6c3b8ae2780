// Backward ops of the neighbour path: AccumulateKnnGrad and SelectKnnGrad.
//
// Both ops push gradients from a hit to its neighbours.  The reference's GPU kernels do that with
// float atomicAdd (modules/compiled/accumulate_knn_grad_kernel.cu.cc:102,
// select_knn_grad_kernel.cu.cc:139), so their sums depend on scheduling.  Here the neighbour lists
// are transposed first (incoming.cu): every hit gets the list of edges that point at it, in ascending
// (hit, slot) order, and sums its incoming contributions itself, in that fixed order -- run-to-run
// identical, and for AccumulateKnnGrad the same order as the reference's CPU loop
// (modules/compiled/accumulate_knn_grad_kernel.cc:36-163), so the result is bit-identical to it.
#include "common.cuh"
#include "edge_kernels.cuh"
#include "incoming.cuh"
#include "../../include/hgcalml_b200.h"

namespace hgc {
namespace {

// ---- SelectKnnGrad ------------------------------------------------------------------------------
// One thread per (hit, coordinate): its own part first, in the reference's mixed float/double
// arithmetic (modules/compiled/select_knn_grad_kernel.cu.cc:81-118), then the parts pushed to it by
// the hits that list it as a neighbour (:120-165), in (hit, slot) order instead of atomics.
__global__ void __launch_bounds__(256)
select_grad_kernel(const float *__restrict__ grad_dist, const int *__restrict__ nidx,
                   const float *__restrict__ coord, const int *__restrict__ bounds,
                   const int *__restrict__ edges, float *__restrict__ grad_coord, int n_vert, int K, int C, bool vec4,
                   const int *__restrict__ order)
{
    pdl_begin();
    const long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= (long long)n_vert * C) return;
    const int row = (int)(t / C), c = (int)(t - (long long)row * C);
    const int m = order ? order[row] : row;  // processing order only
    const float xm = coord[(size_t)m * C + c];
    float val = 0.f;
    // four neighbours, then four incoming edges, are requested together; their terms are added one by one
    constexpr int U = 4;
    for (int k0 = 0; k0 < K; k0 += U) {
        int j[U];
        float g[U], x[U];
        if (vec4) {
            const int4 jv = __ldg(reinterpret_cast<const int4 *>(nidx + (size_t)m * K + k0));
            const float4 gv = __ldg(reinterpret_cast<const float4 *>(grad_dist + (size_t)m * K + k0));
            j[0] = jv.x; j[1] = jv.y; j[2] = jv.z; j[3] = jv.w;
            g[0] = gv.x; g[1] = gv.y; g[2] = gv.z; g[3] = gv.w;
        } else {
#pragma unroll
            for (int u = 0; u < U; u++) {
                j[u] = k0 + u < K ? nidx[(size_t)m * K + k0 + u] : -1;
                g[u] = k0 + u < K ? grad_dist[(size_t)m * K + k0 + u] : 0.f;
            }
        }
#pragma unroll
        for (int u = 0; u < U; u++) {
            if (j[u] >= n_vert) j[u] = -1;
            x[u] = j[u] >= 0 ? __ldg(coord + (size_t)j[u] * C + c) : 0.f;
        }
#pragma unroll
        for (int u = 0; u < U; u++)
            if (j[u] >= 0) {
                // the reference rounds val - (2 g) d in double, and to float; the products of floats are exact in double
                const float d = __fsub_rn(x[u], xm);
                val = (float)__fma_rn(-2.0 * (double)g[u], (double)d, (double)val);
            }
    }
    const int end = bounds[m + 1];
    for (int p = bounds[m]; p < end; p += U) {
        float g[U], x[U];
#pragma unroll
        for (int u = 0; u < U; u++) {
            const int e = edges[min(p + u, end - 1)];
            g[u] = __ldg(grad_dist + e);
            x[u] = __ldg(coord + (size_t)(e / K) * C + c);
        }
#pragma unroll
        for (int u = 0; u < U; u++)
            if (p + u < end) {
                // (2 g) d, exact in double, rounded to float: the float product with one factor doubled, which is exact as long
                // as it does not overflow.  d is doubled below one, g above: where 2 g overflows then, so does the product.
                const float d = __fsub_rn(xm, x[u]);
                const bool near = fabsf(d) < 1.f;
                const float a = near ? d : g[u], b = near ? g[u] : d;
                val = __fadd_rn(val, __fmul_rn(a + a, b));
            }
    }
    grad_coord[(size_t)m * C + c] = val;
}

}  // namespace

}  // namespace hgc

using namespace hgc;

extern "C" size_t hgc_knn_grad_workspace_bytes(int n_vert, int n_neigh)
{
    return incoming_bytes(n_vert, n_neigh, 64);  // the widest rows beside flags
}

extern "C" size_t hgc_select_knn_grad_workspace_bytes(int n_vert, int n_neigh) { return incoming_bytes(n_vert, n_neigh); }

static size_t accumulate_grad_bytes(int n_vert, int n_neigh, int n_feat, int mean_and_max, bool aligned)
{
    return incoming_bytes(n_vert, n_neigh, copied_row(n_feat, aligned, !power_of_two(n_neigh)), mean_and_max);
}

extern "C" size_t hgc_accumulate_knn_grad_workspace_bytes(int n_vert, int n_neigh, int n_feat, int mean_and_max)
{
    return accumulate_grad_bytes(n_vert, n_neigh, n_feat, mean_and_max, true);
}

static int check_edge_count(int n_vert, int n_neigh)
{
    if (n_vert < 0 || n_neigh < 0) return HGC_ERR_INVALID_ARGUMENT;
    if ((long long)n_vert * n_neigh >= (1LL << 31) - 4096) return HGC_ERR_UNSUPPORTED;
    return HGC_OK;
}

extern "C" int hgc_accumulate_knn_grad(
        const float *d_grad_from_out_features, const float *d_distances, const float *d_feat,
        const int *d_max_feat_indices, const int *d_neigh_indices,
        float *d_out_grad_distances, float *d_out_grad_features,
        int n_vert, int n_neigh, int n_feat, int n_grad_from_out_feat, int n_moments, int mean_and_max,
        void *workspace, size_t workspace_bytes, hgc_stream_t stream_)
{
    return hgc_accumulate_knn_grad_ordered(d_grad_from_out_features, d_distances, d_feat, d_max_feat_indices,
                                           d_neigh_indices, d_out_grad_distances, d_out_grad_features, n_vert,
                                           n_neigh, n_feat, n_grad_from_out_feat, n_moments, mean_and_max,
                                           nullptr, workspace, workspace_bytes, stream_);
}

extern "C" int hgc_accumulate_knn_grad_ordered(
        const float *d_grad_from_out_features, const float *d_distances, const float *d_feat,
        const int *d_max_feat_indices, const int *d_neigh_indices,
        float *d_out_grad_distances, float *d_out_grad_features,
        int n_vert, int n_neigh, int n_feat, int n_grad_from_out_feat, int n_moments, int mean_and_max,
        const int *d_order, void *workspace, size_t workspace_bytes, hgc_stream_t stream_)
{
    (void)n_moments;
    cudaStream_t stream = static_cast<cudaStream_t>(stream_);
    if (int rc = check_edge_count(n_vert, n_neigh)) return rc;
    if (n_feat < 0 || n_grad_from_out_feat != (mean_and_max ? 2 * n_feat : n_feat)) return HGC_ERR_INVALID_ARGUMENT;
    if (n_vert == 0) return HGC_OK;
    if (n_feat > 0 && (!d_grad_from_out_features || !d_feat || !d_out_grad_features ||
                       (mean_and_max && !d_max_feat_indices)))
        return HGC_ERR_INVALID_ARGUMENT;
    if (n_neigh > 0 && (!d_distances || !d_neigh_indices || !d_out_grad_distances)) return HGC_ERR_INVALID_ARGUMENT;
    const bool mm = mean_and_max != 0;
    const size_t need = accumulate_grad_bytes(n_vert, n_neigh, n_feat, mm, aligned16(d_grad_from_out_features));
    if (int rc = check_workspace(workspace, workspace_bytes, need)) return rc;
    Carver ws(workspace);
    const Incoming b = incoming_layout(ws, n_vert, n_neigh, 0, mm);
    if (n_neigh == 0) {
        HGC_CUDA_TRY(cudaMemsetAsync(ws.status(), 0, kAlign, stream));
        if (n_feat > 0)
            HGC_CUDA_TRY(cudaMemsetAsync(d_out_grad_features, 0, sizeof(float) * (size_t)n_vert * n_feat, stream));
        return HGC_OK;
    }
    if (int rc = build_incoming(d_neigh_indices, n_vert, n_neigh, b, ws.status(), stream)) return rc;
    const long long ne = (long long)n_vert * n_neigh;
    const bool vec4 = n_feat % 4 == 0 && aligned16(d_feat) && aligned16(d_grad_from_out_features) && (!mm || aligned16(d_max_feat_indices));
    HGC_CUDA_TRY(launch_overlapped(n_vert, mm ? vec4 ? edge_dot_kernel<true, true, true> : edge_dot_kernel<true, true, false>
                                              : vec4 ? edge_dot_kernel<true, false, true> : edge_dot_kernel<true, false, false>,
                                   div_up(ne, 256), 256, 0, stream, d_grad_from_out_features, n_grad_from_out_feat, d_feat,
                                   mm ? d_max_feat_indices : nullptr, d_neigh_indices, d_out_grad_distances, ne, n_vert, n_neigh,
                                   n_feat, d_order, mm ? b.flags : nullptr));
    HGC_LAUNCH_CHECK();
    for (int f0 = 0; f0 < n_feat; f0 += 64) {
        if (mm && f0 > 0) {  // the bits of the first slab are a by-product of the weights' gradient
            HGC_CUDA_TRY(launch_overlapped(n_vert, arg_flags_kernel, div_up(n_vert, 8), 256, 0, stream, d_max_feat_indices, d_neigh_indices, b.flags, n_vert,
                                                                    n_neigh, n_feat, f0));
            HGC_LAUNCH_CHECK();
        }
        const int rc = mm ? launch_edge_sum_slab<kSumMeanMax>(d_grad_from_out_features, n_grad_from_out_feat, d_distances,
                                                              b.flags, d_neigh_indices, b, d_out_grad_features, n_vert, n_neigh, n_feat, f0,
                                                              d_order, stream)
                          : launch_edge_sum_slab<kSumMean>(d_grad_from_out_features, n_grad_from_out_feat, d_distances,
                                                           nullptr, d_neigh_indices, b, d_out_grad_features, n_vert, n_neigh, n_feat, f0,
                                                           d_order, stream);
        if (rc) return rc;
    }
    return HGC_OK;
}

extern "C" int hgc_select_knn_grad(
        const float *d_grad_dist, const int *d_indices, const float *d_dist, const float *d_coord,
        float *d_grad_coord, int n_vert, int n_neigh, int n_coords,
        void *workspace, size_t workspace_bytes, hgc_stream_t stream)
{
    return hgc_select_knn_grad_ordered(d_grad_dist, d_indices, d_dist, d_coord, d_grad_coord, n_vert, n_neigh, n_coords,
                                       nullptr, workspace, workspace_bytes, stream);
}

// lists_ready: the workspace holds the transposed lists of this neighbour table already.
static int select_knn_grad(const float *d_grad_dist, const int *d_indices, const float *d_coord, float *d_grad_coord,
                           int n_vert, int n_neigh, int n_coords, const int *d_order, void *workspace,
                           size_t workspace_bytes, bool lists_ready, hgc_stream_t stream_)
{
    cudaStream_t stream = static_cast<cudaStream_t>(stream_);
    if (int rc = check_edge_count(n_vert, n_neigh)) return rc;
    if (n_coords < 0) return HGC_ERR_INVALID_ARGUMENT;
    if (n_vert == 0 || n_coords == 0) return HGC_OK;
    if (!d_coord || !d_grad_coord || (n_neigh > 0 && (!d_grad_dist || !d_indices))) return HGC_ERR_INVALID_ARGUMENT;
    const size_t need = hgc_select_knn_grad_workspace_bytes(n_vert, n_neigh);
    if (int rc = check_workspace(workspace, workspace_bytes, need)) return rc;
    Carver ws(workspace);
    const Incoming b = incoming_layout(ws, n_vert, n_neigh);
    if (n_neigh == 0) {
        HGC_CUDA_TRY(cudaMemsetAsync(ws.status(), 0, kAlign, stream));
        HGC_CUDA_TRY(cudaMemsetAsync(d_grad_coord, 0, sizeof(float) * (size_t)n_vert * n_coords, stream));
        return HGC_OK;
    }
    if (!lists_ready)
        if (int rc = build_incoming(d_indices, n_vert, n_neigh, b, ws.status(), stream)) return rc;
    const long long total = (long long)n_vert * n_coords;
    HGC_CUDA_TRY(launch_overlapped(n_vert, select_grad_kernel, div_up(total, 256), 256, 0, stream, d_grad_dist, d_indices, d_coord, b.bounds, b.edges,
                                                              d_grad_coord, n_vert, n_neigh, n_coords,
                                                              n_neigh % 4 == 0 && ((reinterpret_cast<uintptr_t>(d_grad_dist) | reinterpret_cast<uintptr_t>(d_indices)) & 15u) == 0, d_order));
    HGC_LAUNCH_CHECK();
    return HGC_OK;
}

extern "C" int hgc_select_knn_grad_ordered(
        const float *d_grad_dist, const int *d_indices, const float *d_dist, const float *d_coord,
        float *d_grad_coord, int n_vert, int n_neigh, int n_coords, const int *d_order,
        void *workspace, size_t workspace_bytes, hgc_stream_t stream)
{
    (void)d_dist;  // an input of the op that its kernels never read
    return select_knn_grad(d_grad_dist, d_indices, d_coord, d_grad_coord, n_vert, n_neigh, n_coords, d_order, workspace,
                           workspace_bytes, false, stream);
}

extern "C" int hgc_select_knn_grad_after(
        const float *d_grad_dist, const int *d_indices, const float *d_dist, const float *d_coord,
        float *d_grad_coord, int n_vert, int n_neigh, int n_coords, const int *d_order,
        void *workspace, size_t workspace_bytes, hgc_stream_t stream)
{
    (void)d_dist;
    return select_knn_grad(d_grad_dist, d_indices, d_coord, d_grad_coord, n_vert, n_neigh, n_coords, d_order, workspace,
                           workspace_bytes, true, stream);
}
