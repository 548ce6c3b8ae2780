// Two small ops that live on the same neighbour tables as the main path and are used by the
// graph-condensation layers: LocalDistance and PushKnn.
#include "common.cuh"
#include "edge_kernels.cuh"
#include "incoming.cuh"

namespace hgc {
namespace {

// Squared distance from hit i to its listed neighbour; 0 for padding and for the hit itself
// (modules/compiled/local_distance_kernel.cc:22-70).  Unfused operations in coordinate order.
__global__ void local_distance_kernel(const int *__restrict__ nidx, const float *__restrict__ coords,
                                      float *__restrict__ dist, int C, int n_in, long long n_edges, int K)
{
    pdl_begin();
    const long long e = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (e >= n_edges) return;
    const int i = (int)(e / K);
    const int j = nidx[e];
    float s = 0.f;
    if (j >= 0 && j < n_in && j != i) {
        for (int c = 0; c < C; c++) {
            const float t = __fsub_rn(coords[(size_t)i * C + c], coords[(size_t)j * C + c]);
            s = __fadd_rn(s, __fmul_rn(t, t));
        }
    }
    dist[e] = s;
}

// PushKnnGrad (modules/compiled/push_knn_grad_kernel.cc:22-95): both parts are gathers.  The part w.r.t. the weights,
// w_grad[i,k] = sum_f grad[m_k,f] * feat[i,f] with f in order, is edge_dot_kernel, and for narrow rows this one, a thread
// per (hit, slot) that reads the neighbour's row itself: a row of a few floats is one sector, and edge_dot_kernel's loads
// of 32 floats bring in nothing else (both parts, 200k hits, K = 64: F = 1 323 us against 493, F = 5 378 against 503, F = 13
// 517 against 521; at F = 16 516 against 513).
constexpr int kNarrow = 16;
__global__ void __launch_bounds__(256)
push_grad_weights_kernel(const float *__restrict__ grad, const float *__restrict__ feat, const int *__restrict__ nidx,
                         float *__restrict__ w_grad, long long n_edges, int n_vert, int K, int F,
                         const int *__restrict__ order)
{
    pdl_begin();
    const long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= n_edges) return;
    const int row = (int)(t / K), i = order ? order[row] : row;  // processing order only
    const long long e = (long long)i * K + (t - (long long)row * K);
    const int m = nidx[e];
    float acc = 0.f;
    if (m >= 0 && m < n_vert)
        for (int f = 0; f < F; f++)
            acc = __fadd_rn(acc, __fmul_rn(__ldg(grad + (size_t)m * F + f), feat[(size_t)i * F + f]));
    w_grad[e] = acc;
}

// feat_grad[i,f] = sum_k grad[m_k,f] * w[i,k]: one warp per hit, lanes over the features, k in order.  All lanes read slot
// and weight, from one address.  (Handing them out by shuffles, with the rows of eight neighbours requested together, takes
// longer at every width: 200k hits, K = 64, both gradients, F = 5 448 us against 378, 32 615 against 548, 64 1172 against 1029,
// 200 4583 against 4242.)
__global__ void __launch_bounds__(256)
push_grad_features_kernel(const float *__restrict__ grad, const float *__restrict__ weights,
                          const int *__restrict__ nidx, float *__restrict__ feat_grad, int n_vert, int K, int F,
                          const int *__restrict__ order)
{
    pdl_begin();
    const int lane = threadIdx.x & 31;
    const int slot = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
    if (slot >= n_vert) return;
    const int i = order ? order[slot] : slot;  // processing order only
    for (int f = lane; f < F; f += 32) {
        float acc = 0.f;
        for (int k = 0; k < K; k++) {
            const int m = nidx[(size_t)i * K + k];
            if (m < 0 || m >= n_vert) continue;
            acc = __fadd_rn(acc, __fmul_rn(grad[(size_t)m * F + f], weights[(size_t)i * K + k]));
        }
        feat_grad[(size_t)i * F + f] = acc;
    }
}

}  // namespace
}  // namespace hgc

using namespace hgc;

extern "C" int hgc_push_knn_grad(
        const float *d_grad, const float *d_weights, const float *d_feat, const int *d_idxs,
        float *d_feat_grad, float *d_w_grad, int n_vert, int n_neigh, int n_feat, hgc_stream_t stream)
{
    return hgc_push_knn_grad_ordered(d_grad, d_weights, d_feat, d_idxs, d_feat_grad, d_w_grad, n_vert, n_neigh, n_feat,
                                     nullptr, stream);
}

extern "C" int hgc_push_knn_grad_ordered(
        const float *d_grad, const float *d_weights, const float *d_feat, const int *d_idxs,
        float *d_feat_grad, float *d_w_grad, int n_vert, int n_neigh, int n_feat, const int *d_order, hgc_stream_t stream_)
{
    cudaStream_t stream = static_cast<cudaStream_t>(stream_);
    if (n_vert < 0 || n_neigh < 0 || n_feat < 0) return HGC_ERR_INVALID_ARGUMENT;
    if (n_vert == 0) return HGC_OK;
    const long long ne = (long long)n_vert * n_neigh;
    if (n_feat > 0 && (!d_grad || !d_feat || !d_feat_grad)) return HGC_ERR_INVALID_ARGUMENT;
    if (ne > 0 && (!d_weights || !d_idxs || !d_w_grad)) return HGC_ERR_INVALID_ARGUMENT;
    if (n_feat > 0) {
        HGC_CUDA_TRY(launch_overlapped(n_vert, push_grad_features_kernel, div_up(n_vert, 8), 256, 0, stream, d_grad, d_weights, d_idxs, d_feat_grad,
                                                                        n_vert, n_neigh, n_feat, d_order));
        HGC_LAUNCH_CHECK();
    }
    if (ne > 0) {
        const bool vec4 = n_feat % 4 == 0 && ((reinterpret_cast<uintptr_t>(d_feat) | reinterpret_cast<uintptr_t>(d_grad)) & 15u) == 0;
        if (n_feat < kNarrow)
            HGC_CUDA_TRY(launch_overlapped(n_vert, push_grad_weights_kernel, div_up(ne, 256), 256, 0, stream, d_grad, d_feat, d_idxs, d_w_grad, ne,
                                           n_vert, n_neigh, n_feat, d_order));
        else
            HGC_CUDA_TRY(launch_overlapped(n_vert, vec4 ? edge_dot_kernel<false, false, true> : edge_dot_kernel<false, false, false>,
                                           div_up(ne, 256), 256, 0, stream, d_feat, n_feat, d_grad, nullptr, d_idxs, d_w_grad,
                                           ne, n_vert, n_neigh, n_feat, d_order, nullptr));
        HGC_LAUNCH_CHECK();
    }
    return HGC_OK;
}

extern "C" int hgc_local_distance(
        const int *d_neigh_idxs, const float *d_coords, float *d_distances,
        int n_coords, int n_in_vert, int n_out_vert, int n_neigh, hgc_stream_t stream_)
{
    cudaStream_t stream = static_cast<cudaStream_t>(stream_);
    if (n_coords < 0 || n_in_vert < 0 || n_out_vert < 0 || n_neigh < 0 || n_out_vert > n_in_vert)
        return HGC_ERR_INVALID_ARGUMENT;
    const long long ne = (long long)n_out_vert * n_neigh;
    if (ne == 0) return HGC_OK;
    if (!d_neigh_idxs || !d_distances || (n_coords > 0 && !d_coords)) return HGC_ERR_INVALID_ARGUMENT;
    HGC_CUDA_TRY(launch_pdl(local_distance_kernel, div_up(ne, 256), 256, 0, stream, d_neigh_idxs, d_coords, d_distances, n_coords,
                                                              n_in_vert, ne, n_neigh));
    HGC_LAUNCH_CHECK();
    return HGC_OK;
}

static size_t push_bytes(int n_vert, int n_neigh, int n_feat, bool aligned)
{
    return incoming_bytes(n_vert, n_neigh, copied_row(n_feat, aligned, false), false);
}

extern "C" size_t hgc_push_knn_workspace_bytes(int n_vert, int n_neigh, int n_feat) { return push_bytes(n_vert, n_neigh, n_feat, true); }

extern "C" int hgc_push_knn(
        const float *d_weights, const float *d_feat, const int *d_idxs, float *d_out_feat,
        int n_vert, int n_neigh, int n_feat, void *workspace, size_t workspace_bytes, hgc_stream_t stream)
{
    return hgc_push_knn_ordered(d_weights, d_feat, d_idxs, d_out_feat, n_vert, n_neigh, n_feat, nullptr, workspace,
                                workspace_bytes, stream);
}

extern "C" int hgc_push_knn_ordered(
        const float *d_weights, const float *d_feat, const int *d_idxs, float *d_out_feat,
        int n_vert, int n_neigh, int n_feat, const int *d_order, void *workspace, size_t workspace_bytes, hgc_stream_t stream_)
{
    cudaStream_t stream = static_cast<cudaStream_t>(stream_);
    if (n_vert < 0 || n_neigh < 0 || n_feat < 0) return HGC_ERR_INVALID_ARGUMENT;
    if ((long long)n_vert * n_neigh >= (1LL << 31) - 4096) return HGC_ERR_UNSUPPORTED;
    if (n_vert == 0 || n_feat == 0) return HGC_OK;
    if (!d_feat || !d_out_feat || (n_neigh > 0 && (!d_weights || !d_idxs))) return HGC_ERR_INVALID_ARGUMENT;
    if (n_neigh == 0) {
        HGC_CUDA_TRY(cudaMemsetAsync(d_out_feat, 0, sizeof(float) * (size_t)n_vert * n_feat, stream));
        return HGC_OK;
    }
    const size_t need = push_bytes(n_vert, n_neigh, n_feat, aligned16(d_feat));
    if (int rc = check_workspace(workspace, workspace_bytes, need)) return rc;
    Carver ws(workspace);
    // sums in (hit, slot) order (modules/compiled/push_knn_kernel.cc:35-71; the reference's GPU kernel scatters with
    // atomicAdd, push_knn_kernel.cu.cc:61)
    const Incoming b = incoming_layout(ws, n_vert, n_neigh, 0, false);
    if (int rc = build_incoming(d_idxs, n_vert, n_neigh, b, ws.status(), stream)) return rc;
    for (int f0 = 0; f0 < n_feat; f0 += 64)
        if (int rc = launch_edge_sum_slab<kSumPlain>(d_feat, n_feat, d_weights, nullptr, nullptr, b, d_out_feat, n_vert, n_neigh, n_feat, f0,
                                                     d_order, stream))
            return rc;
    return HGC_OK;
}
