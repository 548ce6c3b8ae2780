// Device side of the grid derivation and of the hit orderings, shared by the kernels that use them.
#pragma once
#include "common.cuh"
#include "binning.cuh"
#include "knn_device.cuh"

namespace hgc {

constexpr int kGridSetupThreads = 256;

// Minimum and maximum of every coordinate over the hits this block (of 256 threads) looks at.
__device__ __forceinline__ void range_of_block(const float *__restrict__ coords, int coord_stride, int n_dims, int n_vert,
                     float *partial /* [gridDim.x][2][kMaxBinDims] */)
{
    float mn[kMaxBinDims], mx[kMaxBinDims];
#pragma unroll
    for (int c = 0; c < kMaxBinDims; c++) { mn[c] = INFINITY; mx[c] = -INFINITY; }
    for (int v = blockIdx.x * blockDim.x + threadIdx.x; v < n_vert; v += gridDim.x * blockDim.x) {
#pragma unroll
        for (int c = 0; c < kMaxBinDims; c++)
            if (c < n_dims) {
                const float x = coords[(size_t)v * coord_stride + c];
                mn[c] = fminf(mn[c], x);
                mx[c] = fmaxf(mx[c], x);
            }
    }
    __shared__ float s_mn[8][kMaxBinDims], s_mx[8][kMaxBinDims];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
    for (int c = 0; c < kMaxBinDims; c++) {
        if (c < n_dims) { mn[c] = warp_min_f32(mn[c]); mx[c] = warp_max_f32(mx[c]); }
        if (lane == 0) { s_mn[warp][c] = mn[c]; s_mx[warp][c] = mx[c]; }
    }
    __syncthreads();
    if (threadIdx.x < kMaxBinDims) {
        const int c = threadIdx.x;
        float a = s_mn[0][c], b = s_mx[0][c];
        for (int w = 1; w < 8; w++) { a = fminf(a, s_mn[w][c]); b = fmaxf(b, s_mx[w][c]); }
        partial[((size_t)blockIdx.x * 2 + 0) * kMaxBinDims + c] = a;
        partial[((size_t)blockIdx.x * 2 + 1) * kMaxBinDims + c] = b;
    }
}

// The grid from the range of the batch, exactly as the Python wrappers derive it
// (modules/bin_by_coordinates_op.py:49-71, modules/binned_select_knn_op.py:57-63), in float32.  One warp; lane c holds minimum
// and maximum of coordinate c, zeros beyond n_all.
__device__ __forceinline__ void grid_from_range(float mn, float mx, int n_dims, int n_all, const int *__restrict__ row_splits, int n_rs,
                                                int n_bins_arg, int n_neigh, int pre_normalized, GridParams *__restrict__ g)
{
    const int c = threadIdx.x & 31;
    // The wrapper shifts by the minimum first; x -> x - mn is monotone, so the shifted extremes
    // are the extremes shifted.
    const float shift = pre_normalized ? 0.f : mn;
    const float smin = __fsub_rn(mn, shift);
    float dmax = __fsub_rn(mx, shift);
    if (smin == dmax) dmax = __fadd_rn(dmax, 1.f);
    dmax = __fadd_rn(dmax, 1e-3f);
    if (!isfinite(dmax)) dmax = 1.f;

    int n_bins = n_bins_arg;
    if (n_bins <= 0) {
        const float first_event = n_rs > 1 ? (float)row_splits[1] : 1.f;
        const float t = powf(__fdiv_rn(first_event, (float)n_neigh / 32.f), 1.f / (float)n_dims);
        n_bins = (int)t;
        n_bins = n_bins < 5 ? 5 : (n_bins > 30 ? 30 : n_bins);
    }
    float bw = c < n_dims ? __fdiv_rn(dmax, (float)n_bins) : -INFINITY;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) bw = fmaxf(bw, __shfl_xor_sync(0xffffffffu, bw, o));
    int nb = 1;
    if (c < n_dims) nb = (int)__fadd_rn(__fdiv_rn(dmax, bw), 1.f);
    int prod = nb;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) prod *= __shfl_xor_sync(0xffffffffu, prod, o);
    if (c < n_dims) { g->shift[c] = shift; g->n_bins[c] = nb; }
    if (c == 0) {
        g->bin_width = bw;
        g->bins_per_event = prod;
        g->n_total_bins = prod * (n_rs - 1);
    }
    // within-bin ordering code: start from the bin width (binned) or the batch range (others)
    float ext = 0.f;
    if (c < n_dims) ext = bw;
    else if (c < n_all) { ext = mx - mn; if (!isfinite(ext)) ext = 0.f; }
    if (c < kMaxBinDims) { g->all_min[c] = mn; g->all_ext[c] = ext; }
    float span = c < n_all ? mx - mn : 0.f;
    if (!isfinite(span)) span = 0.f;
    const float own_span = span;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) span = fmaxf(span, __shfl_xor_sync(0xffffffffu, span, o));
    if (c < kMaxBinDims) g->range[c] = own_span;
    if (c == 0) g->curve_scale = span > 0.f ? 1.f / span : 0.f;
    // lane q holds the cell of coordinate q; the largest one (the first among equals) supplies the next bit
    float cell = c < kMaxBinDims ? fmaxf(ext, 0.f) : -1.f;
    int used = 0;
    for (int k = 0; k < kSubBits; k++) {
        const float top = warp_max_f32(cell);
        const int first = __ffs(__ballot_sync(0xffffffffu, cell == top)) - 1;
        if (c == first) {
            g->sub_seq[k] = c;
            g->sub_bit[k] = 15 - used++;
            cell *= 0.5f;
        }
    }
}

// One block: finishes the min/max reduction and derives the grid.
__device__ __forceinline__ void grid_from_partials(const float *partial, int n_partials, int n_dims, int n_all,
                  const int *__restrict__ row_splits, int n_rs, int n_bins_arg, int n_neigh,
                  int pre_normalized, GridParams *__restrict__ g)
{
    // min / max over the per-block partial results: thread t looks at coordinate t % 8 of every
    // (kGridSetupThreads / 8)-th partial; shuffles combine the lanes of a coordinate, shared memory the warps
    static_assert(kMaxBinDims == 8 && kGridSetupThreads % 32 == 0, "layout of the reduction");
    constexpr int kGridWarps = kGridSetupThreads / 32;
    __shared__ float s_mn[kGridWarps][8], s_mx[kGridWarps][8];
    {
        const int cc = threadIdx.x & 7;
        float a = INFINITY, b = -INFINITY;
        for (int p = threadIdx.x >> 3; p < n_partials; p += kGridSetupThreads / 8) {
            a = fminf(a, __ldcg(partial + ((size_t)p * 2 + 0) * kMaxBinDims + cc));  // perhaps written in this launch
            b = fmaxf(b, __ldcg(partial + ((size_t)p * 2 + 1) * kMaxBinDims + cc));
        }
#pragma unroll
        for (int o = 8; o < 32; o <<= 1) {
            a = fminf(a, __shfl_xor_sync(0xffffffffu, a, o));
            b = fmaxf(b, __shfl_xor_sync(0xffffffffu, b, o));
        }
        if ((threadIdx.x & 31) < 8) { s_mn[threadIdx.x >> 5][cc] = a; s_mx[threadIdx.x >> 5][cc] = b; }
    }
    __syncthreads();
    if (threadIdx.x >= 32) return;  // the rest is one warp's work
    float mn = 0.f, mx = 0.f;
    const int c = threadIdx.x;
    if (c < n_all) {
        mn = INFINITY; mx = -INFINITY;
#pragma unroll
        for (int w = 0; w < kGridWarps; w++) {
            mn = fminf(mn, s_mn[w][c]);
            mx = fmaxf(mx, s_mx[w][c]);
        }
    }
    grid_from_range(mn, mx, n_dims, n_all, row_splits, n_rs, n_bins_arg, n_neigh, pre_normalized, g);
}

// Position on a Hilbert curve: J. Skilling, "Programming the Hilbert curve", AIP Conf. Proc. 707 (2004) 381.
// D coordinates of B bits each; the curve visits neighbouring cells one after another, so that runs of
// consecutive hits are compact in all coordinates at once.
template <int D, int B>
__device__ __forceinline__ unsigned hilbert_code(unsigned (&x)[D])
{
#pragma unroll
    for (int b = B - 1; b > 0; b--) {
        const unsigned q = 1u << b, p = q - 1u;
#pragma unroll
        for (int i = 0; i < D; i++) {
            const unsigned t = (x[0] ^ x[i]) & p;
            const bool inv = (x[i] & q) != 0u;
            x[0] ^= inv ? p : t;
            if (i > 0) x[i] ^= inv ? 0u : t;
        }
    }
#pragma unroll
    for (int i = 1; i < D; i++) x[i] ^= x[i - 1];
    unsigned t = 0u;
#pragma unroll
    for (int b = B - 1; b > 0; b--)
        if (x[D - 1] & (1u << b)) t ^= (1u << b) - 1u;
#pragma unroll
    for (int i = 0; i < D; i++) x[i] ^= t;
    unsigned code = 0u;
#pragma unroll
    for (int b = B - 1; b >= 0; b--)
#pragma unroll
        for (int i = 0; i < D; i++) code = (code << 1) | ((x[i] >> b) & 1u);
    return code;
}

}  // namespace hgc
