// Dense layers in one pass: y = act(x w + bias) in float32.
//
// Every product goes into its sum with one fused multiply-add, k ascending, and the bias is added to the rounded sum.  A float32
// GEMM of the library that does not split k gives the same bits.
#include "common.cuh"

namespace hgc {
namespace {

__device__ __forceinline__ void copy16(float *dst, const float *src, bool in)  // zeros where not `in`
{
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;"
                 :: "r"((unsigned)__cvta_generic_to_shared(dst)), "l"(src), "r"(in ? 16 : 0) : "memory");
}
__device__ __forceinline__ void copy4(float *dst, const float *src, bool in)
{
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;"
                 :: "r"((unsigned)__cvta_generic_to_shared(dst)), "l"(src), "r"(in ? 4 : 0) : "memory");
}
template <bool RELU>
__device__ __forceinline__ float finish(float v, const float *__restrict__ bias, int c)
{
    if (bias != nullptr) v = __fadd_rn(v, __ldg(bias + c));
    if (RELU) v = v <= 0.f ? 0.f : v;  // NaN stays NaN, -0 becomes 0
    return v;
}

constexpr int kThreads = 128;
constexpr int kDepth = 16;             // columns of x that are staged together
constexpr int kPitch = kDepth + 4;     // staged rows are this far apart
constexpr int kStages = 3;

// A block computes 16 TM rows x 8 TN columns, a thread TM rows x TN columns; x and w go through shared memory kDepth deep, the
// next two pieces on their way.  Shared memory hands a warp one float per lane and cycle, which is what bounds small tiles:
// 8 x 4 products from 12 floats per thread (256 threads) took 139 us for 200k x 192 x 64, 8 x 8 from 16 123 us (40 TFLOP/s); 16 x 8
// spills at three blocks per SM, and with all of w kept in shared memory two blocks fit: 160 us.
template <int TM, int TN, bool RELU>
__global__ void __launch_bounds__(kThreads, 4)
dense_kernel(const float *__restrict__ x, int K, const float *__restrict__ w, int n_out, const float *__restrict__ bias,
             float *__restrict__ y, int n_rows, bool vec_w, bool vec_out)
{
    pdl_begin();
    constexpr int kRows = 16 * TM, kCols = 8 * TN, V = TN < 4 ? TN : 4;  // V: columns of a thread that lie next to each other
    extern __shared__ __align__(16) float s_dyn[];
    float *__restrict__ s_x = s_dyn;                            // [kStages][kRows][kPitch]
    float *__restrict__ s_w = s_dyn + kStages * kRows * kPitch;  // [kStages][kDepth][kCols]
    const int t = threadIdx.x;
    const int c0 = blockIdx.y * kCols;
    const long long m0 = (long long)blockIdx.x * kRows;
    const int steps = (K + kDepth - 1) / kDepth;
    auto load = [&](int s) {
        if (s < steps) {
            float *__restrict__ dst = s_x + s % kStages * (kRows * kPitch);
#pragma unroll
            for (int i = t; i < kRows * (kDepth / 4); i += kThreads) {
                const int row = i / (kDepth / 4), k = i % (kDepth / 4) * 4;
                const bool in = m0 + row < n_rows && s * kDepth + k < K;
                copy16(dst + row * kPitch + k, x + (in ? (m0 + row) * K + s * kDepth + k : 0), in);
            }
            float *__restrict__ dst_w = s_w + s % kStages * (kDepth * kCols);
            if (vec_w) {
#pragma unroll
                for (int i = t * 4; i < kDepth * kCols; i += kThreads * 4) {
                    const int k = s * kDepth + i / kCols, c = c0 + i % kCols;
                    const bool in = k < K && c < n_out;
                    copy16(dst_w + i, w + (in ? (size_t)k * n_out + c : 0), in);
                }
            } else {
#pragma unroll 4
                for (int i = t; i < kDepth * kCols; i += kThreads) {
                    const int k = s * kDepth + i / kCols, c = c0 + i % kCols;
                    const bool in = k < K && c < n_out;
                    copy4(dst_w + i, w + (in ? (size_t)k * n_out + c : 0), in);
                }
            }
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
    // rows ty + 16 i, columns tx * V + {0 .. V - 1} + 8 V j
    const int ty = t >> 3, tx = t & 7;
    float acc[TM][TN];
#pragma unroll
    for (int i = 0; i < TM; i++)
#pragma unroll
        for (int c = 0; c < TN; c++) acc[i][c] = 0.f;
#pragma unroll
    for (int s = 0; s < kStages - 1; s++) load(s);
    for (int s = 0; s < steps; s++) {
        asm volatile("cp.async.wait_group %0;" :: "n"(kStages - 2) : "memory");
        __syncthreads();
        load(s + kStages - 1);
        const float *__restrict__ a = s_x + s % kStages * (kRows * kPitch) + ty * kPitch;
        const float *__restrict__ b = s_w + s % kStages * (kDepth * kCols) + tx * V;
#pragma unroll 1
        for (int k = 0; k < kDepth; k += 4) {
            float bx[4][TN];
#pragma unroll
            for (int j = 0; j < 4; j++)
#pragma unroll
                for (int c = 0; c < TN; c += V) {
                    const float *__restrict__ from = b + (k + j) * kCols + c * 8;
                    if constexpr (V == 4) {
                        const float4 q = *reinterpret_cast<const float4 *>(from);
                        bx[j][c] = q.x; bx[j][c + 1] = q.y; bx[j][c + 2] = q.z; bx[j][c + 3] = q.w;
                    } else {
                        const float2 q = *reinterpret_cast<const float2 *>(from);
                        bx[j][c] = q.x; bx[j][c + 1] = q.y;
                    }
                }
#pragma unroll
            for (int i = 0; i < TM; i++) {
                const float4 q = *reinterpret_cast<const float4 *>(a + 16 * i * kPitch + k);
                const float ax[4] = {q.x, q.y, q.z, q.w};
#pragma unroll
                for (int j = 0; j < 4; j++)
#pragma unroll
                    for (int c = 0; c < TN; c++) acc[i][c] = fmaf(ax[j], bx[j][c], acc[i][c]);
            }
        }
    }
#pragma unroll
    for (int i = 0; i < TM; i++) {
        const long long m = m0 + ty + 16 * i;
        if (m >= n_rows) continue;
#pragma unroll
        for (int j = 0; j < TN; j += V) {
            const int c = c0 + tx * V + j * 8;
            float r[V];
#pragma unroll
            for (int v = 0; v < V; v++) r[v] = c + v < n_out ? finish<RELU>(acc[i][j + v], bias, c + v) : 0.f;
            float *__restrict__ dst = y + m * n_out + c;
            if (V == 4 && vec_out) {
                if (c < n_out) *reinterpret_cast<float4 *>(dst) = make_float4(r[0], r[1], r[V > 2 ? 2 : 0], r[V > 3 ? 3 : 0]);
            } else {
#pragma unroll
                for (int v = 0; v < V; v++)
                    if (c + v < n_out) dst[v] = r[v];
            }
        }
    }
}

// Up to eight columns: a thread per row, whose floats go through shared memory 64 at a time.
constexpr int kNarrowDepth = 64;
template <int NC, bool RELU>
__global__ void __launch_bounds__(128)
dense_narrow_kernel(const float *__restrict__ x, int K, const float *__restrict__ w, int n_out, const float *__restrict__ bias,
                    float *__restrict__ y, int n_rows)
{
    pdl_begin();
    constexpr int kPitch = kNarrowDepth + 4;  // 16-byte reads of eight rows meet no bank twice
    __shared__ __align__(16) float s_x[128 * kPitch];
    __shared__ __align__(16) float s_w[kNarrowDepth][NC];
    const int t = threadIdx.x;
    const long long m0 = (long long)blockIdx.x * 128;
    float acc[NC];
#pragma unroll
    for (int c = 0; c < NC; c++) acc[c] = 0.f;
    for (int k0 = 0; k0 < K; k0 += kNarrowDepth) {
        const int depth = min(kNarrowDepth, K - k0), q = depth / 4;
        __syncthreads();
        for (int i = t; i < 128 * q; i += 128) {
            const int row = i / q, k = (i - row * q) * 4;
            const bool in = m0 + row < n_rows;
            copy16(s_x + row * kPitch + k, x + (in ? (m0 + row) * K + k0 + k : 0), in);
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
        for (int i = t; i < depth * NC; i += 128) {
            const int k = i / NC, c = i % NC;
            s_w[k][c] = c < n_out ? __ldg(w + (size_t)(k0 + k) * n_out + c) : 0.f;
        }
        asm volatile("cp.async.wait_group 0;" ::: "memory");
        __syncthreads();
        for (int k = 0; k < depth; k += 4) {
            const float4 v = *reinterpret_cast<const float4 *>(s_x + t * kPitch + k);
            const float a[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
            for (int j = 0; j < 4; j++)
#pragma unroll
                for (int c = 0; c < NC; c++) acc[c] = fmaf(a[j], s_w[k + j][c], acc[c]);
        }
    }
    if (m0 + t >= n_rows) return;
    float *__restrict__ dst = y + (m0 + t) * n_out;
#pragma unroll
    for (int c = 0; c < NC; c++)
        if (c < n_out) dst[c] = finish<RELU>(acc[c], bias, c);
}

template <int TM, int TN, bool RELU>
int launch_rows(const float *x, int K, const float *w, int n_out, const float *bias, float *y, int n_rows, cudaStream_t stream)
{
    const auto kernel = dense_kernel<TM, TN, RELU>;
    constexpr size_t smem = sizeof(float) * kStages * (16 * TM * kPitch + kDepth * 8 * TN);
    static_assert(smem <= 48 * 1024, "more needs cudaFuncSetAttribute");
    const bool vec_out = n_out % 4 == 0 && (reinterpret_cast<uintptr_t>(y) & 15u) == 0;
    HGC_CUDA_TRY(launch_pdl(kernel, dim3(div_up(n_rows, 16 * TM), div_up(n_out, 8 * TN)), kThreads, smem, stream, x, K, w, n_out, bias, y, n_rows,
                            n_out % 4 == 0 && (reinterpret_cast<uintptr_t>(w) & 15u) == 0, vec_out));
    HGC_LAUNCH_CHECK();
    return HGC_OK;
}

template <int TN, bool RELU>
int launch_dense(const float *x, int K, const float *w, int n_out, const float *bias, float *y, int n_rows, cudaStream_t stream)
{
    // Blocks of 128 rows keep every SM busy from about 50k rows on; below that blocks of 32 are shorter chains on more SMs.
    // 64 x 64, us with 128 / 32 rows: 4000 rows 10.4 / 4.9, 20k 13.1 / 9.6, 40k 19.9 / 16.2, 60k 20.5 / 22.5, 200k 54.8 / 68.2.
    if (n_rows >= 49152) return launch_rows<8, TN, RELU>(x, K, w, n_out, bias, y, n_rows, stream);
    return launch_rows<2, TN, RELU>(x, K, w, n_out, bias, y, n_rows, stream);
}

template <bool RELU>
int run_dense(const float *x, int K, const float *w, int n_out, const float *bias, float *y, int n_rows, cudaStream_t stream)
{
    if (n_out <= 8) {
        HGC_CUDA_TRY(launch_pdl(n_out <= 4 ? dense_narrow_kernel<4, RELU> : dense_narrow_kernel<8, RELU>, div_up(n_rows, 128), 128, 0, stream,
                                x, K, w, n_out, bias, y, n_rows));
        HGC_LAUNCH_CHECK();
        return HGC_OK;
    }
    if (n_out <= 16) return launch_dense<2, RELU>(x, K, w, n_out, bias, y, n_rows, stream);
    if (n_out <= 32) return launch_dense<4, RELU>(x, K, w, n_out, bias, y, n_rows, stream);
    return launch_dense<8, RELU>(x, K, w, n_out, bias, y, n_rows, stream);
}

}  // namespace
}  // namespace hgc

using namespace hgc;

extern "C" int hgc_dense(const float *d_x, const float *d_w, const float *d_bias, float *d_y, int n, int n_in, int n_out, int relu,
                         hgc_stream_t stream_)
{
    cudaStream_t stream = static_cast<cudaStream_t>(stream_);
    if (n < 0 || n_in < 1 || n_out < 0) return HGC_ERR_INVALID_ARGUMENT;
    if (n == 0 || n_out == 0) return HGC_OK;
    if (!d_x || !d_w || !d_y) return HGC_ERR_INVALID_ARGUMENT;
    // rows of whole 16-byte vectors, which is how they are staged
    if (n_in % 4 != 0 || (reinterpret_cast<uintptr_t>(d_x) & 15u) != 0) return HGC_ERR_UNSUPPORTED;
    return relu ? run_dense<true>(d_x, n_in, d_w, n_out, d_bias, d_y, n, stream)
                : run_dense<false>(d_x, n_in, d_w, n_out, d_bias, d_y, n, stream);
}
