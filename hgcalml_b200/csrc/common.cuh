// Shared host/device helpers of the hgcalml_b200 CUDA library (sm_100a only).
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>
#include <stddef.h>
#include <utility>

#include "../../include/hgcalml_b200.h"

namespace hgc {

constexpr int kWarp = 32;
constexpr size_t kAlign = 256;

inline size_t align_up(size_t x) { return (x + kAlign - 1) / kAlign * kAlign; }

// Bump allocator over the caller's workspace.  The first kAlign bytes hold the status word.
struct Carver {
    char *base;
    size_t used;
    explicit Carver(void *p) : base(static_cast<char *>(p)), used(kAlign) {}
    template <typename T> T *take(size_t n) {
        T *r = reinterpret_cast<T *>(base + used);
        used += align_up(n * sizeof(T));
        return r;
    }
    unsigned *status() const { return reinterpret_cast<unsigned *>(base); }
};

// The same arithmetic without a base pointer, for the *_workspace_bytes queries.
struct Sizer {
    size_t used = kAlign;
    template <typename T> void take(size_t n) { used += align_up(n * sizeof(T)); }
};

void set_cuda_error(cudaError_t e);

#define HGC_CUDA_TRY(expr)                                  \
    do {                                                    \
        cudaError_t hgc_e_ = (expr);                        \
        if (hgc_e_ != cudaSuccess) {                        \
            ::hgc::set_cuda_error(hgc_e_);                  \
            return HGC_ERR_CUDA;                            \
        }                                                   \
    } while (0)

// Multiprocessors of the calling thread's current device (asked for once per device); sizes persistent grids.
int sm_count();
// Launches a kernel that may start while the kernel before it in the stream is still finishing: its blocks become resident
// and wait in pdl_begin(), which takes about a microsecond off every step from one kernel to the next.  Every kernel
// launched this way begins with pdl_begin(), in all of its blocks, so that "the kernel before has completed" holds
// through any chain of them.
// Kernels that are short at every size are always launched so: the condensate path, keep_noise, the epilogues of dense
// layers, LocalDistance, the op-level sorts (4 x 200k hits condensed 460 -> 440 us, 100k 285 -> 266; two GravNet layers
// with message passing on 200k hits 2864 -> 2848).  So are the dense layers themselves, which gain by it at every size (us, launched
// so up to 65536 rows only / always: six layers of 64 x 64, 64 x 4 and 192 x 64 on 70k rows 149.5 / 140.2, 200k 363.6 / 362.1, 400k 705.0 /
// 698.4; 64 x 4 on 400k 26.7 / 23.9): their blocks share nothing through L1 with the kernel before.
// launch_overlapped is for the kernels whose length grows with the batch (search, orders, accumulation, backward ops): up to
// kOverlapHits hits.  Blocks that become resident early take room from the kernel that is still running and inherit its
// split between L1 and shared memory.  Search and accumulation, K = 16, F = 32, in us, not overlapped / overlapped: 20k hits
// 154/135, 40k 196/185, 64k 254/239, 70k 274/280, 100k 340/325, 150k 453/457, 200k 595/590, 300k 760/787, 400k 918/946;
// K = F = 64: 20k 195/184, 64k 455/449, 70k 480/487, 100k 625/623, 150k 882/893, 400k 1729/1776; a training step on 200k
// hits 3390/3496.  Between 65k and 200k hits neither is always better; the line lies where the gain ends.
template <typename... Params, typename... Args>
inline cudaError_t launch_pdl(void (*kernel)(Params...), dim3 grid, dim3 block, size_t smem, cudaStream_t stream, Args &&...args)
{
    cudaLaunchAttribute attr;
    attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr.val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = grid;
    cfg.blockDim = block;
    cfg.dynamicSmemBytes = smem;
    cfg.stream = stream;
    cfg.attrs = &attr;
    cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, kernel, std::forward<Args>(args)...);
}
constexpr int kOverlapHits = 65536;
template <typename... Params, typename... Args>
inline cudaError_t launch_overlapped(int n_hits, void (*kernel)(Params...), dim3 grid, dim3 block, size_t smem,
                                     cudaStream_t stream, Args &&...args)
{
    if (n_hits <= kOverlapHits) return launch_pdl(kernel, grid, block, smem, stream, std::forward<Args>(args)...);
    kernel<<<grid, block, smem, stream>>>(std::forward<Args>(args)...);
    return cudaGetLastError();
}
// Waits for the kernel before this one in the stream (a no-op in an ordinary launch) and lets the next one's blocks in.
__device__ __forceinline__ void pdl_begin()
{
    asm volatile("griddepcontrol.wait;" ::: "memory");
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
}

void count_launch();
#define HGC_LAUNCH_CHECK()                   \
    do {                                     \
        ::hgc::count_launch();               \
        HGC_CUDA_TRY(cudaGetLastError());    \
    } while (0)

inline int check_workspace(const void *ws, size_t have, size_t need) {
    if (need == 0) return HGC_OK;
    if (ws == nullptr || (reinterpret_cast<uintptr_t>(ws) % kAlign) != 0 || have < need)
        return HGC_ERR_WORKSPACE;
    return HGC_OK;
}

inline int div_up(long long a, long long b) { return (int)((a + b - 1) / b); }

__device__ __forceinline__ void flag_status(unsigned *status, unsigned bit) {
    // Idempotent bit set; a plain racy store of the same value would do, atomicOr keeps other bits.
    if (status) atomicOr(status, bit);
}

__device__ __forceinline__ int lane_id() { return threadIdx.x & 31; }

// ---- internal device-wide primitives (radix_sort.cu) ---------------------------------------

// Stable LSD radix sort of (key, value) pairs on keys in [0, 2^key_bits).  No atomics: per-warp
// digit counters combined by scans, so the result is deterministic.  values_in == nullptr means
// value i = i.  Sorted data ends up in keys_out / vals_out; keys_tmp / vals_tmp are ping-pong
// buffers of n ints each, block_hist has sort_hist_ints(n) ints.
size_t sort_hist_ints(int n);
int sort_pairs(const int *keys_in, const int *vals_in, int *keys_out, int *vals_out,
               int *keys_tmp, int *vals_tmp, int *block_hist, int n, int key_bits,
               cudaStream_t stream);

// Exclusive prefix sum of `len` ints in place; tile_sums needs scan_scratch_ints(len) ints.
size_t scan_scratch_ints(int len);
int exclusive_scan_ints(int *data, int len, int *tile_sums, cudaStream_t stream);

// bin_boundaries[b] = first position in the ascending key array whose key is >= b, for b in
// [0, n_bins]; keys >= n_bins (sentinels) sort last and are not counted.
int boundaries_from_sorted_keys(const int *sorted_keys, int n, int *bin_boundaries, int n_bins,
                                cudaStream_t stream);

inline int bits_for(long long max_value) {
    int b = 1;
    while ((1LL << b) <= max_value) b++;
    return b;
}

}  // namespace hgc
