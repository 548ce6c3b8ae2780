// Condensates as the kernels hold them, shared by the op-level and the wrapper-level entry.
#pragma once
#include "common.cuh"

namespace hgc {

struct CondList {        // per event e, entries [row_splits_h[e], row_splits_h[e] + count[e])
    float *centre;       // [n_h][dims]
    float *radius_sq;    // [n_h]
    int *subset_pos;     // [n_h]  position in the *_h arrays
    int *lonely;         // [n_h]  1: masked hit that only claims itself
    int *count;          // [num_rows]
};

// A condensate is held as NR float4: its coordinates and, in the last slot, its squared radius (-1
// for a masked condensate, which covers nothing but itself): NR = 1 up to 3 dimensions, 2 up to 7,
// 3 for 8.
template <int NR> struct Rec { float v[NR * 4]; };
template <int NR> __host__ __device__ constexpr int rec_dims() { return NR == 3 ? 8 : NR * 4 - 1; }
template <int NR> __host__ __device__ constexpr int rec_r2_slot() { return NR == 3 ? 8 : NR * 4 - 1; }
inline int rec_size(int dims) { return dims <= 3 ? 1 : dims <= 7 ? 2 : 3; }

template <int NR>
__device__ __forceinline__ Rec<NR> load_rec(const float4 *p)
{
    Rec<NR> r;
#pragma unroll
    for (int u = 0; u < NR; u++) {
        const float4 q = p[u];
        r.v[4 * u] = q.x; r.v[4 * u + 1] = q.y; r.v[4 * u + 2] = q.z; r.v[4 * u + 3] = q.w;
    }
    return r;
}
template <int NR>
__device__ __forceinline__ void store_rec(float4 *p, const Rec<NR> &r)
{
#pragma unroll
    for (int u = 0; u < NR; u++) p[u] = make_float4(r.v[4 * u], r.v[4 * u + 1], r.v[4 * u + 2], r.v[4 * u + 3]);
}

// Squared distance over the first `dims` slots: subtract, multiply, add, each rounded on its own, in
// coordinate order (the reference's loop, binned_assign_to_condensates_kernel.cc:88-91,103-106).
template <int NR>
__device__ __forceinline__ float rec_distsq(const Rec<NR> &c, const Rec<NR> &x, int dims)
{
    float s = 0.f;
#pragma unroll
    for (int d = 0; d < rec_dims<NR>(); d++)
        if (d < dims) {
            const float t = __fsub_rn(c.v[d], x.v[d]);
            s = __fadd_rn(s, __fmul_rn(t, t));
        }
    return s;
}

// A float's order as an unsigned integer.
__device__ __forceinline__ unsigned ordered_bits(float f)
{
    const unsigned b = __float_as_uint(f);
    return (b & 0x80000000u) ? ~b : (b | 0x80000000u);
}

// Sort key of a high-beta hit: 0 for hits that are taken in position order, else 1 + descending beta.
__device__ __forceinline__ unsigned priority_key(float beta, bool flagged)
{
    if (flagged) return 0u;
    const unsigned desc = ~ordered_bits(beta);
    return desc == 0xffffffffu ? desc : desc + 1u;
}

// The claim pass over windows of the priority order (condensates.cu).  With use_grid given (device memory) it does
// nothing unless *use_grid is 0.
size_t claim_stage_ints(int num_rows);
int launch_claim_windows(int dims, const float *ccoords_h, const float *dist_h, const int *mask_h,
                         const int *original_indices_h, const int *row_splits_h, const int *order, int *status_h,
                         int *alpha_indices, int *stage, const CondList &cl, int num_rows, const int *use_grid,
                         cudaStream_t stream);

}  // namespace hgc
