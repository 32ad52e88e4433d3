// Shared by the vector kernels of the CG solve (km_cg.cu) and its operator by blockwise interpolation
// (km_cg_nodes.cu): rows of (n, k) vectors, and inner products that do not depend on how rows are
// dealt out to GPUs.
#pragma once

#include "km_common.cuh"

namespace km {

constexpr int CG_THREADS = 128;  // = rows of a row block

// Adds `v[c]`, c < KC, over the 128 threads of the CTA in a fixed order; the totals arrive in
// thread c (c < KC) of warp 0 as the return value.
template <int KC>
__device__ __forceinline__ float cg_block_reduce(float (&v)[KC], float (*warp_part)[32]) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
    for (int c = 0; c < KC; c++) {
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) v[c] += __shfl_xor_sync(0xffffffffu, v[c], o);
    }
    if (lane == 0) {
#pragma unroll
        for (int c = 0; c < KC; c++) warp_part[warp][c] = v[c];
    }
    __syncthreads();
    float total = 0.0f;
    if (warp == 0 && lane < KC) total = (warp_part[0][lane] + warp_part[1][lane]) + (warp_part[2][lane] + warp_part[3][lane]);
    __syncthreads();
    return total;
}

// k columns of one row, starting at column c0: 16-byte accesses when `vec`.
template <int KC>
__device__ __forceinline__ void cg_load_row(const float *row, int c0, int k, bool vec, float (&v)[KC]) {
    if (KC >= 4 && vec && c0 + KC <= k) {
#pragma unroll
        for (int c = 0; c < KC; c += 4) {
            const float4 t = *reinterpret_cast<const float4 *>(row + c0 + c);
            v[c] = t.x, v[c + 1] = t.y, v[c + 2] = t.z, v[c + 3] = t.w;
        }
    } else {
#pragma unroll
        for (int c = 0; c < KC; c++) v[c] = c0 + c < k ? row[c0 + c] : 0.0f;
    }
}
template <int KC>
__device__ __forceinline__ void cg_store_row(float *row, int c0, int k, bool vec, const float (&v)[KC]) {
    if (KC >= 4 && vec && c0 + KC <= k) {
#pragma unroll
        for (int c = 0; c < KC; c += 4) *reinterpret_cast<float4 *>(row + c0 + c) = make_float4(v[c], v[c + 1], v[c + 2], v[c + 3]);
    } else {
#pragma unroll
        for (int c = 0; c < KC; c++)
            if (c0 + c < k) row[c0 + c] = v[c];
    }
}

// The gathered segment sums of an inner product: base[rank * rank_stride_bytes + slot * k + c].
struct CgTotals {
    const unsigned char *base;
    int64_t rank_stride;  // bytes
    int ranks, slots;
};

// Their sum, in slot order.
__device__ __forceinline__ double cg_total(const CgTotals &g, int64_t k, int c) {
    double t = 0.0;
    for (int rk = 0; rk < g.ranks; rk++) {
        const double *seg = reinterpret_cast<const double *>(g.base + rk * g.rank_stride);
        for (int s = 0; s < g.slots; s++) t += seg[s * k + c];
    }
    return t;
}

}  // namespace km
