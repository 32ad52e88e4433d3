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

// Their sums for columns c0 .. c0 + KC - 1, by all 128 threads of a CTA, in to[0 .. KC).  The order does not
// depend on how segments are dealt out to ranks: lane l of a warp adds segments l, l + 32, .. (segments past
// the last are zero), then a fixed tree over the lanes.  (Added one after the other by one thread they
// took 5 us of every update: 64 loads, none of which waits for the one before.)
template <int KC>
__device__ __forceinline__ void cg_totals(const CgTotals &g, int64_t k, int c0, double (&to)[KC]) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int segments = g.ranks * g.slots;
    for (int c = warp; c < KC && c0 + c < k; c += 4) {
        double t = 0.0;
        for (int s = lane; s < segments; s += 32) {
            const int rank = g.ranks == 1 ? 0 : s / g.slots, slot = g.ranks == 1 ? s : s - rank * g.slots;
            t += reinterpret_cast<const double *>(g.base + rank * g.rank_stride)[slot * k + c0 + c];
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) t += __shfl_xor_sync(0xffffffffu, t, o);
        if (lane == 0) to[c] = t;
    }
    __syncthreads();
}

}  // namespace km
