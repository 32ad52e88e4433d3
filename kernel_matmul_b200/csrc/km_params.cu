// Kernel parameters from their raw (unconstrained) values: theta = lower_bound + softplus(raw).
//
// A kernel module has P raw tensors of the batch shape and hands the ops ONE (batch.., P) tensor in
// native order.  As tensor expressions that is P softplus, P additions, a stack and, with a cutoff
// that follows the lengthscale, a max, a stack of maxima, a max, two conversions and a product --
// two dozen launches per training step, most of the time of a step on a few thousand points.  Here
// it is one launch in each direction; the values are those of the tensor expressions (softplus with
// the linear tail from 20 on, one fp32 addition; the cutoff in fp64, rounded once).
#include "km_common.cuh"

namespace km {

struct RawParams {
    const float *raw[KM_MAX_PARAMS];
    float *grad[KM_MAX_PARAMS];
};

__device__ __forceinline__ float softplus(float x) { return x > 20.0f ? x : log1pf(expf(x)); }

// One CTA: a few values.
__global__ void __launch_bounds__(256) positive_params_kernel(int P, int64_t count, RawParams in, float lower_bound, float *out,
                                                               unsigned lengthscales, double cutoff_factor, float *cutoff) {
    __shared__ float warp_max[8];
    float largest = -INFINITY;
    bool nan = false;
    for (int64_t i = threadIdx.x; i < count * P; i += blockDim.x) {
        const int64_t e = i / P;
        const int q = (int)(i % P);
        const float v = lower_bound + softplus(in.raw[q][e]);
        out[i] = v;
        if ((lengthscales >> q) & 1u) {
            largest = fmaxf(largest, v);
            nan = nan || isnan(v);
        }
    }
    if (cutoff == nullptr) return;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) largest = fmaxf(largest, __shfl_xor_sync(0xffffffffu, largest, o));
    if ((threadIdx.x & 31) == 0) warp_max[threadIdx.x >> 5] = largest;
    const int any_nan = __syncthreads_or(nan ? 1 : 0);
    if (threadIdx.x == 0) {
        for (int w = 1; w < 8; w++) largest = fmaxf(largest, warp_max[w]);
        *cutoff = any_nan ? __int_as_float(0x7fc00000) : (float)((double)largest * cutoff_factor);
    }
}

__global__ void __launch_bounds__(256) positive_params_bwd_kernel(int P, int64_t count, RawParams io, const float *grad_out,
                                                                   int64_t grad_stride_e, int64_t grad_stride_q) {
    for (int64_t i = threadIdx.x; i < count * P; i += blockDim.x) {
        const int64_t e = i / P;
        const int q = (int)(i % P);
        const float x = io.raw[q][e], g = grad_out[e * grad_stride_e + q * grad_stride_q];
        const float z = expf(x);
        io.grad[q][e] = x > 20.0f ? g : g * z / (z + 1.0f);
    }
}

static int params_checks(const char *name, int32_t P, int64_t count, const float *const *raw) {
    KM_REQUIRE(P >= 1 && P <= KM_MAX_PARAMS && count >= 0 && count <= (1LL << 32), KM_ERR_INVALID_ARGUMENT, "%s: bad sizes", name);
    KM_REQUIRE(raw != nullptr, KM_ERR_INVALID_ARGUMENT, "%s: null pointer", name);
    for (int q = 0; q < P; q++) KM_REQUIRE(count == 0 || raw[q] != nullptr, KM_ERR_INVALID_ARGUMENT, "%s: null pointer", name);
    return KM_OK;
}

}  // namespace km

extern "C" int km_positive_params_f32(int32_t P, int64_t count, const float *const *raw, float lower_bound, float *params,
                                      uint32_t lengthscales, double cutoff_factor, float *cutoff, void *stream) {
    using namespace km;
    const int rc = params_checks("km_positive_params_f32", P, count, raw);
    if (rc != KM_OK) return rc;
    if (count == 0) return KM_OK;
    KM_REQUIRE(params != nullptr, KM_ERR_INVALID_ARGUMENT, "km_positive_params_f32: null pointer");
    RawParams in = {};
    for (int q = 0; q < P; q++) in.raw[q] = raw[q];
    positive_params_kernel<<<1, 256, 0, static_cast<cudaStream_t>(stream)>>>(P, count, in, lower_bound, params, lengthscales,
                                                                             cutoff_factor, cutoff);
    KM_CHECK_LAUNCH("km_positive_params_f32 launch");
    return KM_OK;
}

extern "C" int km_positive_params_bwd_f32(int32_t P, int64_t count, const float *const *raw, const float *grad_params,
                                          int64_t stride_batch, int64_t stride_param, float *const *grad_raw, void *stream) {
    using namespace km;
    const int rc = params_checks("km_positive_params_bwd_f32", P, count, raw);
    if (rc != KM_OK) return rc;
    if (count == 0) return KM_OK;
    KM_REQUIRE(grad_params != nullptr && grad_raw != nullptr, KM_ERR_INVALID_ARGUMENT, "km_positive_params_bwd_f32: null pointer");
    RawParams io = {};
    for (int q = 0; q < P; q++) {
        KM_REQUIRE(grad_raw[q] != nullptr, KM_ERR_INVALID_ARGUMENT, "km_positive_params_bwd_f32: null pointer");
        io.raw[q] = raw[q];
        io.grad[q] = grad_raw[q];
    }
    positive_params_bwd_kernel<<<1, 256, 0, static_cast<cudaStream_t>(stream)>>>(P, count, io, grad_params, stride_batch, stride_param);
    KM_CHECK_LAUNCH("km_positive_params_bwd_f32 launch");
    return KM_OK;
}
