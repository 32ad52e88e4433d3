// Blockwise interpolation of the banded kernel matrix: device functions shared by the products and
// gradients (km_nodes.cu) and by the CG operator (km_cg_nodes.cu).
//
// A row block sees whole column blocks of 128 points, and sorted inputs put the 128 points of a block
// into an interval that is short against what kappa varies over.  On a pair of such intervals kappa(x - y)
// is, to fp32 rounding, a polynomial of low degree in x and in y, so with P Chebyshev points xi of
// every block's interval and the Lagrange polynomials lambda on them
//     kappa(x_i - x_j) = sum_pq lambda_p(x_i) kappa(xi_p - xi_q) lambda_q(x_j) + O(eps),   P = 8 .. 64,
// and  K rhs = Lambda_1 ( K(xi, xi) ( Lambda_2^T rhs ) ):  (128 / P)^2 = 4 .. 256 times fewer kernel entries.
// The band is kept exactly (ranges aligned to blocks; others are left to the direct kernels), and a
// gradient is the same gradient of the small problem with left and right replaced by Lambda^T left and
// Lambda^T right.
//
// P follows from the inputs (nodes_needed): for f analytic in the Bernstein ellipse with parameter rho
// around an interval of half-length h, the interpolation error on P Chebyshev points is at most
// 4 M(rho) rho^-P / (rho - 1) (e.g. Trefethen, Approximation Theory and Approximation Practice, theorem 8.2)
// with M the largest |f| on the ellipse, whose points have imaginary parts up to b = h (rho - 1 / rho) / 2:
//     |exp(-z^2 / 2 l^2)| <= exp(b^2 / 2 l^2),   |cos(W z)| <= cosh(W b) <= exp(W b),
//     |exp(-2 sin^2(W z / 2) / l_p)| <= exp((cosh(W b) - 1) / l_p)
// and a factor (1 + b^2 / l^2) for the gradients' powers of tau.  The bound is evaluated on the device for
// the longest interval and every kernel of the call, and P taken so that it is below 1e-8 of
// kappa's maximum: less than the rounding of an fp32 value near 1 (6e-8), than the SFU's exp and cos
// (1e-7 and 5e-7) and than the fp16 pairs of the tensor-core kernels (3e-8).
#pragma once

#include "km_common.cuh"

namespace km {

constexpr int NODES_MAX = 64;           // P of a call is a multiple of 4 up to this
constexpr float NODES_EPS = 1e-8f;      // bound on the interpolation error, relative to kappa's maximum
constexpr float NODES_MIN_H = 1e-18f;   // half-length given to an interval of coincident points

// Interval of one block: points c + h t, |t| <= 1.
struct NodeBox {
    float c, h;
};

// Smallest P whose error bound is below NODES_EPS on an interval of half-length h; > NODES_MAX if
// none (or for non-finite arguments).  `lane` of 32 lanes tries one rho; the result is in every lane.
template <int KT>
__device__ __forceinline__ int nodes_needed(const float *theta, int64_t stride, float h, int lane) {
    const float rho = 1.1f * exp2f(0.17f * (float)lane);  // 1.1 .. 42
    const float b = 0.5f * h * (rho - 1.0f / rho);
    const float ell = theta[0];
    const float be = b * b / (ell * ell);
    float log_m = 0.5f * be + log1pf(be);
    if constexpr (KT == KM_KERNEL_SPECTRAL) log_m += 2.0f * KM_PI_F * fabsf(theta[stride]) * b;
    if constexpr (KT == KM_KERNEL_LOCALLY_PERIODIC)
        log_m += (coshf(2.0f * KM_PI_F * b / fabsf(theta[2 * stride])) - 1.0f) / fabsf(theta[stride]);
    const float need = (log_m + logf(4.0f / (rho - 1.0f)) - logf(NODES_EPS)) / logf(rho);
    float p = (need >= 1.0f && need < 1e6f) ? need : (need < 1.0f ? 1.0f : 1e6f);  // (NaN: no P)
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) p = fminf(p, __shfl_xor_sync(0xffffffffu, p, o));
    return (int)ceilf(p);
}

// Offset of node q of P from the centre of its interval.  Every kernel calls this one function, so
// that positions agree to the bit with those the Lagrange polynomials were formed for.
__device__ __forceinline__ float node_offset(float h, int q, int P) { return h * cospif((2.0f * q + 1.0f) / (2.0f * P)); }

// Barycentric weights of the rounded offsets `delta` (shared memory, P values), scaled by (2 / h)^P:
// thread q < P forms 1 / prod_r (delta_q - delta_r) in fp64.
__device__ __forceinline__ float node_weight(const float *delta, float h, int q, int P) {
    const double s = 2.0 / (double)h;
    double w = 1.0;
    for (int r = 0; r < P; r++)
        if (r != q) w *= ((double)delta[q] - (double)delta[r]) * s;
    return (float)(1.0 / w);
}

}  // namespace km
