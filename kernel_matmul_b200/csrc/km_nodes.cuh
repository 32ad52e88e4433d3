// Blockwise interpolation of the banded kernel matrix: device functions shared by the products and
// gradients (km_nodes.cu) and by the CG operator (km_cg_nodes.cu).
//
// A row block sees whole column blocks of 128 points, and sorted inputs put the 128 points of a block
// into an interval that is short against what kappa varies over.  On a pair of such intervals kappa(x - y)
// is, to fp32 rounding, a polynomial of low degree in x and in y, so with P Chebyshev points xi of
// every block's interval and the Lagrange polynomials lambda on them
//     kappa(x_i - x_j) = sum_pq lambda_p(x_i) kappa(xi_p - xi_q) lambda_q(x_j) + O(eps),   P = 8 .. 80,
// and  K rhs = Lambda_1 ( K(xi, xi) ( Lambda_2^T rhs ) ):  (128 / P)^2 = 2.5 .. 256 times fewer kernel entries.
// The band is kept exactly (ranges aligned to blocks; others are left to the direct kernels), and a
// gradient is the same gradient of the small problem with left and right replaced by Lambda^T left and
// Lambda^T right.
//
// Each block has an interval around its own centre whose half-length is one of four (the longest
// block's, and that divided by 1.15, 1.32 and 1.52); P follows from half-length and kernel.  Node offsets,
// weights and phase factors are then the same for all blocks of one half-length.
//
// P follows from the inputs (nodes_needed): for f analytic in the Bernstein ellipse with parameter rho
// around an interval of half-length h, the error of interpolation at P Chebyshev points (degree P - 1) is at most
// 4 M(rho) rho^-(P - 1) / (rho - 1) (e.g. Trefethen, Approximation Theory and Approximation Practice, theorem 8.2)
// with M the largest |f| on the ellipse, whose points have imaginary parts up to b = h (rho - 1 / rho) / 2:
//     |exp(-z^2 / 2 l^2)| <= exp(b^2 / 2 l^2),   |cos(W z)| <= cosh(W b) <= exp(W b),
//     |exp(-2 sin^2(W z / 2) / l_p)| <= exp((cosh(W b) - 1) / l_p)
// and a factor (1 + b^2 / l^2) for the gradients' powers of tau.  The device takes the smallest P with
// 4 M rho^-P / (rho - 1) below 3e-8 of kappa's maximum (half an ulp of an fp32 value near 1) for some rho, for the four
// half-lengths and every kernel of the call.  That is a rule and no bound -- it leaves out a power of rho, the second
// variable (a factor of 1 + Lebesgue's constant, 3 to 4) and the growth of the periodic factors of gradients --, so what
// it gives is measured: in fp64, over lengthscales of 0.5 - 3, frequencies up to 2, periods from 1.2 and blocks of 50 - 250
// points per unit, the largest error of an entry is 2.6e-8 of kappa's maximum (RBF), 1.5e-8 (spectral) and 6.5e-9
// (locally periodic), and of a gradient's factor 2.1e-7, 7.9e-8 and 1.2e-7 of its own maximum (at 6 to 18 nodes, for
// the lengthscale, the lengthscale and the period).  Rounding comes to it: the SFU's exp and cos (1e-7 and 5e-7), and
// fp32 Lagrange matrices.  Of whole products and gradients the errors stand beside the rules that choose this way
// (csrc_torch/km_host.h).
#pragma once

#include "km_common.cuh"

namespace km {

constexpr int NODES_MAX = 80;           // most nodes of a block; P is even
constexpr float NODES_EPS = 3e-8f;      // of kappa's maximum, in the rule for the number of nodes: half an ulp of 1
// The blocks of a call use intervals of one of NODES_LEVELS half-lengths: the longest block's, divided
// by powers of NODES_RATIO.  The longest of some hundred blocks of uniform points is 1.3 times the mean.
constexpr int NODES_LEVELS = 4;
constexpr float NODES_RATIO = 1.15f;
// Half-length given to an interval of coincident points: short enough for the square of a distance between
// its nodes to vanish, as that of the points does.
constexpr float NODES_MIN_H = 1e-25f;
// Operands that are not finite, or near overflow, at the nodes are left to the direct kernels: sums of
// Lagrange polynomials of either sign would turn an infinity into NaN.
constexpr float NODES_MAX_OPERAND = 1e30f;

// Smallest P for which the rule above stays below NODES_EPS on an interval of half-length h; > NODES_MAX if
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

// Node q of P on an interval of half-length h, as an offset from its centre.
__device__ __forceinline__ float node_offset(float h, int q, int P) { return h * cospif((2.0f * q + 1.0f) / (2.0f * P)); }

// Barycentric weight of node q, scaled by (2 / h)^P: 1 / prod_r (delta_q - delta_r) of the ROUNDED
// offsets, in fp64, so that the Lagrange polynomials are those of the very points kappa is taken at.
__device__ __forceinline__ float node_weight(const float *delta, float h, int q, int P) {
    const double s = 2.0 / (double)h, d = (double)delta[q];
    double w[2] = {1.0, 1.0};  // (P is even)
    for (int r = 0; r < P; r += 2) {
        if (r != q) w[0] *= (d - (double)delta[r]) * s;
        if (r + 1 != q) w[1] *= (d - (double)delta[r + 1]) * s;
    }
    return (float)(1.0 / (w[0] * w[1]));
}

}  // namespace km
