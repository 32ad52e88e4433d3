// Host side of the ops, shared by the bindings (km_torch.cpp), the autograd functions
// (km_autograd.cpp) and the CG loop (km_cg_host.cpp): argument checks, broadcasting, choice of the
// kernel, allocation, launch through the C ABI of libkm_b200.so.  No arithmetic happens here.
//
// All of this used to be Python (broadcast_shapes, expand, one ctypes structure per argument, a
// device copy and an event per tensor-core launch): 70 - 150 us of host time per op call where the
// smallest kernels take 5 us.  Here a call costs a few microseconds.
#pragma once

#include <ATen/ATen.h>
#include <c10/cuda/CUDAGuard.h>
#include <c10/cuda/CUDAStream.h>
#include <c10/util/SmallVector.h>

#include <stdexcept>
#include <string>

#include "../../include/km_b200.h"

namespace kmh {

using at::Tensor;
using Shape = c10::SmallVector<int64_t, 6>;

// An entry point of libkm_b200 returned a non-zero status (kernel_matmul_b200._lib.KmError in Python).
struct StatusError : std::runtime_error {
    using std::runtime_error::runtime_error;
};
// A tensor-core launch gave up at a hand-off wait (kernel_matmul_b200.ops.KernelGaveUpError).
struct GaveUpError : std::runtime_error {
    using std::runtime_error::runtime_error;
};
// Bad value of an argument (ValueError).
struct ArgumentError : std::runtime_error {
    using std::runtime_error::runtime_error;
};

enum Path : int64_t { PATH_AUTO = 0, PATH_FMA = 1, PATH_TC = 2, PATH_NODES = 3 };

// rhs widths from which a product, column counts from which a gradient runs on the tensor cores
// (tcgen05) when it has at least TENSOR_CORE_MIN_ITEMS (batch, row block) items: the cost of those
// kernels hardly depends on the width, and their pre-passes are two or three small launches.
constexpr int64_t TENSOR_CORE_MIN_K = 9, GRAD_TENSOR_CORE_MIN_K = 8, TENSOR_CORE_MIN_ITEMS = 256;

// The automatic path tries blockwise interpolation (km_matmul_nodes_f32) only where the tensor-core kernels
// run otherwise, and from this many (batch, row block) items: its four small passes take about 10 us more
// than they save below.  Against 64 bits products of random operands have relative errors (2-norm) of 2.1e-7 - 3.2e-7
// by interpolation, 8.9e-7 - 1.4e-6 on the tensor cores and 2.4e-7 - 1.0e-6 on the FMA pipe, which holds small
// entries to 1e-6 of themselves (one-hot columns, entries of 1e-4 - 1e-3 of the largest, worst relative error: RBF 3e-6,
// 3e-4 and 1e-6, locally periodic with a lengthscale of 0.6 3e-5, 2e-4 and 2e-6): what ran on the FMA pipe stays there.
// Gradients of random operands are off by 1e-11 - 2.6e-10 of the sum of their terms' magnitudes, 1.6e-10 - 1e-9 on the tensor
// cores; of single entries, constant and smooth operands by up to 4e-7, 6e-7 there (an RBF lengthscale's by up to 1.2e-7
// against 1.0e-7).
//
// Bands of 6 blocks and more gain from 512 items on; gradients of up to 16 columns gain nothing on 6 blocks there (factor
// 0.9 - 1.05 of the direct kernels' time; products 0.7 - 0.8), bands of 3 blocks lose up to 1.1 on products of up to
// four kernels and up to 1.6 on such gradients, and gain from 2048 items on.  A call that the device declines (bands not
// aligned to blocks, intervals too long) takes 1.03 - 1.25 times its time, a gradient of 9 columns on 512 items 1.4.
constexpr int64_t NODES_MIN_ITEMS = 512;
// Row blocks of a kernel from which it does: the plan takes 0.25 us per kernel, in one CTA, and the last column blocks of a
// band are as dear as the first.  512 and 2048 kernels on one block each took 150 and 490 us, directly 27 and 51;
// 256 on three blocks 111 and 47, 64 on eight blocks 70 and 44; 32 on 32 blocks 0.8 - 0.9 of the direct time at a
// band of 6 blocks.
constexpr int64_t NODES_MIN_ROW_BLOCKS = 32;
// With a band, both sides share an interval: where one has this many times the other's points, the blocks
// of the sparser may be too long for it (5003 test points against 50 021 at 100 per unit: 100 nodes and more) and the
// call would pay 25 us for finding out.  Not measured over densities and lengthscales: smooth kernels on dense points,
// which a longer interval would do for, are evaluated directly too.
constexpr int64_t NODES_MAX_RATIO = 8;
// Without a cutoff: kernel entries from which it does (the points have to be put in order first).
constexpr int64_t NODES_MIN_ENTRIES = 1LL << 27;

void check_f32(const Tensor &x);
void check_i32(const Tensor &x);
int num_params(int64_t kernel_type);
inline void raise_on(int rc) {
    if (rc != KM_OK) throw StatusError("[km status " + std::to_string(rc) + "] " + km_last_error());
}
// Raises GaveUpError if a tensor-core launch on `device` has reported a give-up.
void poll_gave_up(int device);

// One op call: the broadcast batch shape and the arguments as views of the C ABI.
struct Problem {
    int kid;
    int device;
    int64_t m, n, row_blocks;
    Shape batch;
    km_batch kb{};
    km_view x1, x2, params, start, end;
    c10::SmallVector<Tensor, 4> keep;  // copies made for more batch dims than the ABI carries

    Problem(int64_t kernel_type, const Tensor &x1, const Tensor &x2, const Tensor &params, const Tensor &start, const Tensor &end,
            std::initializer_list<std::pair<const Tensor *, int>> extra);
    // `t` with its last `nonbatch` dims, broadcast over the batch
    km_view view(const Tensor &t, int nonbatch);
    Tensor empty(std::initializer_list<int64_t> tail, const Tensor &like) const;
    int64_t items() const;
    // Presumably every row block sees all columns: the ranges come from ranges.make_ranges without a
    // cutoff, which lays them out as the two halves of one storage, end first.  (A hint: the values are
    // looked at on the device.)
    bool one_range() const { return all_columns_; }
    // `k` columns, of an op that takes the tensor cores from `min_k` columns on
    bool try_nodes(int64_t path, int64_t k, int64_t min_k) const {
        if (path == PATH_NODES) return true;
        if (path != PATH_AUTO || k < min_k || items() < TENSOR_CORE_MIN_ITEMS || row_blocks < NODES_MIN_ROW_BLOCKS) return false;
        if (one_range()) return m * n * (items() / row_blocks) >= NODES_MIN_ENTRIES;
        return items() >= NODES_MIN_ITEMS && std::max(m, n) < NODES_MAX_RATIO * std::min(m, n);
    }
    void *stream() const { return c10::cuda::getCurrentCUDAStream(device).stream(); }

  private:
    bool flat_ = false, all_columns_ = false;
};

Tensor workspace(const Tensor &like, size_t bytes);

// The ops (signatures of the reference's native modules).  `tc`: set to whether the tensor cores ran.
Tensor matmul(int64_t kernel_type, const Tensor &x1, const Tensor &x2, const Tensor &rhs, const Tensor &params, const Tensor &start,
              const Tensor &end, int64_t path, bool *tc = nullptr);
// gradient of sum_c left[:, c]^T K right[:, c] with respect to params
Tensor bilinear(int64_t kernel_type, const Tensor &x1, const Tensor &x2, const Tensor &left, const Tensor &right,
                const Tensor &params, const Tensor &start, const Tensor &end, int64_t path, bool *tc = nullptr);
Tensor dense(int64_t kernel_type, const Tensor &x1, const Tensor &x2, const Tensor &params, const Tensor &start, const Tensor &end);
Tensor dense_bwd(int64_t kernel_type, const Tensor &x1, const Tensor &x2, const Tensor &params, const Tensor &start,
                 const Tensor &end, const Tensor &out_grad);
// `distances`: where to put the distances of the lookups, from which their gradient needs no points (left
// undefined where the device has no memory for them)
Tensor index(int64_t kernel_type, const Tensor &x1, const Tensor &x2, const Tensor &params, const Tensor &start, const Tensor &end,
             const std::vector<Tensor> &batch_indices, const Tensor &row, const Tensor &col, Tensor *distances = nullptr);
Tensor index_bwd(int64_t kernel_type, const Tensor &x1, const Tensor &x2, const Tensor &params, const Tensor &start,
                 const Tensor &end, const std::vector<Tensor> &batch_indices, const Tensor &row, const Tensor &col,
                 const Tensor &out_grad, const Tensor *distances = nullptr);

// matmul for a window of row blocks, optionally summed over the batch, with everything but the launch
// done once: for loops that call the same product on the same buffers (whose contents change) many
// times, as a CG solve does.
class RowsProduct {
  public:
    RowsProduct(int64_t kernel_type, const Tensor &x1, const Tensor &x2, const Tensor &rhs, const Tensor &params, const Tensor &start,
                const Tensor &end, int64_t row_block_begin, int64_t row_block_count, bool sum_batches,
                const std::optional<Tensor> &out, int64_t path, const std::optional<Tensor> &phases);
    void run();  // on the current stream, with scratch of its own
    const Tensor &out() const { return out_; }
    bool tensor_cores() const { return tc_; }

  private:
    void set_views();
    Problem p_;
    Tensor out_, phases_;
    std::vector<Tensor> keep_;
    km_view rhs_, vout_;
    int64_t k_, begin_, count_;
    bool sum_, tc_;
};

// The differentiable forms (gradient for params only), km_autograd.cpp.
Tensor matmul_ad(int64_t kernel_type, const Tensor &x1, const Tensor &x2, const Tensor &rhs, const Tensor &params,
                 const Tensor &start, const Tensor &end);
Tensor dense_ad(int64_t kernel_type, const Tensor &x1, const Tensor &x2, const Tensor &params, const Tensor &start, const Tensor &end);
Tensor index_ad(int64_t kernel_type, const Tensor &x1, const Tensor &x2, const Tensor &params, const Tensor &start,
                const Tensor &end, const std::vector<Tensor> &batch_indices, const Tensor &row, const Tensor &col);
// (batch.., P) parameters lower_bound + softplus(raw[q]) and, with a cutoff_factor, the (1,) tensor
// cutoff_factor * the largest value among the parameters whose bit is set in `lengthscales`
std::pair<Tensor, Tensor> positive_params(const std::vector<Tensor> &raw, double lower_bound, int64_t lengthscales,
                                          std::optional<double> cutoff_factor);

}  // namespace kmh
