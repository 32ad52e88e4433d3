#pragma once

#include <ATen/cuda/CUDAEvent.h>

#include "km_host.h"

namespace kmh {

// The buffers of a solve on one GPU (kernel_matmul_b200.cg.CGSolver).
struct CgState {
    Tensor x, r, p, kp, bp, rs, ynorm, history, alphas, betas, send1, send2;
    int64_t n, k, blocks, seg_blocks, slots;
    double sigma2;
    float *row(const Tensor &t, int64_t i) const { return t.data_ptr<float>() + i * k; }
    float *rs_row(int64_t it) const { return row(rs, it & 1); }
};

class NodeOperator {
  public:
    // Looks at the band -- and, of a sum of spectral components, at points and parameters -- for a window of row
    // blocks of n points; `plan()` tells what came of it.
    NodeOperator(int64_t n, const std::optional<Tensor> &x, const std::optional<Tensor> &params, const Tensor &start, const Tensor &end,
                 int64_t row_block_begin, int64_t row_block_count);
    // int64 on the device: lo, hi, checksum, nodes per block (0: not this way), widest band in blocks
    Tensor plan() const { return plan_.slice(0, 0, 5); }
    // Copies points, parameters and band and lays the operator out from the copies, which is what all products use.
    // False, and nothing is kept, where the device has not that much memory left.
    bool build(int64_t lo, int64_t hi, int64_t nodes, int64_t max_blocks);
    // Whether any of them has another value than its copy by now, however it was written to (waits for the
    // device; not under stream capture).
    bool changed() const;
    // out = the window's rows of K v
    void matvec(const Tensor &v, const Tensor &out) const;

    // Called before products on the current stream: they come after the layout, which may have been made on
    // another, and its memory is not given away before they are done.
    void use() const;
    Tensor nodes(int64_t k) const;
    void compress(const Tensor &v, int64_t k, float *nodes) const;
    void update_p(const CgState &s, int64_t it, float *nodes) const;
    void product(int64_t k, const float *nodes, float *out, const float *p, double sigma2, float *block_partials) const;

  private:
    void *stream() const { return c10::cuda::getCurrentCUDAStream(start_.device().index()).stream(); }
    int64_t n_, R_, begin_, count_, P_ = 0, max_blocks_ = 0, blk0_ = 0, blk1_ = 0;
    km_view params_view(const Tensor &params) const;
    Tensor x_, params_, start_, end_;                      // the caller's
    Tensor own_x_, own_params_, own_start_, own_end_;      // contiguous copies
    Tensor centre_, plan_, lambda_, matrix_;
    mutable at::cuda::CUDAEvent laid_out_;
    std::optional<c10::cuda::CUDAStream> laid_out_on_;
    km_batch kb_{};
};

void cg_run(const CgState &s, const NodeOperator *nodes, RowsProduct *rows, int64_t first, int64_t count);

// z_c^T log(A) z_c for every column of a CG run, fp64 on the device
Tensor log_forms(const Tensor &alphas, const Tensor &betas, const Tensor &residual_norms, const Tensor &z_norm2, double converged);

}  // namespace kmh
