// The CG solve's operator by blockwise interpolation, and whole runs of iterations without the
// interpreter: an iteration on a few thousand points is five kernels of 2 us, and their launches from
// Python took 350 us.
#include "km_cg_host.h"

#include <c10/cuda/CUDAGraphsC10Utils.h>

namespace kmh {

NodeOperator::NodeOperator(int64_t n, const std::optional<Tensor> &x, const std::optional<Tensor> &params, const Tensor &start,
                           const Tensor &end, int64_t row_block_begin, int64_t row_block_count)
    : n_(n), begin_(row_block_begin), count_(row_block_count) {
    check_i32(start), check_i32(end);
    R_ = (n_ + KM_BLOCK_SIZE - 1) / KM_BLOCK_SIZE;
    TORCH_CHECK(start.numel() >= R_ && end.numel() >= R_, "start / end must have ", R_, " entries");
    TORCH_CHECK(start.dim() == 1 && end.dim() == 1, "start and end must have one dimension");
    start_ = start, end_ = end;
    const c10::cuda::CUDAGuard guard(start_.device());
    const auto opt = start_.options().requires_grad(false);
    plan_ = at::empty({KM_NODE_PLAN_BYTES / 8}, opt.dtype(at::kLong));
    km_view params_now{};
    if (x.has_value()) {
        check_f32(*x), check_f32(*params);
        x_ = *x, params_ = *params;
        TORCH_CHECK(x_.dim() == 1 && x_.size(0) == n_ && params_.dim() >= 1 && params_.size(-1) == num_params(KM_KERNEL_SPECTRAL) &&
                        params_.dim() - 1 <= KM_MAX_BATCH_DIMS,
                    "x must be (n,) and params (.., 3)");
        kb_.ndim = (int)params_.dim() - 1;
        for (int d = 0; d < kb_.ndim; d++) kb_.size[d] = params_.size(d);
        params_now = params_view(params_);
        centre_ = at::empty({std::max<int64_t>(R_, 1)}, opt.dtype(at::kFloat));
    }
    const Tensor s = start_.contiguous(), e = end_.contiguous();
    raise_on(km_node_operator_plan_f32(&kb_, n_, x ? x_.const_data_ptr<float>() : nullptr, x ? x_.stride(0) : 0, x ? &params_now : nullptr,
                                       s.const_data_ptr<int32_t>(), e.const_data_ptr<int32_t>(), begin_, count_,
                                       x ? centre_.data_ptr<float>() : nullptr, plan_.data_ptr(), stream()));
}

km_view NodeOperator::params_view(const Tensor &params) const {
    km_view v{};
    v.data = params.data_ptr();
    for (int d = 0; d < kb_.ndim; d++) v.batch_stride[d] = params.stride(d);
    v.stride[0] = params.stride(kb_.ndim);
    return v;
}

bool NodeOperator::build(int64_t lo, int64_t hi, int64_t nodes, int64_t max_blocks) {
    const c10::cuda::CUDAGuard guard(x_.device());
    const auto opt = x_.options().requires_grad(false);
    const auto copy = [](const Tensor &t) { return t.detach().clone(at::MemoryFormat::Contiguous); };
    P_ = nodes, max_blocks_ = max_blocks;
    blk0_ = std::max<int64_t>(0, lo) / KM_BLOCK_SIZE, blk1_ = (std::min(hi, n_) + KM_BLOCK_SIZE - 1) / KM_BLOCK_SIZE;
    blk0_ = std::min(blk0_, blk1_);
    try {
        lambda_ = at::empty({R_ * P_ * KM_BLOCK_SIZE}, opt);
        matrix_ = at::empty({std::max<int64_t>(1, count_ * max_blocks * P_ * P_)}, opt);
        own_x_ = copy(x_), own_params_ = copy(params_), own_start_ = copy(start_), own_end_ = copy(end_);
    } catch (const c10::OutOfMemoryError &) {
        lambda_ = matrix_ = own_x_ = own_params_ = own_start_ = own_end_ = Tensor();
        return false;
    }
    const km_view own_params = params_view(own_params_);
    raise_on(km_node_operator_build_f32(&kb_, n_, own_x_.const_data_ptr<float>(), 1, &own_params, own_start_.const_data_ptr<int32_t>(),
                                        own_end_.const_data_ptr<int32_t>(), begin_, count_, centre_.const_data_ptr<float>(),
                                        plan_.data_ptr(), P_, max_blocks_, lambda_.data_ptr<float>(), matrix_.data_ptr<float>(), stream()));
    laid_out_on_ = c10::cuda::getCurrentCUDAStream(x_.device().index());
    laid_out_.record(*laid_out_on_);
    return true;
}

void NodeOperator::use() const {
    TORCH_CHECK(laid_out_on_.has_value(), "the operator has not been laid out");
    const auto now = c10::cuda::getCurrentCUDAStream(own_x_.device().index());
    // (a capture waits for nothing outside it, and begins behind a synchronisation)
    if (now == *laid_out_on_ || c10::cuda::currentStreamCaptureStatusMayInitCtx() != c10::cuda::CaptureStatus::None) return;
    laid_out_.block(now);
    for (const Tensor *t : {&lambda_, &matrix_, &own_start_, &own_end_, &own_x_, &own_params_}) t->record_stream(now);
}

bool NodeOperator::changed() const {
    // (a tensor may have been given other memory)
    if (x_.sizes() != own_x_.sizes() || params_.sizes() != own_params_.sizes() || start_.sizes() != own_start_.sizes() ||
        end_.sizes() != own_end_.sizes())
        return true;
    const c10::cuda::CUDAGuard guard(own_x_.device());
    use();
    const Tensor flag = at::empty({1}, own_start_.options());
    const km_view params_now = params_view(params_);
    km_view s{}, e{};
    s.data = start_.data_ptr(), s.stride[0] = start_.stride(0), e.data = end_.data_ptr(), e.stride[0] = end_.stride(0);
    raise_on(km_node_operator_changed(&kb_, n_, x_.const_data_ptr<float>(), x_.stride(0), &params_now, &s, &e,
                                      own_x_.const_data_ptr<float>(), own_params_.const_data_ptr<float>(),
                                      own_start_.const_data_ptr<int32_t>(), own_end_.const_data_ptr<int32_t>(), flag.data_ptr<int32_t>(),
                                      stream()));
    return flag.item<int32_t>() != 0;
}

// Scratch of a product: one per call or run, on its stream, so that an operator may be applied on several
// streams and threads at a time.
Tensor NodeOperator::nodes(int64_t k) const {
    return at::empty({R_ * P_ * ((k + 3) / 4 * 4)}, x_.options().requires_grad(false));
}

void NodeOperator::compress(const Tensor &v, int64_t k, float *nodes) const {
    raise_on(km_node_compress_f32(k, n_, P_, lambda_.const_data_ptr<float>(), v.const_data_ptr<float>(), nodes, blk0_, blk1_, stream()));
}

void NodeOperator::update_p(const CgState &s, int64_t it, float *nodes) const {
    const int64_t k = s.k;
    raise_on(km_node_update_p_f32(k, n_, P_, lambda_.const_data_ptr<float>(), s.p.data_ptr<float>(), s.r.const_data_ptr<float>(), nodes, 0, R_,
                                  s.send2.data_ptr(), s.send2.numel(), 1, (int32_t)s.slots, s.rs_row(it), s.rs_row(it + 1),
                                  s.ynorm.const_data_ptr<float>(), s.row(s.history, it + 1), s.row(s.betas, it), stream()));
}

void NodeOperator::product(int64_t k, const float *nodes, float *out, const float *p, double sigma2, float *block_partials) const {
    raise_on(km_node_product_f32(k, n_, P_, max_blocks_, own_start_.const_data_ptr<int32_t>(), own_end_.const_data_ptr<int32_t>(),
                                 lambda_.const_data_ptr<float>(), matrix_.const_data_ptr<float>(), nodes, begin_, count_, out, p, (float)sigma2,
                                 block_partials, stream()));
}

void NodeOperator::matvec(const Tensor &v, const Tensor &out) const {
    check_f32(v), check_f32(out);
    TORCH_CHECK(v.dim() == 2 && v.size(0) == n_ && v.is_contiguous() && out.dim() == 2 && out.is_contiguous() && out.size(1) == v.size(1),
                "v must be a contiguous (n, k) tensor and out (rows, k)");
    const int64_t rows = std::max<int64_t>(0, std::min(n_, (begin_ + count_) * KM_BLOCK_SIZE) - begin_ * KM_BLOCK_SIZE);
    TORCH_CHECK(out.size(0) == rows && v.size(1) <= KM_NODE_MAX_COLUMNS, "out must have ", rows, " rows and at most ",
                KM_NODE_MAX_COLUMNS, " columns");
    const c10::cuda::CUDAGuard guard(x_.device());
    use();
    const Tensor scratch = nodes(v.size(1));
    compress(v, v.size(1), scratch.data_ptr<float>());
    product(v.size(1), scratch.const_data_ptr<float>(), out.data_ptr<float>(), nullptr, 0.0, nullptr);
}

// Iterations first .. first + count - 1 of a solve on one GPU: what CGSolver.step() does, from here.  With
// `nodes` the product, q and the partial sums of p . q are one kernel, and the update of p and its
// compression another; otherwise `rows` is the product.
void cg_run(const CgState &s, const NodeOperator *nodes, RowsProduct *rows, int64_t first, int64_t count) {
    const c10::cuda::CUDAGuard guard(s.p.device());
    void *stream = c10::cuda::getCurrentCUDAStream(s.p.device().index()).stream();
    const int64_t k = s.k, n = s.n;
    float *x = s.x.data_ptr<float>(), *r = s.r.data_ptr<float>(), *p = s.p.data_ptr<float>(), *q = s.kp.data_ptr<float>();
    float *bp = s.bp.data_ptr<float>();
    const auto totals = [&](const Tensor &to) {
        raise_on(km_cg_segment_sums_f32(k, bp, s.blocks, s.seg_blocks, static_cast<double *>(to.data_ptr()), stream));
    };
    TORCH_CHECK((nodes != nullptr) != (rows != nullptr), "one kind of product");
    if (nodes != nullptr) nodes->use();
    const Tensor scratch = nodes != nullptr ? nodes->nodes(k) : Tensor();
    float *at_nodes = nodes != nullptr ? scratch.data_ptr<float>() : nullptr;
    for (int64_t it = first; it < first + count; it++) {
        if (nodes != nullptr) {
            if (it == first) nodes->compress(s.p, k, at_nodes);
            nodes->product(k, at_nodes, q, p, s.sigma2, bp);
        } else {
            rows->run();
            raise_on(km_cg_q_dots_f32(k, q, p, (float)s.sigma2, 0, n, bp, nullptr, 0, nullptr, 0, stream));
        }
        totals(s.send1);
        raise_on(km_cg_update_xr_f32(k, x, r, p, q, nullptr, 0, nullptr, 0, 0, n, 0, n, s.send1.data_ptr(), s.send1.numel(), 1, (int32_t)s.slots,
                                     s.rs_row(it), bp, s.row(s.alphas, it), stream));
        totals(s.send2);
        if (nodes != nullptr && it + 1 < first + count)
            nodes->update_p(s, it, at_nodes);
        else
            raise_on(km_cg_update_p_f32(k, p, r, 0, n, s.send2.data_ptr(), s.send2.numel(), 1, (int32_t)s.slots, s.rs_row(it), s.rs_row(it + 1),
                                        s.ynorm.const_data_ptr<float>(), s.row(s.history, it + 1), s.row(s.betas, it), stream));
    }
}

Tensor log_forms(const Tensor &alphas, const Tensor &betas, const Tensor &residual_norms, const Tensor &z_norm2, double converged) {
    for (const Tensor *t : {&alphas, &betas, &residual_norms, &z_norm2}) check_f32(*t);
    TORCH_CHECK(alphas.dim() == 2 && betas.sizes() == alphas.sizes() && residual_norms.dim() == 2 &&
                    residual_norms.size(0) == alphas.size(0) + 1 && residual_norms.size(1) == alphas.size(1) && z_norm2.dim() == 1 &&
                    z_norm2.size(0) == alphas.size(1),
                "alphas and betas must be (m, k), residual_norms (m + 1, k) and z_norm2 (k,)");
    const c10::cuda::CUDAGuard guard(alphas.device());
    const Tensor a = alphas.contiguous(), b = betas.contiguous(), r = residual_norms.contiguous(), z = z_norm2.contiguous();
    Tensor out = at::empty({alphas.size(1)}, alphas.options().dtype(at::kDouble).requires_grad(false));
    raise_on(km_cg_log_forms_f32(a.size(0), a.size(1), a.const_data_ptr<float>(), b.const_data_ptr<float>(), r.const_data_ptr<float>(),
                                 z.const_data_ptr<float>(), (float)converged, out.data_ptr<double>(),
                                 c10::cuda::getCurrentCUDAStream(alphas.device().index()).stream()));
    return out;
}

}  // namespace kmh
