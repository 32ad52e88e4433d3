// The differentiable ops: gradients for the kernel parameters only, as in the reference's three
// autograd Functions (kernel_matmul/linear_operator.py:22-76; its index backward unpacks eight saved
// tensors into seven names, :71-72, which fails as soon as batch indices are present).  In C++ the
// backward of a training step runs without the interpreter.
#include <c10/core/impl/TorchDispatchModeTLS.h>
#include <torch/csrc/autograd/custom_function.h>
#include <torch/csrc/jit/frontend/tracer.h>

#include "km_host.h"

namespace kmh {

using torch::autograd::AutogradContext;
using torch::autograd::variable_list;

struct MatmulFunction : torch::autograd::Function<MatmulFunction> {
    static Tensor forward(AutogradContext *ctx, const Tensor &x1, const Tensor &x2, const Tensor &rhs, const Tensor &params,
                          const Tensor &start, const Tensor &end, int64_t kernel_type) {
        ctx->save_for_backward({x1, x2, rhs, params, start, end});
        ctx->saved_data["kernel_type"] = kernel_type;
        return matmul(kernel_type, x1, x2, rhs, params, start, end, PATH_AUTO);
    }
    static variable_list backward(AutogradContext *ctx, variable_list grads) {
        const auto s = ctx->get_saved_variables();
        Tensor g;
        if (ctx->needs_input_grad(3))
            g = at::sum_to(bilinear(ctx->saved_data["kernel_type"].toInt(), s[0], s[1], grads[0], s[2], s[3], s[4], s[5], PATH_AUTO),
                           s[3].sizes());
        return {Tensor(), Tensor(), Tensor(), g, Tensor(), Tensor(), Tensor()};
    }
};

struct DenseFunction : torch::autograd::Function<DenseFunction> {
    static Tensor forward(AutogradContext *ctx, const Tensor &x1, const Tensor &x2, const Tensor &params, const Tensor &start,
                          const Tensor &end, int64_t kernel_type) {
        ctx->save_for_backward({x1, x2, params, start, end});
        ctx->saved_data["kernel_type"] = kernel_type;
        return dense(kernel_type, x1, x2, params, start, end);
    }
    static variable_list backward(AutogradContext *ctx, variable_list grads) {
        const auto s = ctx->get_saved_variables();
        Tensor g;
        if (ctx->needs_input_grad(2))
            g = at::sum_to(dense_bwd(ctx->saved_data["kernel_type"].toInt(), s[0], s[1], s[2], s[3], s[4], grads[0]), s[2].sizes());
        return {Tensor(), Tensor(), g, Tensor(), Tensor(), Tensor()};
    }
};

struct IndexFunction : torch::autograd::Function<IndexFunction> {
    static Tensor forward(AutogradContext *ctx, const Tensor &x1, const Tensor &x2, const Tensor &params, const Tensor &start,
                          const Tensor &end, const std::vector<Tensor> &batch_indices, const Tensor &row, const Tensor &col,
                          int64_t kernel_type) {
        Tensor distances;
        Tensor out = index(kernel_type, x1, x2, params, start, end, batch_indices, row, col, params.requires_grad() ? &distances : nullptr);
        variable_list saved{x1, x2, params, start, end, row, col, distances};
        saved.insert(saved.end(), batch_indices.begin(), batch_indices.end());
        ctx->save_for_backward(std::move(saved));
        ctx->saved_data["kernel_type"] = kernel_type;
        return out;
    }
    static variable_list backward(AutogradContext *ctx, variable_list grads) {
        const auto s = ctx->get_saved_variables();
        Tensor g;
        if (ctx->needs_input_grad(2))
            g = at::sum_to(index_bwd(ctx->saved_data["kernel_type"].toInt(), s[0], s[1], s[2], s[3], s[4], {s.begin() + 8, s.end()},
                                     s[5], s[6], grads[0], s[7].defined() ? &s[7] : nullptr),
                           s[2].sizes());
        variable_list r(9);
        r[2] = g;
        return r;
    }
};

// params (batch.., P) and, with a `cutoff_factor`, the cutoff of the largest lengthscale.
struct PositiveParams : torch::autograd::Function<PositiveParams> {
    static variable_list forward(AutogradContext *ctx, at::TensorList raw_in, double lower_bound, int64_t lengthscales,
                                 std::optional<double> cutoff_factor) {
        std::vector<Tensor> raw, dense;
        const float *ptr[KM_MAX_PARAMS];
        TORCH_CHECK(raw_in.size() >= 1 && raw_in.size() <= KM_MAX_PARAMS, "1 to ", KM_MAX_PARAMS, " raw parameters");
        for (const Tensor &t : raw_in) {
            check_f32(t);
            TORCH_CHECK(t.sizes() == raw_in[0].sizes() && t.device() == raw_in[0].device(), "raw parameters must share shape and device");
            raw.push_back(t);  // (saved as given: the gradient's own derivative goes through it)
            dense.push_back(t.contiguous());
            ptr[raw.size() - 1] = dense.back().const_data_ptr<float>();
        }
        const c10::cuda::CUDAGuard guard(raw[0].device());
        Shape shape(raw[0].sizes().begin(), raw[0].sizes().end());
        shape.push_back((int64_t)raw.size());
        const auto opt = raw[0].options().requires_grad(false);
        Tensor params = at::empty(shape, opt), cutoff = at::empty({1}, opt);
        raise_on(km_positive_params_f32((int32_t)raw.size(), raw[0].numel(), ptr, (float)lower_bound, params.data_ptr<float>(),
                                        (uint32_t)lengthscales, cutoff_factor.value_or(0.0), cutoff_factor ? cutoff.data_ptr<float>() : nullptr,
                                        c10::cuda::getCurrentCUDAStream(raw[0].device().index()).stream()));
        ctx->save_for_backward(raw);
        ctx->mark_non_differentiable({cutoff});
        return {params, cutoff};
    }
    static variable_list backward(AutogradContext *ctx, variable_list grads) {
        const auto raw = ctx->get_saved_variables();
        const Tensor &g = grads[0];
        const c10::cuda::CUDAGuard guard(raw[0].device());
        variable_list out(raw.size() + 3);
        if (!g.defined()) return out;
        if (at::GradMode::is_enabled()) {  // (create_graph: the gradient itself is differentiable)
            for (size_t q = 0; q < raw.size(); q++)
                out[q] = at::where(raw[q] > 20.0, g.select(-1, (int64_t)q), g.select(-1, (int64_t)q) * at::sigmoid(raw[q]));
            return out;
        }
        const float *ptr[KM_MAX_PARAMS];
        float *to[KM_MAX_PARAMS];
        std::vector<Tensor> dense;
        Tensor flat = g.reshape({-1, (int64_t)raw.size()});
        for (size_t q = 0; q < raw.size(); q++) {
            dense.push_back(raw[q].contiguous());
            ptr[q] = dense.back().const_data_ptr<float>();
            out[q] = at::empty(raw[q].sizes(), raw[q].options().requires_grad(false));
            to[q] = out[q].data_ptr<float>();
        }
        raise_on(km_positive_params_bwd_f32((int32_t)raw.size(), raw[0].numel(), ptr, flat.const_data_ptr<float>(), flat.stride(0),
                                            flat.stride(1), to, c10::cuda::getCurrentCUDAStream(raw[0].device().index()).stream()));
        return out;
    }
};

// Whether a call has to go through the autograd function: for a gradient, or -- so that it is refused
// there, not ignored -- for a forward-mode tangent.
static bool recording(std::initializer_list<const Tensor *> inputs) {
    for (const Tensor *t : inputs)
        if ((t->requires_grad() && at::GradMode::is_enabled()) || t->_fw_grad(0).defined()) return true;
    return false;
}

Tensor matmul_ad(int64_t kernel_type, const Tensor &x1, const Tensor &x2, const Tensor &rhs, const Tensor &params,
                 const Tensor &start, const Tensor &end) {
    if (!recording({&x1, &x2, &rhs, &params})) return matmul(kernel_type, x1, x2, rhs, params, start, end, PATH_AUTO);
    return MatmulFunction::apply(x1, x2, rhs, params, start, end, kernel_type);
}

Tensor dense_ad(int64_t kernel_type, const Tensor &x1, const Tensor &x2, const Tensor &params, const Tensor &start, const Tensor &end) {
    if (!recording({&x1, &x2, &params})) return dense(kernel_type, x1, x2, params, start, end);
    return DenseFunction::apply(x1, x2, params, start, end, kernel_type);
}

Tensor index_ad(int64_t kernel_type, const Tensor &x1, const Tensor &x2, const Tensor &params, const Tensor &start,
                const Tensor &end, const std::vector<Tensor> &batch_indices, const Tensor &row, const Tensor &col) {
    if (!recording({&x1, &x2, &params})) return index(kernel_type, x1, x2, params, start, end, batch_indices, row, col);
    return IndexFunction::apply(x1, x2, params, start, end, batch_indices, row, col, kernel_type);
}

// Tensors on which the kernels of PositiveParams cannot stand in for tensor expressions: under jit
// tracing, forward-mode differentiation, torch.func transforms, dispatch modes and subclasses, or empty.
static bool needs_expressions(const std::vector<Tensor> &raw) {
    constexpr c10::DispatchKeySet wrapped({c10::DispatchKey::Python, c10::DispatchKey::FuncTorchBatched,
                                           c10::DispatchKey::FuncTorchGradWrapper, c10::DispatchKey::Functionalize});
    if (torch::jit::tracer::isTracing() || c10::impl::TorchDispatchModeTLS::any_modes_set()) return true;
    for (const Tensor &t : raw)
        if (t.key_set().has_any(wrapped) || t.numel() == 0 || t._fw_grad(0).defined()) return true;
    return false;
}

std::pair<Tensor, Tensor> positive_params(const std::vector<Tensor> &raw, double lower_bound, int64_t lengthscales,
                                          std::optional<double> cutoff_factor) {
    if (!needs_expressions(raw)) {
        variable_list r = PositiveParams::apply(at::TensorList(raw), lower_bound, lengthscales, cutoff_factor);
        return {r[0], r[1]};
    }
    std::vector<Tensor> values, largest;
    for (size_t q = 0; q < raw.size(); q++) {
        values.push_back(at::softplus(raw[q]) + lower_bound);
        if (cutoff_factor && ((lengthscales >> q) & 1)) largest.push_back(values.back().detach().max());
    }
    Tensor cutoff;
    if (!largest.empty()) cutoff = (at::stack(largest).max().to(at::kDouble) * *cutoff_factor).to(at::kFloat).reshape({1});
    return {at::stack(values, -1), cutoff};
}

}  // namespace kmh
