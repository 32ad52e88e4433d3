#include "km_host.h"

#include <ATen/ExpandUtils.h>

#include <sstream>

namespace kmh {

static const char *const KERNEL_NAMES[] = {"rbf", "spectral", "locally_periodic"};

static void check_cuda(const Tensor &x) { TORCH_CHECK(x.is_cuda(), "x must be a CUDA tensor"); }
void check_f32(const Tensor &x) {
    check_cuda(x);
    TORCH_CHECK(x.scalar_type() == at::kFloat, "x must be float32");
}
void check_i32(const Tensor &x) {
    check_cuda(x);
    TORCH_CHECK(x.scalar_type() == at::kInt, "x must be int32");
}

int num_params(int64_t kernel_type) {
    const int p = km_num_params((int)kernel_type);
    TORCH_CHECK(p > 0, "Unknown kernel type: ", kernel_type);
    return p;
}

void poll_gave_up(int device) {
    int32_t what = 0;
    raise_on(km_take_gave_up(device, &what));
    if (what != 0)
        throw GaveUpError(std::string(what == 1 ? "matmul" : "gradient") +
                          ": a bounded wait inside the tensor-core kernel gave up (status word != 0); "
                          "the results of that call are invalid");
}

static void add_batch(Shape &batch, const Tensor &t, int nonbatch) {
    TORCH_CHECK(t.dim() >= nonbatch, "tensor of rank ", t.dim(), " needs at least ", nonbatch, " trailing dims");
    const int64_t lead = t.dim() - nonbatch;
    while ((int64_t)batch.size() < lead) batch.insert(batch.begin(), 1);
    const int64_t shift = (int64_t)batch.size() - lead;
    for (int64_t d = 0; d < lead; d++) {
        int64_t &have = batch[shift + d];
        const int64_t size = t.size(d);
        if (size == have || size == 1) continue;
        TORCH_CHECK(have == 1, "batch dimensions do not broadcast: ", have, " against ", size, " in batch dim ", shift + d);
        have = size;
    }
}

Problem::Problem(int64_t kernel_type, const Tensor &tx1, const Tensor &tx2, const Tensor &tparams, const Tensor &tstart,
                 const Tensor &tend, std::initializer_list<std::pair<const Tensor *, int>> extra) {
    const int P = num_params(kernel_type);
    kid = (int)kernel_type;
    check_f32(tx1), check_f32(tx2), check_f32(tparams), check_i32(tstart), check_i32(tend);
    for (const auto &e : extra) check_f32(*e.first);
    const auto dev = tx1.device();
    auto same = [&](const Tensor &t) { TORCH_CHECK(t.device() == dev, "all tensors must be on the same CUDA device"); };
    same(tx2), same(tparams), same(tstart), same(tend);
    for (const auto &e : extra) same(*e.first);
    device = dev.index();
    poll_gave_up(device);
    TORCH_CHECK(tx1.dim() >= 1 && tx2.dim() >= 1 && tparams.dim() >= 1 && tstart.dim() >= 1 && tend.dim() >= 1,
                "tensor of rank 0 needs at least 1 trailing dims");
    TORCH_CHECK(tparams.size(-1) == P, "params must have ", P, " entries in the last dim for kernel '", KERNEL_NAMES[kid], "', got ",
                tparams.size(-1));
    m = tx1.size(-1);
    n = tx2.size(-1);
    row_blocks = (m + KM_BLOCK_SIZE - 1) / KM_BLOCK_SIZE;
    TORCH_CHECK(tstart.size(-1) == row_blocks && tend.size(-1) == row_blocks, "start/end must have ceil(m/", KM_BLOCK_SIZE, ") = ",
                row_blocks, " entries, got ", tstart.size(-1), " and ", tend.size(-1));
    add_batch(batch, tx1, 1), add_batch(batch, tx2, 1), add_batch(batch, tparams, 1), add_batch(batch, tstart, 1),
        add_batch(batch, tend, 1);
    for (const auto &e : extra) add_batch(batch, *e.first, e.second);
    flat_ = batch.size() > KM_MAX_BATCH_DIMS;
    if (flat_) {
        kb.ndim = 1;
        kb.size[0] = items() / std::max<int64_t>(row_blocks, 1);
        if (row_blocks == 0) {
            kb.size[0] = 1;
            for (int64_t b : batch) kb.size[0] *= b;
        }
    } else {
        kb.ndim = (int32_t)batch.size();
        for (size_t d = 0; d < batch.size(); d++) kb.size[d] = batch[d];
    }
    x1 = view(tx1, 1), x2 = view(tx2, 1), params = view(tparams, 1), start = view(tstart, 1), end = view(tend, 1);
    all_columns_ = row_blocks > 1 && tstart.storage_offset() > 0 && tend.storage_offset() == 0 && tstart.strides() == tend.strides() &&
                   tstart.is_alias_of(tend) &&
                   tstart.storage().nbytes() == 2 * sizeof(int32_t) * (size_t)tstart.storage_offset();
}

int64_t Problem::items() const {
    int64_t v = row_blocks;
    for (int64_t b : batch) v *= b;
    return v;
}

km_view Problem::view(const Tensor &t, int nonbatch) {
    km_view v{};
    if (flat_) {  // more batch dims than the ABI carries: flatten them (a copy only if not collapsible)
        Shape wide(batch), narrow{-1};
        for (int64_t d = t.dim() - nonbatch; d < t.dim(); d++) wide.push_back(t.size(d)), narrow.push_back(t.size(d));
        if (kb.size[0] == 0) narrow[0] = 0;
        keep.push_back(t.expand(wide).reshape(narrow));
        const Tensor &f = keep.back();
        v.data = f.data_ptr();
        v.batch_stride[0] = f.stride(0);
        for (int d = 0; d < nonbatch; d++) v.stride[d] = f.stride(1 + d);
        return v;
    }
    v.data = t.data_ptr();
    const int64_t lead = t.dim() - nonbatch, shift = (int64_t)batch.size() - lead;
    for (int64_t d = 0; d < lead; d++) v.batch_stride[shift + d] = t.size(d) == 1 ? 0 : t.stride(d);
    for (int d = 0; d < nonbatch; d++) v.stride[d] = t.stride(lead + d);
    return v;
}

Tensor Problem::empty(std::initializer_list<int64_t> tail, const Tensor &like) const {
    Shape s(batch);
    s.insert(s.end(), tail.begin(), tail.end());
    return at::empty(s, like.options().requires_grad(false));
}

Tensor workspace(const Tensor &like, size_t bytes) {
    return at::empty({(int64_t)std::max<size_t>(bytes, 256)}, like.options().dtype(at::kByte).requires_grad(false));
}

// The same, or an undefined tensor where the device has not that much memory left.
static Tensor workspace_if_free(const Tensor &like, size_t bytes) {
    try {
        return workspace(like, bytes);
    } catch (const c10::OutOfMemoryError &) {
        return Tensor();
    }
}

static std::string shape_of(const Tensor &t) {
    std::ostringstream s;
    s << t.sizes();
    return s.str();
}

Tensor matmul(int64_t kernel_type, const Tensor &x1, const Tensor &x2, const Tensor &rhs, const Tensor &params, const Tensor &start,
              const Tensor &end, int64_t path, bool *tc) {
    Problem p(kernel_type, x1, x2, params, start, end, {{&rhs, 2}});
    TORCH_CHECK(rhs.size(-2) == p.n, "rhs must have n = ", p.n, " rows, got ", rhs.size(-2));
    const int64_t k = rhs.size(-1);
    const c10::cuda::CUDAGuard guard(x1.device());
    Tensor out = p.empty({p.m, k}, x1);
    const km_view vr = p.view(rhs, 2), vo = p.view(out, 2);
    if (p.try_nodes(path, k, TENSOR_CORE_MIN_K)) {
        const size_t bytes = km_matmul_nodes_workspace_bytes(&p.kb, p.m, p.n, k, &p.x1, &p.x2, &vr, p.one_range());
        const Tensor ws = bytes > 0 ? workspace_if_free(x1, bytes) : Tensor();
        if (ws.defined()) {
            raise_on(km_matmul_nodes_f32(p.kid, &p.kb, p.m, p.n, k, &p.x1, &p.x2, &vr, &p.params, &p.start, &p.end, &vo, p.one_range(),
                                         ws.data_ptr(), ws.numel(), p.stream()));
            return out;
        }
    }
    const bool use_tc = path == PATH_TC || (path != PATH_FMA && k >= TENSOR_CORE_MIN_K && p.items() >= TENSOR_CORE_MIN_ITEMS);
    if (tc) *tc = use_tc;
    if (use_tc) {
        const size_t bytes = km_matmul_tc_workspace_bytes(&p.kb, p.n, k, &vr);
        Tensor ws = workspace(x1, bytes);
        raise_on(km_matmul_tc_f32(p.kid, &p.kb, p.m, p.n, k, &p.x1, &p.x2, &vr, &p.params, &p.start, &p.end, &vo, ws.data_ptr(),
                                  ws.numel(), p.stream()));
    } else {
        raise_on(km_matmul_f32(p.kid, &p.kb, p.m, p.n, k, &p.x1, &p.x2, &vr, &p.params, &p.start, &p.end, &vo, p.stream()));
    }
    return out;
}

Tensor bilinear(int64_t kernel_type, const Tensor &x1, const Tensor &x2, const Tensor &left, const Tensor &right,
                const Tensor &params, const Tensor &start, const Tensor &end, int64_t path, bool *tc) {
    Problem p(kernel_type, x1, x2, params, start, end, {{&left, 2}, {&right, 2}});
    TORCH_CHECK(left.size(-2) == p.m && right.size(-2) == p.n && left.size(-1) == right.size(-1), "left must be (.., ", p.m,
                ", k) and right (.., ", p.n, ", k); got ", shape_of(left), " and ", shape_of(right));
    const int64_t k = left.size(-1);
    const c10::cuda::CUDAGuard guard(x1.device());
    Tensor grad = p.empty({num_params(kernel_type)}, x1);
    const km_view vl = p.view(left, 2), vr = p.view(right, 2), vg = p.view(grad, 1);
    if (p.try_nodes(path, k, GRAD_TENSOR_CORE_MIN_K)) {
        const size_t bytes = km_grad_nodes_workspace_bytes(p.kid, &p.kb, p.m, p.n, k, &p.x1, &p.x2, &vl, &vr, p.one_range());
        const Tensor ws = bytes > 0 ? workspace_if_free(x1, bytes) : Tensor();
        if (ws.defined()) {
            raise_on(km_bilinear_derivative_nodes_f32(p.kid, &p.kb, p.m, p.n, k, &p.x1, &p.x2, &vl, &vr, &p.params, &p.start, &p.end, &vg,
                                                      p.one_range(), ws.data_ptr(), ws.numel(), p.stream()));
            return grad;
        }
    }
    const bool use_tc = path == PATH_TC || (path != PATH_FMA && k >= GRAD_TENSOR_CORE_MIN_K && p.items() >= TENSOR_CORE_MIN_ITEMS);
    if (tc) *tc = use_tc;
    const size_t bytes = use_tc ? km_grad_tc_workspace_bytes(&p.kb, p.m, p.n, k, &vr) : km_grad_workspace_bytes(p.kid, &p.kb, p.m);
    Tensor ws = workspace(x1, bytes);
    raise_on((use_tc ? km_bilinear_derivative_tc_f32 : km_bilinear_derivative_f32)(
        p.kid, &p.kb, p.m, p.n, k, &p.x1, &p.x2, &vl, &vr, &p.params, &p.start, &p.end, &vg, ws.data_ptr(), ws.numel(), p.stream()));
    return grad;
}

RowsProduct::RowsProduct(int64_t kernel_type, const Tensor &x1, const Tensor &x2, const Tensor &rhs, const Tensor &params,
                         const Tensor &start, const Tensor &end, int64_t row_block_begin, int64_t row_block_count, bool sum_batches,
                         const std::optional<Tensor> &out, int64_t path, const std::optional<Tensor> &phases)
    : p_(kernel_type, x1, x2, params, start, end, {{&rhs, 2}}), keep_{x1, x2, rhs, params, start, end} {
    TORCH_CHECK(rhs.size(-2) == p_.n, "rhs must have n = ", p_.n, " rows, got ", rhs.size(-2));
    k_ = rhs.size(-1);
    const int64_t R = p_.row_blocks;
    begin_ = row_block_begin;
    count_ = row_block_count < 0 ? R - row_block_begin : row_block_count;
    TORCH_CHECK(begin_ >= 0 && count_ >= 0 && begin_ + count_ <= R, "row-block window [", begin_, ", ", begin_ + count_,
                ") outside [0, ", R, ")");
    const int64_t rows = std::max<int64_t>(0, std::min(p_.m, (begin_ + count_) * KM_BLOCK_SIZE) - begin_ * KM_BLOCK_SIZE);
    Shape shape;
    if (!sum_batches) shape = p_.batch;
    shape.push_back(rows), shape.push_back(k_);
    if (out.has_value()) {
        TORCH_CHECK(out->sizes() == at::IntArrayRef(shape) && out->scalar_type() == at::kFloat && out->device() == x1.device(),
                    "out must be a float32 tensor of shape ", at::IntArrayRef(shape), " on ", x1.device());
        out_ = *out;
    } else {
        out_ = at::empty(shape, x1.options().requires_grad(false));
    }
    sum_ = sum_batches && !p_.batch.empty();  // a single kernel: nothing to sum
    TORCH_CHECK(!(sum_ && path == PATH_TC), "the batch sum runs on the FMA pipe only");
    int64_t items = count_;
    for (int64_t b : p_.batch) items *= b;
    tc_ = !sum_ && rows > 0 && (path == PATH_TC || (path == PATH_AUTO && k_ >= TENSOR_CORE_MIN_K && items >= TENSOR_CORE_MIN_ITEMS));
    set_views();
    if (sum_ && phases.has_value()) phases_ = *phases;
}

void RowsProduct::set_views() {
    rhs_ = p_.view(keep_[2], 2);
    if (sum_) {
        vout_ = km_view{};
        vout_.data = out_.data_ptr();
        vout_.stride[0] = out_.stride(0), vout_.stride[1] = out_.stride(1);
    } else {
        vout_ = p_.view(out_, 2);
    }
}

void RowsProduct::run() {
    poll_gave_up(p_.device);
    const c10::cuda::CUDAGuard guard((c10::DeviceIndex)p_.device);
    if (!p_.keep.empty()) {  // (more batch dims than the ABI carries: what was flattened may be a copy, of other contents by now)
        p_ = Problem(p_.kid, keep_[0], keep_[1], keep_[3], keep_[4], keep_[5], {{&keep_[2], 2}});
        set_views();
    }
    void *stream = p_.stream();
    if (tc_) {
        const Tensor ws = workspace(keep_[0], km_matmul_tc_workspace_bytes(&p_.kb, p_.n, k_, &rhs_));
        raise_on(km_matmul_tc_rows_f32(p_.kid, &p_.kb, p_.m, p_.n, k_, &p_.x1, &p_.x2, &rhs_, &p_.params, &p_.start, &p_.end, &vout_,
                                       begin_, count_, ws.data_ptr(), ws.numel(), stream));
    } else if (phases_.defined())
        raise_on(km_matmul_rows_phases_f32(p_.kid, &p_.kb, p_.m, p_.n, k_, &p_.x1, &p_.x2, &rhs_, &p_.params, &p_.start, &p_.end,
                                           &vout_, begin_, count_, phases_.data_ptr(), phases_.numel(), stream));
    else
        raise_on(km_matmul_rows_f32(p_.kid, &p_.kb, p_.m, p_.n, k_, &p_.x1, &p_.x2, &rhs_, &p_.params, &p_.start, &p_.end, &vout_,
                                    begin_, count_, sum_ ? 1 : 0, stream));
}

Tensor dense(int64_t kernel_type, const Tensor &x1, const Tensor &x2, const Tensor &params, const Tensor &start, const Tensor &end) {
    Problem p(kernel_type, x1, x2, params, start, end, {});
    const c10::cuda::CUDAGuard guard(x1.device());
    Tensor out = p.empty({p.m, p.n}, x1);
    const km_view vo = p.view(out, 2);
    raise_on(km_dense_f32(p.kid, &p.kb, p.m, p.n, &p.x1, &p.x2, &p.params, &p.start, &p.end, &vo, p.stream()));
    return out;
}

Tensor dense_bwd(int64_t kernel_type, const Tensor &x1, const Tensor &x2, const Tensor &params, const Tensor &start,
                 const Tensor &end, const Tensor &out_grad) {
    Problem p(kernel_type, x1, x2, params, start, end, {{&out_grad, 2}});
    TORCH_CHECK(out_grad.size(-2) == p.m && out_grad.size(-1) == p.n, "out_grad must be (.., ", p.m, ", ", p.n, "), got ",
                shape_of(out_grad));
    const c10::cuda::CUDAGuard guard(x1.device());
    Tensor grad = p.empty({num_params(kernel_type)}, x1);
    const km_view vog = p.view(out_grad, 2), vg = p.view(grad, 1);
    Tensor ws = workspace(x1, km_grad_workspace_bytes(p.kid, &p.kb, p.m));
    raise_on(km_dense_bwd_f32(p.kid, &p.kb, p.m, p.n, &p.x1, &p.x2, &p.params, &p.start, &p.end, &vog, &vg, ws.data_ptr(), ws.numel(),
                              p.stream()));
    return grad;
}

// Index tensors of one call, broadcast to one shape and contiguous.
struct Lookups {
    std::vector<int64_t> shape;
    std::vector<Tensor> flat;  // batch indices..., row, col
    const int32_t *batch[KM_MAX_BATCH_DIMS] = {nullptr, nullptr, nullptr, nullptr};
    const int32_t *row, *col;
    int64_t count;

    Lookups(const Problem &p, const char *name, const std::vector<Tensor> &batch_indices, const Tensor &r, const Tensor &c) {
        TORCH_CHECK(p.batch.size() <= KM_MAX_BATCH_DIMS, name, " supports at most ", KM_MAX_BATCH_DIMS, " batch dims");
        TORCH_CHECK(batch_indices.size() == p.batch.size(), "expected ", p.batch.size(), " batch index tensors, got ",
                    batch_indices.size());
        shape = at::infer_size(r.sizes(), c.sizes());
        for (const Tensor &b : batch_indices) shape = at::infer_size(shape, b.sizes());
        for (const Tensor &b : batch_indices) add(p, b);
        add(p, r), add(p, c);
        for (size_t d = 0; d < batch_indices.size(); d++) batch[d] = flat[d].const_data_ptr<int32_t>();
        row = flat[flat.size() - 2].const_data_ptr<int32_t>();
        col = flat.back().const_data_ptr<int32_t>();
        count = flat.back().numel();
    }
    void add(const Problem &p, const Tensor &t) {
        check_i32(t);
        TORCH_CHECK(t.device().index() == p.device, "all tensors must be on the same CUDA device");
        flat.push_back(t.sizes() == at::IntArrayRef(shape) ? t.contiguous() : t.expand(shape).contiguous());
    }
};

Tensor index(int64_t kernel_type, const Tensor &x1, const Tensor &x2, const Tensor &params, const Tensor &start, const Tensor &end,
             const std::vector<Tensor> &batch_indices, const Tensor &row, const Tensor &col, Tensor *distances) {
    Problem p(kernel_type, x1, x2, params, start, end, {});
    Lookups l(p, "index", batch_indices, row, col);
    const c10::cuda::CUDAGuard guard(x1.device());
    Tensor out = at::empty(l.shape, x1.options().requires_grad(false));
    if (distances != nullptr) {
        try {
            *distances = at::empty(l.shape, x1.options().requires_grad(false));
        } catch (const c10::OutOfMemoryError &) {  // the gradient goes back to the points
        }
    }
    if (distances != nullptr && distances->defined()) {
        raise_on(km_index_distances_f32(p.kid, &p.kb, p.m, p.n, l.count, &p.x1, &p.x2, &p.params, &p.start, &p.end, l.batch, l.row, l.col,
                                        out.data_ptr<float>(), distances->data_ptr<float>(), p.stream()));
    } else {
        raise_on(km_index_f32(p.kid, &p.kb, p.m, p.n, l.count, &p.x1, &p.x2, &p.params, &p.start, &p.end, l.batch, l.row, l.col,
                              out.data_ptr<float>(), p.stream()));
    }
    return out;
}

Tensor index_bwd(int64_t kernel_type, const Tensor &x1, const Tensor &x2, const Tensor &params, const Tensor &start,
                 const Tensor &end, const std::vector<Tensor> &batch_indices, const Tensor &row, const Tensor &col,
                 const Tensor &out_grad, const Tensor *distances) {
    Problem p(kernel_type, x1, x2, params, start, end, {});
    Lookups l(p, "index_bwd", batch_indices, row, col);
    check_f32(out_grad);
    const c10::cuda::CUDAGuard guard(x1.device());
    Tensor og = out_grad.expand(l.shape).contiguous();
    Tensor grad = p.empty({num_params(kernel_type)}, x1);
    const km_view vg = p.view(grad, 1);
    Tensor ws = workspace(x1, km_index_bwd_workspace_bytes(p.kid, &p.kb));
    if (distances != nullptr) {
        const Tensor d = distances->contiguous();
        raise_on(km_index_bwd_distances_f32(p.kid, &p.kb, l.count, &p.params, l.batch, d.const_data_ptr<float>(), og.const_data_ptr<float>(),
                                            &vg, ws.data_ptr(), ws.numel(), p.stream()));
    } else {
        raise_on(km_index_bwd_f32(p.kid, &p.kb, p.m, p.n, l.count, &p.x1, &p.x2, &p.params, &p.start, &p.end, l.batch, l.row, l.col,
                                  og.const_data_ptr<float>(), &vg, ws.data_ptr(), ws.numel(), p.stream()));
    }
    return grad;
}

}  // namespace kmh
