// kernel_matmul_b200._C -- the thin PyTorch C++ extension over the C ABI of libkm_b200.so.
//
// One ahead-of-time module with the ten functions the reference reaches through its per-op
// pybind11 modules (native/<op>/<op>.cpp `call`, native/ranges/ranges.cpp:152-156), the kernel
// type passed as a runtime integer (KM_KERNEL_*) instead of a -DKM_KERNEL_* define.  Each
// function checks its arguments with the reference's messages (native/common/entrypoint.h:3-14),
// allocates outputs and workspaces through ATen on x1's device, and launches on the current
// PyTorch stream under a device guard with the GIL released.  No arithmetic happens here.
#include <torch/extension.h>

#include <c10/cuda/CUDAGuard.h>
#include <c10/cuda/CUDAStream.h>

#include <vector>

#include "km_cg_host.h"

namespace {

namespace py = pybind11;
using kmh::Shape;
using torch::Tensor;

void *stream_of(const torch::Tensor &t) { return c10::cuda::getCurrentCUDAStream(t.device().index()).stream(); }

// ranges.make_ranges(x1, x2, cutoff, block_size, align)  (native/ranges/ranges.cpp:8-62), on the device
std::tuple<torch::Tensor, torch::Tensor> make_ranges(torch::Tensor x1, torch::Tensor x2, double cutoff, int64_t block_size,
                                                     bool align) {
    kmh::check_f32(x1), kmh::check_f32(x2);
    TORCH_CHECK(x1.dim() == 2 && x2.dim() == 2 && x1.size(0) == x2.size(0), "x1 and x2 must be (B, m) and (B, n)");
    const c10::cuda::CUDAGuard guard(x1.device());
    torch::Tensor a = x1.contiguous(), b = x2.contiguous();
    const int64_t B = a.size(0), m = a.size(1), n = b.size(1), R = (m + block_size - 1) / block_size;
    auto iopt = x1.options().dtype(torch::kInt32);
    torch::Tensor start = torch::empty({B, R}, iopt), end = torch::empty({B, R}, iopt), flags = torch::empty({std::max<int64_t>(B, 1)}, iopt);
    kmh::raise_on(km_make_ranges_f32(B, m, n, a.data_ptr<float>(), b.data_ptr<float>(), (float)cutoff, (int32_t)block_size,
                                align ? 1 : 0, start.data_ptr<int32_t>(), end.data_ptr<int32_t>(), flags.data_ptr<int32_t>(),
                                stream_of(x1)));
    return {start, end};
}

// ranges.make_ranges_symmetric(x, cutoff, block_size)  (native/ranges/ranges.cpp:64-101)
std::tuple<torch::Tensor, torch::Tensor> make_ranges_symmetric(torch::Tensor x, double cutoff, int64_t block_size) {
    kmh::check_f32(x);
    TORCH_CHECK(x.dim() == 2, "x must be (B, n)");
    const c10::cuda::CUDAGuard guard(x.device());
    torch::Tensor a = x.contiguous();
    const int64_t B = a.size(0), n = a.size(1), R = (n + block_size - 1) / block_size;
    auto iopt = x.options().dtype(torch::kInt32);
    torch::Tensor start = torch::empty({B, R}, iopt), end = torch::empty({B, R}, iopt), flags = torch::empty({std::max<int64_t>(B, 1)}, iopt);
    kmh::raise_on(km_make_ranges_symmetric_f32(B, n, a.data_ptr<float>(), (float)cutoff, (int32_t)block_size,
                                          start.data_ptr<int32_t>(), end.data_ptr<int32_t>(), flags.data_ptr<int32_t>(),
                                          stream_of(x)));
    return {start, end};
}

// ranges.transpose_ranges(start, end, x1_size, x2_size, block_size)  (native/ranges/ranges.cpp:103-150)
std::tuple<torch::Tensor, torch::Tensor> transpose_ranges(torch::Tensor start, torch::Tensor end, int64_t x1_size,
                                                          int64_t x2_size, int64_t block_size) {
    kmh::check_i32(start), kmh::check_i32(end);
    TORCH_CHECK(start.dim() == 2 && end.sizes() == start.sizes(), "start and end must be (B, R)");
    const c10::cuda::CUDAGuard guard(start.device());
    torch::Tensor s = start.contiguous(), e = end.contiguous();
    const int64_t B = s.size(0), R = s.size(1), C = (x2_size + block_size - 1) / block_size;
    torch::Tensor st = torch::empty({B, C}, s.options()), et = torch::empty({B, C}, s.options());
    kmh::raise_on(km_transpose_ranges_i32(B, R, s.data_ptr<int32_t>(), e.data_ptr<int32_t>(), x1_size, x2_size, (int32_t)block_size,
                                     st.data_ptr<int32_t>(), et.data_ptr<int32_t>(), stream_of(start)));
    return {st, et};
}


// Band of inputs (batch.., n1) [and (batch.., n2)]: kernel_matmul_b200.ranges.make_ranges for fp32 CUDA
// tensors and a given cutoff.
std::tuple<Tensor, Tensor> band(double cutoff, const Tensor &x1, const std::optional<Tensor> &x2, int64_t block, bool align) {
    kmh::check_f32(x1);
    const c10::cuda::CUDAGuard guard(x1.device());
    const int64_t m = x1.size(-1), R = (m + block - 1) / block;
    int64_t B = 1;
    Shape shape;
    for (int64_t d = 0; d + 1 < x1.dim(); d++) B *= x1.size(d), shape.push_back(x1.size(d));
    shape.push_back(R);
    const Tensor a = x1.contiguous();
    const auto iopt = x1.options().dtype(torch::kInt32).requires_grad(false);
    Tensor start = at::empty(shape, iopt), end = at::empty(shape, iopt), flags = at::empty({std::max<int64_t>(B, 1)}, iopt);
    if (x2.has_value()) {
        kmh::check_f32(*x2);
        TORCH_CHECK(x2->dim() == x1.dim() && x2->sizes().slice(0, x1.dim() - 1) == x1.sizes().slice(0, x1.dim() - 1),
                    "x1 and x2 must share their batch dimensions");
        TORCH_CHECK(x2->device() == x1.device(), "all tensors must be on the same CUDA device");
        const Tensor c = x2->contiguous();
        kmh::raise_on(km_make_ranges_f32(B, m, x2->size(-1), a.const_data_ptr<float>(), c.const_data_ptr<float>(), (float)cutoff,
                                         (int32_t)block, align ? 1 : 0, start.data_ptr<int32_t>(), end.data_ptr<int32_t>(),
                                         flags.data_ptr<int32_t>(), stream_of(x1)));
    } else {
        kmh::raise_on(km_make_ranges_symmetric_f32(B, m, a.const_data_ptr<float>(), (float)cutoff, (int32_t)block,
                                                   start.data_ptr<int32_t>(), end.data_ptr<int32_t>(), flags.data_ptr<int32_t>(),
                                                   stream_of(x1)));
    }
    return {start, end};
}

// Symmetric bands of B kernels with cutoffs (B,) over x (n,) or (B, n): (B, R) each, or (R,) with `single`.
std::tuple<Tensor, Tensor> band_cutoffs(const Tensor &cutoffs, const Tensor &x, int64_t block, bool single) {
    kmh::check_f32(cutoffs), kmh::check_f32(x);
    TORCH_CHECK(cutoffs.device() == x.device(), "all tensors must be on the same CUDA device");
    const c10::cuda::CUDAGuard guard(x.device());
    const int64_t n = x.size(-1), R = (n + block - 1) / block, B = cutoffs.size(0);
    const Tensor a = x.contiguous(), c = cutoffs.contiguous();
    const auto iopt = x.options().dtype(torch::kInt32).requires_grad(false);
    const Shape shape = single ? Shape{R} : Shape{B, R};
    Tensor start = at::empty(shape, iopt), end = at::empty(shape, iopt), flags = at::empty({std::max<int64_t>(B, 1)}, iopt);
    kmh::raise_on(km_make_ranges_symmetric_cutoffs_f32(B, n, a.const_data_ptr<float>(), x.dim() == 2 ? n : 0, c.const_data_ptr<float>(),
                                                       (int32_t)block, start.data_ptr<int32_t>(), end.data_ptr<int32_t>(),
                                                       flags.data_ptr<int32_t>(), stream_of(x)));
    return {start, end};
}

// The arguments of an operator (x1 (.., M, 1), x2 (.., N, 1), params, start, end) expanded to their
// common batch shape; x1 and x2 also without the last dim, as the native ops take them.
std::vector<Tensor> expand_operator(const Tensor &x1, const Tensor &x2, const Tensor &params, const Tensor &start, const Tensor &end) {
    std::vector<int64_t> batch(x1.sizes().begin(), x1.sizes().end() - 2);
    const auto grow = [&](const Tensor &t, int nonbatch) {
        TORCH_CHECK(t.dim() >= nonbatch, "tensor of rank ", t.dim(), " needs at least ", nonbatch, " dims");
        batch = at::infer_size(batch, t.sizes().slice(0, t.dim() - nonbatch));
    };
    grow(x2, 2), grow(params, 1), grow(start, 1), grow(end, 1);
    const auto widen = [&](const Tensor &t, int nonbatch) {
        if (t.sizes().slice(0, t.dim() - nonbatch) == at::IntArrayRef(batch)) return t;
        std::vector<int64_t> s(batch);
        s.insert(s.end(), t.sizes().end() - nonbatch, t.sizes().end());
        return t.expand(s);
    };
    const Tensor a = widen(x1, 2), c = widen(x2, 2);
    return {a, c, widen(params, 1), widen(start, 1), widen(end, 1), a.squeeze(-1), x2.is_same(x1) ? a.squeeze(-1) : c.squeeze(-1)};
}

}  // namespace

PYBIND11_MODULE(TORCH_EXTENSION_NAME, m) {
    m.doc() = "B200 kernel-matmul ops: PyTorch binding of libkm_b200.so";
    m.attr("KERNEL_RBF") = (int)KM_KERNEL_RBF;
    m.attr("KERNEL_SPECTRAL") = (int)KM_KERNEL_SPECTRAL;
    m.attr("KERNEL_LOCALLY_PERIODIC") = (int)KM_KERNEL_LOCALLY_PERIODIC;
    m.attr("TENSOR_CORE_MIN_K") = kmh::TENSOR_CORE_MIN_K;
    m.attr("GRAD_TENSOR_CORE_MIN_K") = kmh::GRAD_TENSOR_CORE_MIN_K;
    m.attr("NODE_MAX_COLUMNS") = KM_NODE_MAX_COLUMNS;
    m.attr("TENSOR_CORE_MIN_ITEMS") = kmh::TENSOR_CORE_MIN_ITEMS;
    // the package's own error types; without the package (the extension loaded by itself) RuntimeError
    py::register_exception_translator([](std::exception_ptr p) {
        const auto set = [](const char *module, const char *name, const std::exception &e) {
            try {
                PyErr_SetString(py::module_::import(module).attr(name).ptr(), e.what());
            } catch (py::error_already_set &) {
                PyErr_Clear();
                PyErr_SetString(PyExc_RuntimeError, e.what());
            }
        };
        try {
            if (p) std::rethrow_exception(p);
        } catch (const kmh::StatusError &e) {
            set("kernel_matmul_b200._lib", "KmError", e);
        } catch (const kmh::GaveUpError &e) {
            set("kernel_matmul_b200.ops", "KernelGaveUpError", e);
        }
    });

    using nogil = py::call_guard<py::gil_scoped_release>;
    // the ten functions of the reference's native modules
    m.def(
        "matmul",
        [](int64_t kt, const Tensor &x1, const Tensor &x2, const Tensor &rhs, const Tensor &params, const Tensor &start,
           const Tensor &end, bool tensor_cores_auto) {
            return kmh::matmul(kt, x1, x2, rhs, params, start, end, tensor_cores_auto ? kmh::PATH_AUTO : kmh::PATH_FMA);
        },
        py::arg("kernel_type"), py::arg("x1"), py::arg("x2"), py::arg("rhs"), py::arg("params"), py::arg("start"), py::arg("end"),
        py::arg("tensor_cores_auto") = true, nogil());
    m.def("matmul_bwd",
          [](int64_t kt, const Tensor &x1, const Tensor &x2, const Tensor &rhs, const Tensor &params, const Tensor &start,
             const Tensor &end, const Tensor &out_grad) {
              return kmh::bilinear(kt, x1, x2, out_grad, rhs, params, start, end, kmh::PATH_AUTO);
          },
          nogil());
    m.def("bilinear_derivative",
          [](int64_t kt, const Tensor &x1, const Tensor &x2, const Tensor &left, const Tensor &right, const Tensor &params,
             const Tensor &start, const Tensor &end) {
              return kmh::bilinear(kt, x1, x2, left, right, params, start, end, kmh::PATH_AUTO);
          },
          nogil());
    m.def("dense", &kmh::dense, nogil());
    m.def("dense_bwd", &kmh::dense_bwd, nogil());
    using torch::Tensor;
    using Indices = std::vector<Tensor>;
    m.def("index", [](int64_t kt, const Tensor &x1, const Tensor &x2, const Tensor &params, const Tensor &start, const Tensor &end,
                      const Indices &batch, const Tensor &row, const Tensor &col) {
        return kmh::index(kt, x1, x2, params, start, end, batch, row, col);
    }, nogil());
    m.def("index_bwd", [](int64_t kt, const Tensor &x1, const Tensor &x2, const Tensor &params, const Tensor &start, const Tensor &end,
                          const Indices &batch, const Tensor &row, const Tensor &col, const Tensor &out_grad) {
        return kmh::index_bwd(kt, x1, x2, params, start, end, batch, row, col, out_grad);
    }, nogil());
    m.def("make_ranges", &make_ranges);
    m.def("make_ranges_symmetric", &make_ranges_symmetric);
    m.def("transpose_ranges", &transpose_ranges);

    // what the Python layer is built on
    m.def("op_matmul",
          [](int64_t kt, const Tensor &x1, const Tensor &x2, const Tensor &rhs, const Tensor &params, const Tensor &start,
             const Tensor &end, int64_t path) {
              bool tc = false;
              Tensor out = kmh::matmul(kt, x1, x2, rhs, params, start, end, path, &tc);
              return std::make_pair(out, tc);
          },
          nogil());
    m.def("op_bilinear",
          [](int64_t kt, const Tensor &x1, const Tensor &x2, const Tensor &left, const Tensor &right, const Tensor &params,
             const Tensor &start, const Tensor &end, int64_t path) {
              bool tc = false;
              Tensor grad = kmh::bilinear(kt, x1, x2, left, right, params, start, end, path, &tc);
              return std::make_pair(grad, tc);
          },
          nogil());
    py::class_<kmh::RowsProduct>(m, "RowsProduct")
        .def(py::init<int64_t, const Tensor &, const Tensor &, const Tensor &, const Tensor &, const Tensor &, const Tensor &, int64_t,
                      int64_t, bool, const std::optional<Tensor> &, int64_t, const std::optional<Tensor> &>())
        .def("__call__", &kmh::RowsProduct::run, nogil())
        .def_property_readonly("out", &kmh::RowsProduct::out)
        .def_property_readonly("tensor_cores", &kmh::RowsProduct::tensor_cores);
    py::class_<kmh::NodeOperator>(m, "NodeOperator")
        .def(py::init<int64_t, const std::optional<Tensor> &, const std::optional<Tensor> &, const Tensor &, const Tensor &, int64_t,
                      int64_t>())
        .def("plan", &kmh::NodeOperator::plan)
        .def("build", &kmh::NodeOperator::build, nogil())
        .def("changed", &kmh::NodeOperator::changed, nogil())
        .def("matvec", &kmh::NodeOperator::matvec, nogil());
    py::class_<kmh::CgState>(m, "CgState")
        .def(py::init([](const Tensor &x, const Tensor &r, const Tensor &p, const Tensor &kp, const Tensor &bp, const Tensor &rs,
                         const Tensor &ynorm, const Tensor &history, const Tensor &alphas, const Tensor &betas, const Tensor &send1,
                         const Tensor &send2, int64_t n, int64_t k, int64_t blocks, int64_t seg_blocks, int64_t slots, double sigma2) {
            return kmh::CgState{x, r, p, kp, bp, rs, ynorm, history, alphas, betas, send1, send2, n, k, blocks, seg_blocks, slots, sigma2};
        }));
    m.def("cg_run", [](const kmh::CgState &s, kmh::NodeOperator *nodes, kmh::RowsProduct *rows, int64_t first, int64_t count) {
        py::gil_scoped_release release;
        kmh::cg_run(s, nodes, rows, first, count);
    });
    m.def("log_forms", &kmh::log_forms, nogil());
    m.def("matmul_ad", &kmh::matmul_ad, nogil());
    m.def("dense_ad", &kmh::dense_ad, nogil());
    m.def("index_ad", &kmh::index_ad, nogil());
    m.def("positive_params", &kmh::positive_params, nogil());
    m.def("poll_gave_up", &kmh::poll_gave_up);
    m.def("band", &band, nogil());
    m.def("band_cutoffs", &band_cutoffs, nogil());
    m.def("expand_operator", &expand_operator, nogil());
}
