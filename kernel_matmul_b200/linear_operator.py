"""Autograd glue and the operator object of the hot path.

``KernelMatmulOperator`` holds ``(x1, x2, params, start, end, kernel_type)`` and offers the
operations the reference's ``KernelMatmulLinearOperator`` implements
(``kernel_matmul/linear_operator.py:79-289``): ``matmul``, ``to_dense``, ``bilinear_derivative``,
``get_indices``, ``transpose``, ``expand_batch``, ``size``.  It depends on PyTorch only.

When the third-party ``linear_operator`` package is importable, ``KernelMatmulLinearOperator``
is that package's ``LinearOperator`` subclass with the same constructor and private hooks
(``_matmul``, ``_size``, ``_transpose_nonbatch``, ``to_dense``, ``_expand_batch``,
``_bilinear_derivative``, ``_get_indices``, ``to``, ``type``) as the reference; without it the
name is bound to ``KernelMatmulOperator`` so that code using only the operator-level methods
still runs.

Products, ``to_dense`` and ``get_indices`` are differentiable in ``params`` only, as the
reference's three autograd Functions (``linear_operator.py:22-76``); the functions are in C++
(``csrc_torch/km_autograd.cpp``), so that neither direction pays for the interpreter.
"""
from __future__ import annotations

from typing import Any

import torch
from torch import Tensor

from . import _C, ranges
from ._lib import KERNEL_TYPES
from .configurations import get_kernel_type_defines

try:  # optional third-party base class
    from linear_operator import LinearOperator as _LinearOperator
    from linear_operator.utils.generic import _to_helper

    HAVE_LINEAR_OPERATOR = True
except Exception:  # noqa: BLE001 - absent or broken installation: operator-level API only
    _LinearOperator = None
    HAVE_LINEAR_OPERATOR = False


class _TracedProduct(torch.autograd.Function):
    """The op calls as calls that ``torch.jit.trace`` records (it sees nothing of the C++ functions, and
    would keep their results as constants)."""

    @staticmethod
    def forward(ctx, x1v, x2v, rhs, params, start, end, kid):
        ctx.save_for_backward(x1v, x2v, rhs, params, start, end)
        ctx.kid = kid
        return _C.op_matmul(kid, x1v, x2v, rhs, params, start, end, 0)[0]

    @staticmethod
    def backward(ctx, grad):
        x1v, x2v, rhs, params, start, end = ctx.saved_tensors
        g = _C.op_bilinear(ctx.kid, x1v, x2v, grad, rhs, params, start, end, 0)[0]
        return None, None, None, g.sum_to_size(params.shape), None, None, None


class _TracedDense(torch.autograd.Function):
    @staticmethod
    def forward(ctx, x1v, x2v, params, start, end, kid):
        ctx.save_for_backward(x1v, x2v, params, start, end)
        ctx.kid = kid
        return _C.dense(kid, x1v, x2v, params, start, end)

    @staticmethod
    def backward(ctx, grad):
        return None, None, _C.dense_bwd(ctx.kid, *ctx.saved_tensors, grad), None, None, None


class _TracedIndex(torch.autograd.Function):
    @staticmethod
    def forward(ctx, x1v, x2v, params, start, end, kid, row, col, *batch):
        ctx.save_for_backward(x1v, x2v, params, start, end, row, col, *batch)
        ctx.kid = kid
        return _C.index(kid, x1v, x2v, params, start, end, list(batch), row, col)

    @staticmethod
    def backward(ctx, grad):
        x1v, x2v, params, start, end, row, col, *batch = ctx.saved_tensors
        g = _C.index_bwd(ctx.kid, x1v, x2v, params, start, end, batch, row, col, grad)
        return None, None, g, None, None, None, None, None, *[None for _ in batch]


class _OperatorCore:
    """State and arithmetic shared by the plain operator and the LinearOperator subclass."""

    def _init_core(self, x1, x2, params, start, end, kernel_type, symmetric, compile_pool) -> None:
        if kernel_type is None:
            raise ValueError("kernel_type must be specified")
        if x1.dim() < 2 or x2.dim() < 2 or x1.size(-1) != 1 or x2.size(-1) != 1:
            raise ValueError("x1 and x2 must have shapes (..., M, 1) and (..., N, 1), respectively")
        if symmetric is None:
            symmetric = x1.shape == x2.shape and torch.equal(x1, x2)
        self._x1, self._x2, self._params, self._start, self._end, self._x1v, self._x2v = _C.expand_operator(
            x1, x2, params, start, end)
        self._kernel_type = kernel_type
        self._batch_shape = self._x1.shape[:-2]
        self._symmetric = bool(symmetric)

    # -- helpers ---------------------------------------------------------------------------
    @property
    def _kid(self) -> int:
        """Runtime kernel type of the ops.  An operator of another kernel can be made and asked for its shape;
        its products are refused, by name."""
        if self._kernel_type not in KERNEL_TYPES:
            get_kernel_type_defines(self._kernel_type)  # raises
        return KERNEL_TYPES[self._kernel_type]

    def _core_size(self) -> torch.Size:
        return torch.Size((*self._batch_shape, self._x1.size(-2), self._x2.size(-2)))

    def _core_matmul(self, rhs: Tensor) -> Tensor:
        n = self._x2.size(-2)
        if rhs.size(-2) != n:  # (a broadcast over the rows, or an error)
            rhs = rhs.expand(*rhs.shape[:-2], n, rhs.size(-1))
        if torch.jit.is_tracing():
            return _TracedProduct.apply(self._x1v, self._x2v, rhs, self._params, self._start, self._end, self._kid)
        return _C.matmul_ad(self._kid, self._x1v, self._x2v, rhs, self._params, self._start, self._end)

    def _core_to_dense(self) -> Tensor:
        if torch.jit.is_tracing():
            return _TracedDense.apply(self._x1v, self._x2v, self._params, self._start, self._end, self._kid)
        return _C.dense_ad(self._kid, self._x1v, self._x2v, self._params, self._start, self._end)

    def _core_bilinear_derivative(self, left_vecs: Tensor, right_vecs: Tensor) -> Tensor:
        return _C.op_bilinear(self._kid, self._x1v, self._x2v, left_vecs, right_vecs, self._params, self._start, self._end, 0)[0]

    def _core_get_indices(self, row_index: Tensor, col_index: Tensor, *batch_indices: Tensor) -> Tensor:
        def prepare(index: Tensor) -> Tensor:
            return index.to(device=self._x1.device, dtype=torch.int)

        row, col, batch = prepare(row_index), prepare(col_index), [prepare(b) for b in batch_indices]
        if torch.jit.is_tracing():
            return _TracedIndex.apply(self._x1v, self._x2v, self._params, self._start, self._end, self._kid, row, col, *batch)
        return _C.index_ad(self._kid, self._x1v, self._x2v, self._params, self._start, self._end, batch, row, col)

    def _core_transpose_args(self):
        start_t, end_t = ranges.transpose_ranges(self._start, self._end, self._x1.size(-2), self._x2.size(-2))
        return self._x2, self._x1, self._params, start_t, end_t

    def _core_expand_args(self, batch_shape):
        return (
            self._x1.expand(*batch_shape, *self._x1.shape[-2:]),
            self._x2.expand(*batch_shape, *self._x2.shape[-2:]),
            self._params.expand(*batch_shape, self._params.shape[-1]),
            self._start.expand(*batch_shape, self._start.shape[-1]),
            self._end.expand(*batch_shape, self._end.shape[-1]),
        )


class KernelMatmulOperator(_OperatorCore):
    """The banded kernel matrix ``K(x1, x2; params)`` as an implicit operator (PyTorch only).

    Args:
        x1: ``(..., M, 1)``;  x2: ``(..., N, 1)``;  params: ``(..., P)``;
        start, end: ``(..., ceil(M / 128))`` int32 column ranges per row block;
        kernel_type: ``"rbf"``, ``"spectral"`` or ``"locally_periodic"``;
        symmetric: whether ``K`` is symmetric (computed from ``x1 == x2`` when ``None``).
    """

    def __init__(self, x1, x2, params, start, end, kernel_type: str | None = None,
                 symmetric: bool | None = None, compile_pool: Any = None):
        self._init_core(x1, x2, params, start, end, kernel_type, symmetric, compile_pool)

    @property
    def shape(self) -> torch.Size:
        return self._core_size()

    def size(self, dim: int | None = None):
        s = self._core_size()
        return s if dim is None else s[dim]

    @property
    def batch_shape(self) -> torch.Size:
        return self._batch_shape

    def matmul(self, rhs: Tensor) -> Tensor:
        squeeze = rhs.dim() == 1
        out = self._core_matmul(rhs.unsqueeze(-1) if squeeze else rhs)
        return out.squeeze(-1) if squeeze else out

    __matmul__ = matmul

    def to_dense(self) -> Tensor:
        return self._core_to_dense()

    def bilinear_derivative(self, left_vecs: Tensor, right_vecs: Tensor) -> Tensor:
        """Gradient wrt params of ``sum_c left[:, c]^T K right[:, c]`` -> ``(..., P)``."""
        return self._core_bilinear_derivative(left_vecs, right_vecs)

    def get_indices(self, row_index: Tensor, col_index: Tensor, *batch_indices: Tensor) -> Tensor:
        return self._core_get_indices(row_index, col_index, *batch_indices)

    def transpose(self) -> "KernelMatmulOperator":
        if self._symmetric:
            return self
        x1, x2, params, start, end = self._core_transpose_args()
        return KernelMatmulOperator(x1, x2, params, start, end, kernel_type=self._kernel_type)

    def expand_batch(self, batch_shape) -> "KernelMatmulOperator":
        return KernelMatmulOperator(*self._core_expand_args(batch_shape), kernel_type=self._kernel_type)


if HAVE_LINEAR_OPERATOR:

    class KernelMatmulLinearOperator(_OperatorCore, _LinearOperator):
        """``linear_operator.LinearOperator`` backed by the km_b200 kernels; constructor and
        hooks as in the reference (kernel_matmul/linear_operator.py:79-289)."""

        def __init__(self, x1, x2, params, start, end, kernel_type: str | None = None,
                     symmetric: bool | None = None, compile_pool: Any = None):
            _LinearOperator.__init__(
                self, x1, x2, params, start, end,
                kernel_type=kernel_type, symmetric=symmetric, compile_pool=compile_pool,
            )
            self._init_core(x1, x2, params, start, end, kernel_type, symmetric, compile_pool)

        def _matmul(self, rhs: Tensor) -> Tensor:
            return self._core_matmul(rhs)

        def _size(self) -> torch.Size:
            return self._core_size()

        def _transpose_nonbatch(self):
            if self._symmetric:
                return self
            x1, x2, params, start, end = self._core_transpose_args()
            return KernelMatmulLinearOperator(x1, x2, params, start, end, kernel_type=self._kernel_type)

        def to_dense(self) -> Tensor:
            return self._core_to_dense()

        def _expand_batch(self, batch_shape):
            return KernelMatmulLinearOperator(*self._core_expand_args(batch_shape), kernel_type=self._kernel_type)

        def to(self, *args, **kwargs):
            device, dtype = _to_helper(*args, **kwargs)
            if (device is not None and device.type != "cuda") or (dtype is not None and dtype != torch.float32):
                raise NotImplementedError("KernelMatmulLinearOperator only supports CUDA and float32")
            return super().to(*args, **kwargs)

        def type(self, dtype):
            if dtype != torch.float32:
                raise NotImplementedError("KernelMatmulLinearOperator only supports CUDA and float32")
            return super().type(dtype)

        def _bilinear_derivative(self, left_vecs: Tensor, right_vecs: Tensor):
            return None, None, self._core_bilinear_derivative(left_vecs, right_vecs), None, None

        def _get_indices(self, row_index: Tensor, col_index: Tensor, *batch_indices: Tensor) -> Tensor:
            return self._core_get_indices(row_index, col_index, *batch_indices)

else:
    KernelMatmulLinearOperator = KernelMatmulOperator
