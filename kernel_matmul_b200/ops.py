"""The native ops of the hot path, with the call signatures of the reference's per-op modules.

Each function is what ``load_native(<op>, defines).call`` is in the reference
(``native/<op>/<op>.cpp``), with the kernel type as a runtime argument instead of a
``-DKM_KERNEL_*`` define.  PyTorch is used for device memory and the current stream only;
all arithmetic runs in ``libkm_b200.so`` through its C ABI (``include/km_b200.h``).

Conventions shared with the reference: fp32 CUDA tensors, int32 ranges and indices; arbitrary
leading batch dims shared by all arguments (expanded / stride-0 views are used as they are,
never materialised); gradients are produced for ``params`` only.
"""
from __future__ import annotations

import ctypes
from typing import Sequence

import torch
from torch import Tensor

from . import _C
from ._lib import KM_MAX_BATCH_DIMS, KERNEL_TYPES, KmBatch, KmView, lib
from ._lib import check as _check

BLOCK_SIZE = 128
NUM_PARAMS = {"rbf": 2, "spectral": 3, "locally_periodic": 4}


def _kernel_id(kernel_type: str) -> int:
    try:
        return KERNEL_TYPES[kernel_type]
    except KeyError:
        raise ValueError(f"Unknown kernel type: {kernel_type}") from None


_PATHS = {"auto": 0, "fma": 1, "tc": 2, "nodes": 3}


def _path_id(path: str) -> int:
    try:
        return _PATHS[path]
    except KeyError:
        raise ValueError(f"unknown path {path!r}") from None


def _check_f32(x: Tensor) -> None:
    # native/common/entrypoint.h:3-5
    if not isinstance(x, Tensor) or not x.is_cuda:
        raise RuntimeError("x must be a CUDA tensor")
    if x.dtype != torch.float32:
        raise RuntimeError("x must be float32")


def _check_i32(x: Tensor) -> None:
    # native/common/entrypoint.h:7-14
    if not isinstance(x, Tensor) or not x.is_cuda:
        raise RuntimeError("x must be a CUDA tensor")
    if x.dtype != torch.int32:
        raise RuntimeError("x must be int32")


def _same_device(*tensors: Tensor) -> torch.device:
    dev = tensors[0].device
    for t in tensors[1:]:
        if t.device != dev:
            raise RuntimeError("all tensors must be on the same CUDA device")
    return dev


def _common_batch(tensors_nb: Sequence[tuple[Tensor, int]]) -> tuple[int, ...]:
    shapes = []
    for t, nb in tensors_nb:
        if t.dim() < nb:
            raise RuntimeError(f"tensor of rank {t.dim()} needs at least {nb} trailing dims")
        shapes.append(t.shape[: t.dim() - nb])
    try:
        return tuple(torch.broadcast_shapes(*shapes))
    except RuntimeError as exc:
        raise RuntimeError(f"batch dimensions do not broadcast: {[tuple(s) for s in shapes]}") from exc


def _expand(t: Tensor, batch: tuple[int, ...], nb: int) -> Tensor:
    core = t.shape[t.dim() - nb :]
    t = t.expand(*batch, *core)
    if len(batch) > KM_MAX_BATCH_DIMS:
        # more batch dims than the ABI carries: flatten them (copies only if not collapsible)
        t = t.reshape(-1, *core)
    return t


def _km_batch(batch: tuple[int, ...]) -> KmBatch:
    if len(batch) > KM_MAX_BATCH_DIMS:
        n = 1
        for s in batch:
            n *= s
        batch = (n,)
    b = KmBatch()
    b.ndim = len(batch)
    for d, s in enumerate(batch):
        b.size[d] = s
    return b


def _view(t: Tensor, nb: int) -> KmView:
    v = KmView()
    v.data = t.data_ptr()
    st = t.stride()
    nbatch = t.dim() - nb
    for d in range(nbatch):
        v.batch_stride[d] = st[d]
    for d in range(nb):
        v.stride[d] = st[nbatch + d]
    return v


def _stream(dev: torch.device) -> ctypes.c_void_p:
    return ctypes.c_void_p(torch.cuda.current_stream(dev).cuda_stream)


class KernelGaveUpError(RuntimeError):
    """A tensor-core kernel stopped at a hand-off wait that ran out (status word != 0).  The
    results of that launch are invalid (and NaN where the failing CTAs would have written).

    A kernel that gives up writes a word of mapped host memory (``km_take_gave_up``); every op call
    looks at the word of its device first, without waiting for anything, and raises if a launch that
    has finished since the last look gave up."""


def check(device: torch.device | int | None = None) -> None:
    """Wait for every launch made so far (on ``device``, default: all devices with a context) and
    raise ``KernelGaveUpError`` if a tensor-core launch gave up at a hand-off wait.  Op calls do the
    same check, without waiting, for the launches that have already finished."""
    if device is None:
        if not torch.cuda.is_initialized():
            return
        devices = [torch.device("cuda", i) for i in range(torch.cuda.device_count()) if torch.cuda.memory_reserved(i) > 0]
    else:
        devices = [torch.device("cuda", device) if isinstance(device, int) else torch.device(device)]
    for d in devices:
        torch.cuda.synchronize(d)
        _C.poll_gave_up(d.index if d.index is not None else torch.cuda.current_device())


#: rhs widths from which ``matmul`` runs the contraction on the tensor cores (tcgen05; fp16
#: hi/lo operand split, kernel tiles handed over in tensor memory).  The cost of that kernel
#: hardly depends on the width; below 9 columns the FMA pipe is as fast.
TENSOR_CORE_MIN_K = _C.TENSOR_CORE_MIN_K
#: The tensor-core kernels run a pre-pass over the rhs (two or three small launches); they are
#: chosen on ``path="auto"`` only for problems with at least this many (batch, row block) items.
TENSOR_CORE_MIN_ITEMS = _C.TENSOR_CORE_MIN_ITEMS
#: column count from which the gradient ops take the tensor-core kernel on ``path="auto"``
#: (if the problem has ``TENSOR_CORE_MIN_ITEMS`` work items)
GRAD_TENSOR_CORE_MIN_K = _C.GRAD_TENSOR_CORE_MIN_K


def _is_cuda(*tensors: Tensor) -> None:
    for t in tensors:
        if not isinstance(t, Tensor):
            raise RuntimeError("x must be a CUDA tensor")


def matmul(kernel_type: str, x1: Tensor, x2: Tensor, rhs: Tensor, params: Tensor, start: Tensor, end: Tensor,
           *, path: str = "auto") -> Tensor:
    """``K(x1, x2; params)[masked by ranges] @ rhs`` -> ``(*batch, m, k)``.

    Reference: ``matmul.call(x1, x2, rhs, params, start, end)`` (native/matmul/matmul.cpp:6-17).
    ``path``: ``"fma"`` (FP32 pipe), ``"tc"`` (tensor cores; fp32-level accuracy through operand
    splitting) or ``"auto"`` (tensor cores from ``TENSOR_CORE_MIN_K`` rhs columns, if the problem
    has ``TENSOR_CORE_MIN_ITEMS`` work items).
    """
    kid = _kernel_id(kernel_type)
    _is_cuda(x1, x2, rhs, params, start, end)
    out, tc = _C.op_matmul(kid, x1, x2, rhs, params, start, end, _path_id(path))
    if tc:
        out._km_tensor_cores = True
    return out


def used_tensor_cores(result: Tensor) -> bool:
    """Whether the op call that returned ``result`` ran its tensor-core kernel."""
    return bool(getattr(result, "_km_tensor_cores", False))


def tc_status(out: Tensor) -> int:
    """1 if a tensor-core launch on ``out``'s device has given up since the last check, else 0
    (synchronises the device's launches; kept for callers that poll instead of catching
    ``KernelGaveUpError`` from ``check``)."""
    try:
        check(out.device)
    except KernelGaveUpError:
        return 1
    return 0


def prepare_sum_phases(kernel_type: str, x1: Tensor, x2: Tensor, params: Tensor, *, rows: tuple[int, int] | None = None,
                       cols: tuple[int, int] | None = None) -> Tensor | None:
    """Phase images for the batch sum of spectral components (``km_sum_phases_prepare_f32``): the
    per-point vectors ``(cos, sin)(2 pi f_b x)`` of all rows and columns, written once per operator
    in the layouts the tensor-core kernel takes them.  Pass the returned workspace to
    ``matmul_rows(..., sum_batches=True, phases=...)``: products with the same ``x1``, ``x2`` and
    ``params`` (frequencies and output scales; one common lengthscale) then copy the vectors instead
    of evaluating them again for every row block.  ``None`` where it does not apply (another kernel
    type, fewer than 2 or more than 1024 components); ``x1`` / ``x2`` of shape ``(m,)`` / ``(n,)``.
    ``rows`` / ``cols``: write only these rows and columns (what the products of one rank of a
    row-sharded solve read: its own rows and the columns of their bands)."""
    if kernel_type != "spectral" or params.dim() < 2:
        return None
    batch = tuple(params.shape[:-1])
    comps = 1
    for b in batch:
        comps *= int(b)
    if comps < 2 or comps > 1024 or len(batch) > KM_MAX_BATCH_DIMS:
        return None
    if x1.dim() != 1 or x2.dim() != 1:
        raise RuntimeError("prepare_sum_phases takes the shared inputs x1 (m,) and x2 (n,)")
    if params.shape[-1] != NUM_PARAMS[kernel_type]:
        raise RuntimeError(f"params must have {NUM_PARAMS[kernel_type]} entries in the last dim")
    for t in (x1, x2, params):
        _check_f32(t)
    dev = _same_device(x1, x2, params)
    m, n = x1.shape[0], x2.shape[0]
    x1e, x2e = x1.expand(*batch, m), x2.expand(*batch, n)
    kb = _km_batch(batch)
    nbytes = int(lib.km_sum_phases_workspace_bytes(kb, m, n))
    raw = torch.empty(max(nbytes, 256) + 256, dtype=torch.uint8, device=dev)
    ws = raw[(-raw.data_ptr()) % 256:][:max(nbytes, 256)]
    with torch.cuda.device(dev):
        r0, r1 = rows if rows is not None else (0, m)
        c0, c1 = cols if cols is not None else (0, n)
        _check(lib.km_sum_phases_prepare_f32(kb, m, n, _view(x1e, 1), _view(x2e, 1), _view(params, 1), r0, r1, c0, c1,
                                             ctypes.c_void_p(ws.data_ptr()), ws.numel(), _stream(dev)))
    return ws


def matmul_rows(kernel_type: str, x1: Tensor, x2: Tensor, rhs: Tensor, params: Tensor, start: Tensor, end: Tensor,
                *, row_block_begin: int = 0, row_block_count: int | None = None, sum_batches: bool = False,
                out: Tensor | None = None, path: str = "auto", phases: Tensor | None = None) -> Tensor:
    """``matmul`` restricted to the row blocks ``[row_block_begin, row_block_begin + row_block_count)``
    and, with ``sum_batches``, summed over all batch dims inside the kernel.

    Returns ``(*batch, rows, k)`` or, with ``sum_batches``, ``(rows, k)``, where ``rows`` is the
    number of rows of ``x1`` inside the window.  ``out`` may be passed to receive the result
    (e.g. a rank's slice of an all-gather buffer).  ``path`` as in ``matmul`` (the batch sum runs
    on the FMA pipe).  ``phases``: the workspace of ``prepare_sum_phases`` for this operator (batch
    sum only).
    """
    call = _rows_product(kernel_type, x1, x2, rhs, params, start, end, row_block_begin, row_block_count, sum_batches, out, path, phases)
    call()
    if call.tensor_cores:
        call.out._km_tensor_cores = True
    return call.out


def _rows_product(kernel_type, x1, x2, rhs, params, start, end, row_block_begin, row_block_count, sum_batches, out, path, phases):
    kid = _kernel_id(kernel_type)
    _is_cuda(x1, x2, rhs, params, start, end)
    count = -1 if row_block_count is None else row_block_count
    if row_block_count is not None and row_block_count < 0:
        raise RuntimeError(f"negative row-block count {row_block_count}")
    return _C.RowsProduct(kid, x1, x2, rhs, params, start, end, row_block_begin, count, sum_batches, out, _path_id(path), phases)


#: ``matmul_rows`` with everything but the launch done once: arguments validated, the C structures
#: filled, a workspace kept.  For loops that call the same product on the same buffers many times (a
#: CG solve: ``rhs`` and ``out`` are fixed buffers whose CONTENTS change); a call is one launch on the
#: current stream.
PreparedRowsProduct = _C.RowsProduct


def prepare_matmul_rows(kernel_type: str, x1: Tensor, x2: Tensor, rhs: Tensor, params: Tensor, start: Tensor, end: Tensor,
                        *, row_block_begin: int, row_block_count: int, sum_batches: bool, out: Tensor,
                        phases: Tensor | None = None) -> PreparedRowsProduct:
    """A ``PreparedRowsProduct`` that computes what ``matmul_rows(..., out=out)`` computes.  The
    tensors stay alive with it; their contents may change between calls."""
    return _rows_product(kernel_type, x1, x2, rhs, params, start, end, row_block_begin, row_block_count, sum_batches, out, "auto", phases)


def _grad_call(kernel_type, x1, x2, left, right, params, start, end, path: str) -> Tensor:
    kid = _kernel_id(kernel_type)
    _is_cuda(x1, x2, left, right, params, start, end)
    grad, tc = _C.op_bilinear(kid, x1, x2, left, right, params, start, end, _path_id(path))
    if tc:
        grad._km_tensor_cores = True
    return grad


def matmul_bwd(kernel_type: str, x1, x2, rhs, params, start, end, out_grad, *, path: str = "auto") -> Tensor:
    """Gradient of ``sum(out_grad * matmul(...))`` wrt ``params`` -> ``(*batch, P)``.

    Reference: ``matmul_bwd.call(x1, x2, rhs, params, start, end, out_grad)``
    (native/matmul_bwd/matmul_bwd.cpp:6-19).  ``path`` as in ``matmul``.
    """
    return _grad_call(kernel_type, x1, x2, out_grad, rhs, params, start, end, path)


def bilinear_derivative(kernel_type: str, x1, x2, left_vecs, right_vecs, params, start, end, *,
                        path: str = "auto") -> Tensor:
    """Gradient of ``sum_c left[:, c]^T K right[:, c]`` wrt ``params`` -> ``(*batch, P)``.

    Reference: ``bilinear_derivative.call(x1, x2, left_vecs, right_vecs, params, start, end)``
    (native/bilinear_derivative/bilinear_derivative.cpp:6-21).
    """
    return _grad_call(kernel_type, x1, x2, left_vecs, right_vecs, params, start, end, path)


def dense(kernel_type: str, x1, x2, params, start, end) -> Tensor:
    """Masked dense ``K`` -> ``(*batch, m, n)``.  Reference: ``dense.call`` (native/dense/dense.cpp:6-17)."""
    kid = _kernel_id(kernel_type)
    _is_cuda(x1, x2, params, start, end)
    return _C.dense(kid, x1, x2, params, start, end)


def dense_bwd(kernel_type: str, x1, x2, params, start, end, out_grad) -> Tensor:
    """Gradient of ``sum(out_grad * dense(...))`` wrt ``params``.  Reference: ``dense_bwd.call``
    (native/dense_bwd/dense_bwd.cpp:6-17)."""
    kid = _kernel_id(kernel_type)
    _is_cuda(x1, x2, params, start, end, out_grad)
    return _C.dense_bwd(kid, x1, x2, params, start, end, out_grad)


def index(kernel_type: str, x1, x2, params, start, end, batch_indices, row_index, col_index) -> Tensor:
    """``K[batch_indices..., row_index, col_index]`` (0 outside the band) with the shape of the
    index tensors.  Reference: ``index.call`` (native/index/index.cpp:6-24)."""
    kid = _kernel_id(kernel_type)
    _is_cuda(x1, x2, params, start, end, row_index, col_index)
    return _C.index(kid, x1, x2, params, start, end, list(batch_indices), row_index, col_index)


def index_bwd(kernel_type: str, x1, x2, params, start, end, batch_indices, row_index, col_index, out_grad) -> Tensor:
    """Gradient of ``sum(out_grad * index(...))`` wrt ``params`` -> ``(*batch, P)``.
    Reference: ``index_bwd.call`` (native/index_bwd/index_bwd.cpp:6-27)."""
    kid = _kernel_id(kernel_type)
    _is_cuda(x1, x2, params, start, end, row_index, col_index, out_grad)
    return _C.index_bwd(kid, x1, x2, params, start, end, list(batch_indices), row_index, col_index, out_grad)


def count_entries(m: int, n: int, start: Tensor, end: Tensor) -> Tensor:
    """Visited kernel entries ``sum rows(r) * (end - start)`` as a 0-dim int64 device tensor."""
    _check_i32(start)
    _check_i32(end)
    dev = _same_device(start, end)
    batch = _common_batch([(start, 1), (end, 1)])
    se, ee = _expand(start, batch, 1), _expand(end, batch, 1)
    out = torch.empty((), device=dev, dtype=torch.int64)
    with torch.cuda.device(dev):
        _check(lib.km_count_entries(_km_batch(batch), m, n, _view(se, 1), _view(ee, 1),
                                   ctypes.c_void_p(out.data_ptr()), _stream(dev)))
    return out


__all__ = [
    "matmul", "matmul_rows", "prepare_matmul_rows", "PreparedRowsProduct", "tc_status", "check", "used_tensor_cores", "KernelGaveUpError", "matmul_bwd", "bilinear_derivative", "dense", "dense_bwd", "index", "index_bwd",
    "count_entries", "BLOCK_SIZE", "NUM_PARAMS",
]
