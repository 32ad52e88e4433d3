"""``dense`` and ``index`` with their gradients at the edges of their tiles, strips and vector accesses,
against the fp64 oracle; tolerances as in ``test_ops_gpu.py``."""
import pytest
import torch

from conftest import KERNEL_TYPES, assert_grad_close, make_params, memory_left, rel_err

pytestmark = pytest.mark.gpu

TOL = 1e-5


@pytest.mark.parametrize("m,n", [(1, 1), (31, 509), (32, 510), (33, 511), (129, 512), (15, 513), (17, 1023), (145, 1026)])
def test_dense_tiles(m, n):
    """Rows that begin 0 .. 3 floats past a 16-byte boundary, ragged strips and tiles, two kernels."""
    from kernel_matmul_b200 import ops
    from oracle import oracle as O

    x1, x2 = torch.sort(torch.rand(m) * 6)[0], torch.sort(torch.rand(n) * 6)[0]
    start, end = O.make_ranges(1.5, x1, x2)
    for kt in KERNEL_TYPES:
        params = make_params(kt, (2,))
        args = [x1.expand(2, m), x2.expand(2, n), params, start.expand(2, -1), end.expand(2, -1)]
        dev = [a.cuda() for a in args]
        out, ref = ops.dense(kt, *dev), O.dense(kt, *args)
        assert rel_err(out, ref) <= TOL and torch.equal(out.cpu() != 0, ref != 0)
        og = torch.randn(2, m, n)
        term = O.dense_bwd(kt, *args, og, absolute=True)
        assert_grad_close(ops.dense_bwd(kt, *dev, og.cuda()), O.dense_bwd(kt, *args, og), term)
        # a gradient of other strides
        column_major = torch.empty_strided((2, m, n), (m * n, 1, m), device="cuda").copy_(og)
        assert_grad_close(ops.dense_bwd(kt, *dev, column_major), O.dense_bwd(kt, *args, og), term)


@pytest.mark.parametrize("batch", [(), (1,), (3,), (2, 4), (3, 3)])
@pytest.mark.parametrize("count", [1, 3, 4, 1021, 5000])
def test_gather_through_the_operator(batch, count):
    """One kernel, up to eight side by side, more; remainders of four lookups; lookups outside the band and
    index streams that are not aligned; staged ranges (5000 lookups of at most 72 ranges) or not."""
    from kernel_matmul_b200 import ops
    from kernel_matmul_b200.linear_operator import KernelMatmulOperator
    from oracle import oracle as O

    n = 900
    x = torch.sort(torch.rand(n) * 12)[0]
    start, end = O.make_ranges(1.5, x)
    for kt in KERNEL_TYPES:
        params = make_params(kt, batch)
        lead = [t.expand(*batch, -1) for t in (x, start, end)]
        row = torch.randint(0, n, (count,), dtype=torch.int32)
        col = (row + torch.randint(-300, 300, (count,), dtype=torch.int32)).clamp(0, n - 1)
        which = [torch.randint(0, s, (count,), dtype=torch.int32) for s in batch]
        w = torch.randn(count)
        oargs = (kt, lead[0], lead[0], params, lead[1], lead[2], tuple(which), row, col)
        ref, term = O.index(*oargs), O.index_bwd(*oargs, w, absolute=True)
        gref = O.index_bwd(*oargs, w)
        p = params.cuda().requires_grad_(True)
        op = KernelMatmulOperator(x.cuda()[:, None].expand(*batch, n, 1), x.cuda()[:, None].expand(*batch, n, 1), p, lead[1].cuda(),
                                  lead[2].cuda(), kernel_type=kt, symmetric=True)
        dev = [t.cuda() for t in (row, col, *which)]
        out = op.get_indices(*dev)
        assert rel_err(out, ref) <= TOL
        assert_grad_close(torch.autograd.grad(out, p, w.cuda())[0], gref, term)
        # the op itself, from index streams that begin 4 bytes past a 16-byte boundary
        shifted = [torch.cat([t[:1], t])[1:] for t in dev]
        assert all(t.data_ptr() % 16 for t in shifted)
        g = ops.index_bwd(kt, op._x1v, op._x2v, p.detach(), op._start, op._end, tuple(shifted[2:]), shifted[0], shifted[1], w.cuda())
        assert_grad_close(g, gref, term)


def test_gather_of_points_that_are_not_finite():
    """A distance that is NaN is no missing entry: values and gradients are NaN as their terms are."""
    from kernel_matmul_b200 import ranges
    from kernel_matmul_b200.linear_operator import KernelMatmulOperator

    x = torch.sort(torch.rand(300, device="cuda") * 3)[0]
    start, end = ranges.make_ranges(None, x)
    x[7] = float("nan")
    p = torch.tensor([1.0, 1.0], device="cuda", requires_grad=True)
    op = KernelMatmulOperator(x[:, None], x[:, None], p, start, end, kernel_type="rbf", symmetric=True)
    row = torch.tensor([1, 7, 3, 4, 5], dtype=torch.int32, device="cuda")
    out = op.get_indices(row, torch.zeros_like(row))
    assert out.isnan().tolist() == [False, True, False, False, False]
    assert torch.autograd.grad(out.sum(), p)[0].isnan().all()


def test_gather_without_memory_for_the_distances():
    """The values fit, the distances beside them do not: the gradient goes back to the points."""
    from kernel_matmul_b200 import ranges
    from kernel_matmul_b200.linear_operator import KernelMatmulOperator

    n, count = 3000, 1 << 24  # 64 MB of values
    x = torch.sort(torch.rand(n, device="cuda") * 30)[0]
    start, end = ranges.make_ranges(4.0, x)
    row = torch.randint(0, n, (count,), dtype=torch.int32, device="cuda")
    col = (row + torch.randint(-200, 200, (count,), dtype=torch.int32, device="cuda")).clamp_(0, n - 1)
    w = torch.randn(count, device="cuda")
    p = torch.tensor([1.0, 1.2], device="cuda", requires_grad=True)
    op = KernelMatmulOperator(x[:, None], x[:, None], p, start, end, kernel_type="rbf", symmetric=True)
    out = op.get_indices(row, col)
    want = torch.autograd.grad(out, p, w)[0]
    expected = out.detach().cpu()
    del out
    with memory_left((64 + 24) << 20):
        out = op.get_indices(row, col)
        with pytest.raises(torch.OutOfMemoryError):
            torch.empty(count, device="cuda")
        got = torch.autograd.grad(out, p, w)[0]
    assert torch.equal(out.detach().cpu(), expected)
    # (sums of 2^24 terms of either sign: fp32 within a thread's share, fp64 beyond)
    assert_grad_close(got, want, torch.full_like(want, float(w.abs().sum()) * 0.1))
