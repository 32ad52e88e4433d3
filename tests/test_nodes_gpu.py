"""Blockwise interpolation (``csrc/km_nodes.cu``, ``csrc/km_cg_nodes.cu``) against the fp64 oracle, at the
sizes and in the forms where its kernels branch, and the direct kernels where it must step aside.

Tolerances: products 1e-5 of the largest value and gradients as in ``conftest.assert_grad_close``, the
criteria of the direct kernels; the interpolation's own error, up to 3e-8 of kappa's maximum per entry and 2.1e-7
of that of a gradient's factor (``test_nodes_cpu.py``), is below both."""
import pytest
import torch

from conftest import KERNEL_TYPES, assert_grad_close, make_params, memory_left, rel_err
from test_nodes_cpu import nodes_by_level

pytestmark = pytest.mark.gpu

TOL = 1e-5
KID = {"rbf": 0, "spectral": 1, "locally_periodic": 2}


def _both(kt, x1, x2, rhs, left, params, start, end, path="nodes", ranges=None):
    """Product and gradient on ``path`` against the oracle; CPU tensors, moved with their strides of 0 kept."""
    from kernel_matmul_b200 import ops
    from oracle import oracle as O

    def d(t):
        strided = torch.empty_strided(t.shape, t.stride(), dtype=t.dtype, device="cuda")
        if any(s == 0 for s in t.stride()):
            base = t[tuple(slice(0, 1) if s == 0 else slice(None) for s in t.stride())]
            return base.cuda().expand(t.shape)
        return strided.copy_(t)

    s, e = ranges if ranges is not None else (d(start), d(end))
    a1, a2 = d(x1), (d(x2) if x2 is not x1 else None)
    a2 = a1 if a2 is None else a2
    out = ops.matmul(kt, a1, a2, d(rhs), d(params), s, e, path=path)
    ref = O.matmul(kt, x1, x2, rhs, params, start, end)
    assert out.shape == ref.shape and rel_err(out, ref) <= TOL
    grad = ops.bilinear_derivative(kt, a1, a2, d(left), d(rhs), d(params), s, e, path=path)
    gref = O.bilinear_derivative(kt, x1, x2, left, rhs, params, start, end)
    assert_grad_close(grad, gref, O.bilinear_derivative(kt, x1, x2, left, rhs, params, start, end, absolute=True))
    return out, grad


@pytest.mark.parametrize("kt", KERNEL_TYPES)
@pytest.mark.parametrize("k", [1, 3, 4, 5, 8, 9, 16, 17, 24, 25, 33, 65])
def test_column_widths(kt, k):
    """Every chunking of the columns (4, 8, 16, 24, 32, remainders, unaligned rows)."""
    from oracle import oracle as O

    n = 129 + 128 * 5
    x = torch.sort(torch.rand(n) * 6)[0]
    start, end = O.make_ranges(2.0, x)
    _both(kt, x, x, torch.randn(n, k), torch.randn(n, k), make_params(kt, ()), start, end)


@pytest.mark.parametrize("m,n", [(1, 1), (1, 300), (127, 128), (128, 129), (257, 1), (640, 511)])
def test_ragged_blocks(m, n):
    from oracle import oracle as O

    x1, x2 = torch.sort(torch.rand(m) * 4)[0], torch.sort(torch.rand(n) * 4)[0]
    start, end = O.make_ranges(1.5, x1, x2, align=True)
    for kt in KERNEL_TYPES:
        _both(kt, x1, x2, torch.randn(n, 3), torch.randn(m, 3), make_params(kt, ()), start, end)


@pytest.mark.parametrize("spread", [0.02, 1.0, 2.5, 6.0])
def test_node_counts(spread):
    """From 4 nodes per block to more than fit (direct kernels, chosen on the device)."""
    from oracle import oracle as O

    n, k = 1000, 6
    x = torch.sort(torch.rand(n) * (spread * n / 128))[0]
    start, end = O.make_ranges(3.0 * spread, x)
    for kt in KERNEL_TYPES:
        _both(kt, x, x, torch.randn(n, k), torch.randn(n, k), make_params(kt, ()), start, end)


@pytest.mark.parametrize("form", ["shared", "own points", "shared rhs only", "two dims", "column-major rhs", "expanded rhs"])
def test_batch_forms(form):
    """Operands and points that batches share or do not, and operands of other strides."""
    from oracle import oracle as O

    n, k, batch = 700, 7, (2, 3) if form == "two dims" else (3,)
    # lengthscales of a factor of 5: several node counts on one set of points
    params = {kt: make_params(kt, batch) for kt in KERNEL_TYPES}
    for kt in KERNEL_TYPES:
        params[kt][..., 0] *= torch.tensor([1.0, 2.0, 5.0])
    own = form in ("own points", "shared rhs only")
    x = torch.sort(torch.rand(*(batch if own else ()), n) * 8)[0].expand(*batch, n)
    start, end = O.make_ranges(2.0, x[0] if not own and form != "two dims" else x.reshape(-1, n)[0])
    if own:
        start, end = O.make_ranges(2.0, x)
    start, end = start.expand(*batch, -1), end.expand(*batch, -1)
    rhs = torch.randn(*(() if form in ("shared", "shared rhs only") else batch), n, k).expand(*batch, n, k)
    if form == "column-major rhs":
        rhs = torch.randn(*batch, k, n).transpose(-1, -2)
    if form == "expanded rhs":
        rhs = torch.randn(*batch, n, 1).expand(*batch, n, k)
    for kt in KERNEL_TYPES:
        _both(kt, x, x, rhs, torch.randn(*batch, n, k), params[kt], start, end)


def _half_lengths(x):
    """Half-lengths of the 128-point blocks of (.., n) sorted points."""
    blocks = [x[..., i:i + 128] for i in range(0, x.shape[-1], 128)]
    return torch.stack([0.5 * (b[..., -1] - b[..., 0]) for b in blocks], dim=-1)


@pytest.mark.parametrize("kt,why", [("spectral", "more than eight classes"), ("locally_periodic", "more than eight classes"),
                                    ("spectral", "more nodes than there is room for")])
@pytest.mark.parametrize("shared", [True, False])
@pytest.mark.parametrize("k", [5, 20])
def test_levels_that_merge_different_classes(kt, why, shared, k):
    """Kernels that have MORE nodes on shorter intervals, because their class was merged there and not on the
    longest: what a warp stages of an operand is larger than the longest interval's nodes."""
    from oracle import oracle as O

    g = torch.Generator().manual_seed(3)
    n = 1500
    room = why == "more nodes than there is room for"
    batch = 3 if room else 16
    k = min(k, 16) if room and not shared else k
    x = torch.sort(torch.rand(*(() if shared else (batch,)), n, generator=g) * (26 if room and kt == "spectral" else 11))[0]
    halves = _half_lengths(x).reshape(-1, 12)
    longest = halves.max().item()
    levels = sum((halves <= longest / 1.15**i).long() for i in range(1, 4))
    unit, cap = (4, 160) if shared else (2, 160)
    for _ in range(4000):
        u = torch.rand(batch, 4, generator=g)
        if kt == "spectral":
            params = torch.stack([0.7 + 0.8 * u[:, 0], 2.0 + 3.0 * u[:, 1] if room else 6.0 * u[:, 1], 0.8 + u[:, 3]], dim=-1)
        else:
            params = torch.stack([0.7 + 0.8 * u[:, 0], 0.3 + u[:, 1], 0.35 + 2.0 * u[:, 2], 0.8 + u[:, 3]], dim=-1)
        nodes = nodes_by_level(kt, params, longest, unit, cap)
        if nodes.max() > (80 if k <= 16 else 64):
            continue
        at = [levels[0] if shared else levels[i] for i in range(batch)]
        hit = [i for i in range(batch) if any(nodes[i, at[i][c]] > max(nodes[i, 0], nodes[i, at[i][r]]) for r in range(12)
                                               for c in range(max(0, r - 1), min(12, r + 2)))]
        if hit:
            break
    else:
        raise AssertionError("no such parameters found")
    xe = x.expand(batch, n)
    start, end = O.make_ranges(1.2, x)
    _both(kt, xe, xe, torch.randn(n, k).expand(batch, n, k) if shared else torch.randn(batch, n, k), torch.randn(batch, n, k), params,
          start.expand(batch, -1), end.expand(batch, -1))


@pytest.mark.parametrize("case", ["band not aligned", "nan point", "points in no order", "many periods", "empty bands", "equal points"])
def test_steps_aside(case):
    """Inputs that interpolation must leave to the direct kernels, or take with an empty interval."""
    from kernel_matmul_b200 import ops
    from oracle import oracle as O

    n, k = 900, 12
    x = torch.sort(torch.rand(n) * 7)[0]
    kt, params = "spectral", make_params("spectral", ())
    start, end = O.make_ranges(2.0, x)
    if case == "band not aligned":
        start = (start + 1).clamp(max=n)
    elif case == "points in no order":
        x = x[torch.randperm(n)] * 20
        start, end = torch.zeros_like(start), torch.full_like(end, n)
    elif case == "many periods":
        params[1] = 60.0
    elif case == "empty bands":
        start, end = start.clone(), end.clone()
        end[2], start[2] = 128, 128
        start[0], end[0] = 0, 0
    elif case == "equal points":
        x[:] = 0.75
    if case == "nan point":
        x[400] = float("nan")
        args = (kt, x.cuda(), x.cuda(), torch.randn(n, k).cuda(), params.cuda(), start.cuda(), end.cuda())
        assert torch.equal(ops.matmul(*args, path="nodes").isnan(), ops.matmul(*args, path="tc").isnan())
        return
    if case == "many periods":  # the phase of a distance of 7 is 2600: one fp32 rounding of x is 3e-5 of it
        args = (kt, x.cuda(), x.cuda(), torch.randn(n, k).cuda(), params.cuda(), start.cuda(), end.cuda())
        assert torch.equal(ops.matmul(*args, path="nodes"), ops.matmul(*args, path="tc"))
        return
    _both(kt, x, x, torch.randn(n, k), torch.randn(n, k), params, start, end)


@pytest.mark.parametrize("kt", KERNEL_TYPES)
@pytest.mark.parametrize("form", ["band", "all columns"])
def test_what_ran_on_the_fma_pipe_stays_there(kt, form):
    """Up to 8 columns, gradients of up to 7, and fewer than 256 items without a cutoff: to the bit the FMA
    kernels, which hold every entry to about 1e-6 of itself."""
    from kernel_matmul_b200 import ops, ranges

    def check(n, k, grad_k, batch):
        x = torch.sort(torch.rand(n) * (n / 100))[0].cuda()
        start, end = ranges.make_ranges(2.0 if form == "band" else None, x)
        xs, params = x.expand(*batch, n), make_params(kt, batch).cuda()
        args = (params, start.expand(*batch, -1), end.expand(*batch, -1))
        rhs, left = torch.randn(n, max(k, grad_k), device="cuda"), torch.randn(n, max(k, grad_k), device="cuda")
        auto, fma = (ops.matmul(kt, xs, xs, rhs[:, :k], *args, path=p) for p in ("auto", "fma"))
        assert torch.equal(auto, fma)
        auto, fma = (ops.bilinear_derivative(kt, xs, xs, left[:, :grad_k], rhs[:, :grad_k], *args, path=p) for p in ("auto", "fma"))
        assert torch.equal(auto, fma)

    if form == "band":
        check(33000, 8, 7, (2,))  # 516 items
    else:
        check(11600, 16, 16, ())  # 91 items, 2^27 entries
        check(33000, 8, 7, ())


@pytest.mark.parametrize("batch,n,cutoff", [(600, 100, 2.0), (40, 31 * 128, 2.0), (40, 31 * 128, None)])
def test_batches_of_small_problems_are_evaluated_directly(batch, n, cutoff):
    """Whatever their number, kernels of fewer than 32 row blocks run on the tensor cores."""
    from kernel_matmul_b200 import ops, ranges

    x = torch.sort(torch.rand(n) * (n / 100))[0].cuda()
    start, end = ranges.make_ranges(cutoff, x)
    rhs, left = torch.randn(n, 16, device="cuda"), torch.randn(n, 16, device="cuda")
    args = (make_params("rbf", (batch,)).cuda(), start.expand(batch, -1), end.expand(batch, -1))
    assert torch.equal(*(ops.matmul("rbf", x, x, rhs, *args, path=p) for p in ("auto", "tc")))
    assert torch.equal(*(ops.bilinear_derivative("rbf", x, x, left, rhs, *args, path=p) for p in ("auto", "tc")))


@pytest.mark.parametrize("value", [float("inf"), float("-inf"), float("nan"), 3e38])
@pytest.mark.parametrize("k", [3, 12])
def test_operands_that_are_not_finite_or_near_overflow(value, k):
    """The direct kernels' answers, to the bit."""
    from kernel_matmul_b200 import ops, ranges

    n = 1000
    x = torch.sort(torch.rand(n) * 8)[0].cuda()
    start, end = ranges.make_ranges(2.0, x)
    rhs, left = torch.randn(n, k, device="cuda"), torch.randn(n, k, device="cuda")
    bad = rhs.clone()
    bad[500, k - 1] = value
    params = make_params("rbf", ()).cuda()
    eq = lambda a, b: torch.equal(torch.nan_to_num(a, 7.0), torch.nan_to_num(b, 7.0)) and torch.equal(a.isnan(), b.isnan())  # noqa: E731
    direct = "tc" if k >= 9 else "fma"
    assert eq(*(ops.matmul("rbf", x, x, bad, params, start, end, path=p) for p in ("nodes", direct)))
    for lr in ((bad, rhs), (left, bad)):
        assert eq(*(ops.bilinear_derivative("rbf", x, x, *lr, params, start, end, path=p) for p in ("nodes", direct)))


@pytest.mark.parametrize("m,n,order", [(300, 300, "random"), (2000, 1500, "random"), (2000, 2000, "ties"), (1500, 1500, "one point far off"),
                                       (1100, 1100, "equal"), (17000, 700, "random")])
def test_all_columns(m, n, order):
    """No cutoff: points are put in order first (or, too many in one interval of the sort, evaluated directly)."""
    from kernel_matmul_b200 import ranges

    k = 5
    x2 = torch.rand(n) * 9
    if order == "ties":
        x2 = (x2 * 16).round() / 16
    elif order == "one point far off":
        x2[77] = 1e7
    elif order == "equal":
        x2[:] = 3.0
    x1 = x2 if m == n else torch.rand(m) * 9
    s, e = ranges.make_ranges(None, x1.cuda(), x2.cuda())
    assert s.is_contiguous() and e.is_contiguous()
    for kt in KERNEL_TYPES:
        _both(kt, x1, x2, torch.randn(n, k), torch.randn(m, k), make_params(kt, ()), s.cpu(), e.cpu(), ranges=(s, e))


def test_ranges_without_cutoff_are_ordinary_tensors():
    """Every row block's range has its own memory; one that was changed is respected."""
    from kernel_matmul_b200 import ranges

    n = 1000
    x = torch.rand(n) * 9
    s, e = ranges.make_ranges(None, x.cuda())
    e[3] = 256
    s[5] = 128
    assert s.tolist() == [0, 0, 0, 0, 0, 128, 0, 0] and e.tolist() == [n, n, n, 256, n, n, n, n]
    _both("rbf", x, x, torch.randn(n, 4), torch.randn(n, 4), make_params("rbf", ()), s.cpu(), e.cpu(), ranges=(s, e))


@pytest.mark.parametrize("n", [4096, 4097, 5000])
@pytest.mark.parametrize("kt,components,width", [("rbf", 0, 100.0), ("spectral", 3, 100.0), ("spectral", 40, 60.0), ("locally_periodic", 2, 200.0)])
def test_cg_operator_laid_out_once(n, kt, components, width):
    """K v from the node matrix, P <= 16 and beyond, one and several chunks of components and columns;
    operators other than sums of spectral components with one lengthscale are evaluated."""
    from kernel_matmul_b200 import ranges
    from kernel_matmul_b200.cg import ShardedOperator

    from oracle import oracle as O

    x = torch.sort(torch.rand(n) * (n / width))[0]
    params = make_params(kt, (components,) if components else ())
    if kt == "spectral":
        params[..., 0] = 0.9
    start, end = ranges.make_ranges(3.0, x.cuda())
    op = ShardedOperator.from_kernel(kt, x.cuda(), params.cuda(), start, end, 0.1)
    assert (op.current_nodes() is not None) == (kt == "spectral") and op.current_nodes(17) is None
    B = (components,) if components else ()
    rows = torch.arange(n - 384 - n % 128, n)  # the last row blocks (the oracle takes its time)
    first = int(rows[0]) // 128
    for k in (1, 2, 3, 4, 8, 11, 16, 33):
        v = torch.randn(n, k)
        out = op.apply(v.cuda())[first * 128:]
        ref = O.matmul(kt, x[first * 128:].expand(*B, -1), x.expand(*B, n), v.expand(*B, n, k), params, start.cpu()[first:].expand(*B, -1),
                       end.cpu()[first:].expand(*B, -1))
        assert rel_err(out, (ref.sum(0) if B else ref) + 0.1 * v[first * 128:].double()) <= TOL


def test_cg_operator_follows_its_parameters():
    """An operator whose parameters were written to is laid out again; products on several streams do
    not share scratch."""
    from kernel_matmul_b200 import ranges
    from kernel_matmul_b200.cg import ShardedOperator

    n, k = 6000, 8
    x = torch.sort(torch.rand(n) * 60)[0].cuda()
    params = torch.tensor([[1.0, 0.0, 1.2], [1.0, 0.4, 0.7]], device="cuda")
    start, end = ranges.make_ranges(3.0, x)
    op = ShardedOperator.from_kernel("spectral", x, params, start, end, 0.1)
    v = torch.randn(n, k, device="cuda")
    before = op.apply(v)
    params.copy_(torch.tensor([[0.7, 0.1, 0.9], [0.7, 0.5, 0.8]]))
    fresh = ShardedOperator.from_kernel("spectral", x, params.clone(), start, end, 0.1)
    after = op.apply(v)
    assert fresh.current_nodes() is not None and torch.equal(after, fresh.apply(v)) and not torch.equal(after, before)
    params[:, 0] = 0.004  # a block spans many lengthscales: evaluated directly
    assert rel_err(op.apply(v), ShardedOperator.from_kernel("spectral", x, params, start, end, 0.1, phases=False).apply(v)) <= TOL

    vs = [torch.randn(n, k, device="cuda") for _ in range(4)]
    ref = [fresh.apply(w) for w in vs]
    torch.cuda.synchronize()
    streams = [torch.cuda.Stream() for _ in vs]
    for _ in range(20):
        got = []
        for w, st in zip(vs, streams):
            with torch.cuda.stream(st):
                got.append(fresh.apply(w))
        torch.cuda.synchronize()
        assert all(torch.equal(g, r) for g, r in zip(got, ref))


@pytest.mark.parametrize("write", ["data", "inference tensors"])
@pytest.mark.parametrize("what", ["lengthscale", "scale", "points", "wider band", "narrower band"])
@pytest.mark.parametrize("use", ["apply", "steps", "run"])
def test_cg_operator_follows_writes_that_are_not_counted(write, what, use):
    """Version counters do not tell of writes through ``.data`` nor of any to inference tensors."""
    from kernel_matmul_b200 import ranges
    from kernel_matmul_b200.cg import CGSolver, ShardedOperator

    n, k = 4500, 3

    def inputs():
        x = (torch.sort(torch.rand(n, generator=torch.Generator().manual_seed(1)))[0] * 45).cuda()
        return [x, torch.tensor([[0.6, 0.0, 1.2], [0.6, 0.4, 0.7]], device="cuda"), *ranges.make_ranges(2.4, x)]

    def change(t):
        x, params, start, end = (a.data for a in t)
        if what == "lengthscale":
            params[:, 0] = 0.5
        elif what == "scale":
            params[1, 2] = 0.9
        elif what == "points":
            x.mul_(1.01)
        else:
            s, e = ranges.make_ranges(4.0 if what == "wider band" else 1.9, x)
            start.copy_(s), end.copy_(e)

    def result(op):
        y = torch.randn(n, k, generator=torch.Generator().manual_seed(2)).cuda()
        if use == "apply":
            return op.apply(y)
        solver = CGSolver(op, y, 8)
        if use == "run":
            solver.run(8)
        else:
            for _ in range(8):
                solver.step()
        return solver.solution()

    with torch.inference_mode(write == "inference tensors"):
        t = inputs()
        op = ShardedOperator.from_kernel("spectral", *t, 0.2)
        assert op.current_nodes() is not None
        before = result(op)
        change(t)
        after = result(op)
        fresh = ShardedOperator.from_kernel("spectral", *(a.clone() for a in t), 0.2)
        assert fresh.current_nodes() is not None
        assert torch.equal(after, result(fresh)) and not torch.equal(after, before)


def _wide_system():
    """800 000 points, 16 nodes per block and bands of 20 blocks: 130 MB of node matrix, 50 MB of Lagrange matrices."""
    from kernel_matmul_b200 import ranges

    n = 800000
    x = torch.sort(torch.rand(n, device="cuda") * (n / 200))[0]
    params = torch.tensor([[1.5, 0.0, 0.6], [1.5, 2.0, 0.5]], device="cuda")
    return x, params, *ranges.make_ranges(6.0, x), torch.randn(n, 2, device="cuda")


def test_cg_operator_without_memory_for_its_matrix():
    """Evaluated, as where it is asked to be."""
    from kernel_matmul_b200.cg import ShardedOperator

    x, params, start, end, y = _wide_system()
    want = ShardedOperator.from_kernel("spectral", x, params, start, end, 0.1, phases=True).apply(y).cpu()
    with memory_left(135 << 20):  # (90 MB for the phase vectors)
        op = ShardedOperator.from_kernel("spectral", x, params, start, end, 0.1)
        assert op.current_nodes() is None and op.phase_workspace is not None
        assert torch.equal(op.apply(y).cpu(), want)
    assert ShardedOperator.from_kernel("spectral", x, params, start, end, 0.1).current_nodes() is not None


def test_cg_operator_is_laid_out_again_in_its_own_memory():
    from kernel_matmul_b200.cg import ShardedOperator

    x, params, start, end, y = _wide_system()
    op = ShardedOperator.from_kernel("spectral", x, params, start, end, 0.1)
    op.apply(y)
    with memory_left(80 << 20):
        params[1, 2] = 0.7
        again = op.apply(y)
        assert op.current_nodes() is not None
    assert torch.equal(again, ShardedOperator.from_kernel("spectral", x, params, start, end, 0.1).apply(y))


def test_cg_operators_without_points_and_before_their_layout():
    from kernel_matmul_b200 import _C, ranges
    from kernel_matmul_b200.cg import ShardedOperator

    x, params = torch.empty(0, device="cuda"), torch.tensor([[0.6, 0.0, 1.2], [0.6, 0.4, 0.7]], device="cuda")
    none = torch.empty(0, dtype=torch.int32, device="cuda")
    for p in (params, params[0]):
        op = ShardedOperator.from_kernel("spectral", x, p, none, none, 0.1)
        assert op.apply(torch.empty(0, 3, device="cuda")).shape == (0, 3)
    x = torch.sort(torch.rand(5000, device="cuda") * 50)[0]
    start, end = ranges.make_ranges(2.4, x)
    plan = _C.NodeOperator(5000, x, params, start, end, 0, start.shape[0])
    with pytest.raises(RuntimeError, match="not been laid out"):
        plan.matvec(torch.ones(5000, 1, device="cuda"), torch.empty(5000, 1, device="cuda"))


def test_cg_operator_laid_out_on_another_stream():
    """Products on a stream come after a layout that a product on another one has just made, and its memory
    outlives them."""
    from kernel_matmul_b200.cg import ShardedOperator

    x, params, start, end, y = _wide_system()
    op = ShardedOperator.from_kernel("spectral", x, params, start, end, 0.1)
    streams = [torch.cuda.Stream() for _ in range(2)]
    for scale in (0.7, 0.8, 0.9):
        params[1, 2] = scale
        for stream in streams:
            stream.wait_stream(torch.cuda.current_stream())
        got = []
        for stream in streams:  # the first lays out again
            with torch.cuda.stream(stream):
                got.append(op.apply(y))
        torch.cuda.synchronize()
        want = ShardedOperator.from_kernel("spectral", x, params, start, end, 0.1).apply(y)
        assert torch.equal(got[0], want) and torch.equal(got[1], want)


def test_plan_of_the_cg_operator_is_the_same_for_every_window():
    """Nodes and blocks by which all ranks decide whether a system is laid out."""
    from kernel_matmul_b200 import _C, ranges

    n = 6000
    x = torch.sort(torch.rand(n, device="cuda") ** 2 * 60)[0]  # denser, with wider bands, at one end
    params = torch.tensor([[0.6, 0.0, 1.2], [0.6, 0.4, 0.7]], device="cuda")
    start, end = ranges.make_ranges(2.4, x)
    R = start.shape[0]
    plans = [_C.NodeOperator(n, x, params, start, end, b, c).plan().tolist() for b, c in ((0, R), (0, R // 2), (R // 2, R - R // 2), (R, 0))]
    assert all(p[2:] == plans[0][2:] for p in plans) and plans[0][4] == int((end - start).max() + 127) // 128
    assert _C.NodeOperator(n, None, None, start, end, 0, R).plan().tolist()[:4] == plans[0][:3] + [0]


def test_band_that_becomes_wider_during_a_solve_is_not_read():
    """Products read the band that the matrix was laid out for, not the caller's tensors."""
    from kernel_matmul_b200 import ranges
    from kernel_matmul_b200.cg import CGSolver, ShardedOperator

    n, k = 4500, 3
    x = torch.sort(torch.rand(n, device="cuda") * 45)[0]
    params = torch.tensor([[0.6, 0.0, 1.2], [0.6, 0.4, 0.7]], device="cuda")
    start, end = ranges.make_ranges(2.4, x)
    y = torch.randn(n, k, device="cuda")
    ops = [ShardedOperator.from_kernel("spectral", x, params, s, e, 0.2) for s, e in ((start.clone(), end.clone()), (start, end))]
    wide = ranges.make_ranges(4.0, x)
    solvers = [CGSolver(op, y, 8) for op in ops]
    for solver in solvers:
        solver.step()
    start.data.copy_(wide[0]), end.data.copy_(wide[1])
    for solver in solvers:
        for _ in range(7):
            solver.step()
    assert torch.equal(solvers[0].solution(), solvers[1].solution())


@pytest.mark.parametrize("form", ["rbf", "spectral", "locally_periodic", "several lengthscales", "one component", "points of their own"])
@pytest.mark.parametrize("k", [8, 16])
def test_solves_of_operators_that_are_not_laid_out(form, k):
    """Iterates to the bit those of the kernels evaluated in every product, which is what CG steps leave of a
    relative accuracy of 1e-6 per entry (the node matrix has an error relative to its largest entry)."""
    from kernel_matmul_b200 import ranges
    from kernel_matmul_b200.cg import ShardedOperator, conjugate_gradient

    n, kt = 5000, form if form in KERNEL_TYPES else "spectral"
    x = (torch.sort(torch.rand(n))[0] * 50).cuda()
    batch = {"several lengthscales": (3,), "one component": (1,), "points of their own": (2,)}.get(form, ())
    if form == "points of their own":
        kt, x = "rbf", torch.stack([x, x + 0.01])
    params = make_params(kt, batch, 0.3).cuda()  # lengthscales up to 0.6: the band cuts off at 5 of them
    start, end = ranges.make_ranges(3.0, x[0] if x.dim() == 2 else x)
    y = torch.randn(n, k, device="cuda")
    solves = [conjugate_gradient(ShardedOperator.from_kernel(kt, x, params, start, end, 0.2, phases=p), y, 30) for p in (None, False)]
    assert torch.equal(solves[0].solution, solves[1].solution) and torch.equal(solves[0].residual_norms, solves[1].residual_norms)
    assert bool(solves[0].solution.isfinite().all())


def test_log_forms_on_the_device_match_the_eigenvalues():
    """Continued fraction and trapezoid rule against eigenvalues, both fp64: 1e-8 of the value, from
    systems that converge at once to condition number 1e5."""
    from kernel_matmul_b200.gp import lanczos_log_quadratic_forms

    for cond in (1.01, 50.0, 1e5):
        n, m, k = 60, 40, 3
        ev = torch.logspace(0, torch.log10(torch.tensor(cond)).item(), n, dtype=torch.float64) * 0.3
        r = torch.randn(n, k, dtype=torch.float64)
        z2 = (r * r).sum(0)
        p, rs = r.clone(), z2.clone()
        alphas, betas, norms = [], [], [torch.ones(k, dtype=torch.float64)]
        for _ in range(m):
            q = ev[:, None] * p
            a = rs / (p * q).sum(0).clamp_min(1e-300)
            r = r - a * q
            new = (r * r).sum(0)
            alphas.append(a), betas.append(new / rs), norms.append((new / z2).sqrt())
            p, rs = r + betas[-1] * p, new
        args = [torch.stack(t).float() for t in (alphas, betas, norms)] + [z2.float()]
        want = lanczos_log_quadratic_forms(*args)
        got = lanczos_log_quadratic_forms(*(a.cuda() for a in args))
        assert got.device.type == "cpu" and rel_err(got, want) <= 1e-8


@pytest.mark.parametrize("n", [65536, 65537])
def test_band_at_the_limit_of_one_launch(n):
    from kernel_matmul_b200 import ranges
    from oracle import oracle as O

    x = torch.sort(torch.rand(n) * 500)[0]
    y = torch.sort(torch.rand(n + 128) * 500)[0]
    for got, want in ((ranges.make_ranges(1.3, x.cuda()), O.make_ranges(1.3, x)),
                      (ranges.make_ranges(1.3, x.cuda(), y.cuda(), align=True), O.make_ranges(1.3, x, y, align=True))):
        assert torch.equal(got[0].cpu(), want[0]) and torch.equal(got[1].cpu(), want[1])
