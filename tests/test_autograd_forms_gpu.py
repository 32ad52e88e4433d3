"""What the C++ autograd functions and the parameter kernel must do beyond a plain backward pass: second
derivatives, forward mode, tracing, ``torch.func``, hooks on saved tensors; compared with the same
expressions in plain PyTorch."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.fixture
def problem():
    from kernel_matmul_b200 import ranges
    from kernel_matmul_b200.linear_operator import KernelMatmulOperator

    n = 500
    x = torch.sort(torch.rand(n, device="cuda") * 5)[0]
    start, end = ranges.make_ranges(2.0, x)

    def make(params):
        return KernelMatmulOperator(x[:, None], x[:, None], params, start, end, kernel_type="rbf", symmetric=True)

    return n, make


def _expressions(module):
    return torch.stack([module.value(n) for n in module._PARAMS], dim=-1)


def _module(**kw):
    from kernel_matmul_b200 import kernels

    return kernels.SpectralKernelMatmulModule(batch_shape=torch.Size((3,)), **kw).cuda().initialize(
        lengthscale=torch.tensor([0.5, 1.0, 30.0]), frequency=torch.rand(3) + 0.1, outputscale=1.3)


def test_parameters_have_second_derivatives():
    m = _module(cutoff=1.0)
    leaves = list(m.parameters())
    grads = {}
    for name, params in (("kernel", m.params()), ("expressions", _expressions(m))):
        first = torch.autograd.grad((params**3).sum(), leaves, create_graph=True)
        second = torch.autograd.grad(sum((g**2).sum() for g in first), leaves)
        grads[name] = [*first, *second]
    for a, b in zip(grads["kernel"], grads["expressions"]):
        torch.testing.assert_close(a, b, rtol=1e-6, atol=1e-6)


def test_second_derivatives_of_parameters_that_are_not_contiguous():
    from kernel_matmul_b200 import kernels

    m = kernels.SpectralKernelMatmulModule(cutoff=1.0, batch_shape=torch.Size((2, 3))).cuda()
    for name, raw in list(m.named_parameters()):
        setattr(m, name, torch.nn.Parameter(torch.randn(3, 2, device="cuda").t()))
    leaves = list(m.parameters())
    assert not any(p.is_contiguous() for p in leaves)
    grads = {}
    for name, params in (("kernel", m.params()), ("expressions", _expressions(m))):
        first = torch.autograd.grad((params**3).sum(), leaves, create_graph=True)
        second = torch.autograd.grad(sum((g**2).sum() for g in first), leaves)
        grads[name] = [*first, *second]
    for a, b in zip(grads["kernel"], grads["expressions"]):
        torch.testing.assert_close(a, b, rtol=1e-6, atol=1e-6)


def test_parameters_under_forward_mode_vmap_and_tracing():
    import torch.autograd.forward_ad as fwAD

    m = _module(cutoff=1.0)
    names = list(dict(m.named_parameters()))
    raw = tuple(p.detach() for p in m.parameters())
    call = lambda *r: torch.func.functional_call(_Params(m), dict(zip([f"m.{n}" for n in names], r)), ())  # noqa: E731
    want = _expressions(m).detach()
    with fwAD.dual_level():
        dual = call(*(fwAD.make_dual(r, torch.ones_like(r)) for r in raw))
        tangent = fwAD.unpack_dual(dual).tangent
    assert tangent is not None and torch.equal(tangent, torch.stack([torch.sigmoid(r) for r in raw], -1)) or \
        torch.allclose(tangent, torch.stack([torch.sigmoid(r) for r in raw], -1), rtol=1e-6)
    many = torch.func.vmap(call)(*(torch.stack([r, r + 1]) for r in raw))
    assert torch.equal(many[0], want)
    traced = torch.jit.trace(_Params(m), (), check_trace=False)
    with torch.no_grad():
        for p in m.parameters():
            p.add_(0.5)
    torch.testing.assert_close(traced(), _expressions(m))


class _Params(torch.nn.Module):
    def __init__(self, m):
        super().__init__()
        self.m = m

    def forward(self):
        return self.m.params()


@pytest.mark.parametrize("epsilon", [1e-4, 0.3, 1.0])
def test_cutoff_follows_the_lengthscale_for_every_epsilon(epsilon):
    from kernel_matmul_b200 import kernels, ranges

    m = _module(epsilon=epsilon)
    x = torch.sort(torch.rand(1000, device="cuda") * 100)[0]
    op = m(x[:, None], x[:, None])
    cutoff = kernels.dynamic_cutoff(epsilon, [m.value("lengthscale")])
    start, end = ranges.make_ranges(float(cutoff), x)
    assert torch.equal(op._start[0], start) and torch.equal(op._end[0], end)


def test_forward_mode_is_refused_not_ignored(problem):
    import torch.autograd.forward_ad as fwAD

    n, make = problem
    rhs, params = torch.randn(n, 3, device="cuda"), torch.tensor([1.0, 1.0], device="cuda")
    row = torch.arange(10, device="cuda")
    with fwAD.dual_level():
        op = make(fwAD.make_dual(params, torch.ones_like(params)))
        for call in (lambda: op.matmul(rhs), op.to_dense, lambda: op.get_indices(row, row)):
            with pytest.raises((RuntimeError, NotImplementedError), match="(?i)jvp|forward"):
                call()


def test_traced_calls_run_again(problem):
    n, make = problem
    params = torch.tensor([0.8, 1.1], device="cuda")
    row = torch.arange(10, device="cuda")

    def f(p, r):
        op = make(p)
        return op.matmul(r), op.to_dense(), op.get_indices(row, row)

    traced = torch.jit.trace(f, (params, torch.randn(n, 2, device="cuda")), check_trace=False)
    p, r = torch.tensor([1.4, 0.6], device="cuda", requires_grad=True), torch.randn(n, 2, device="cuda")
    got, want = traced(p, r), f(p, r)
    for a, b in zip(got, want):
        assert torch.equal(a, b)
        ga, gb = (torch.autograd.grad(t.sum(), p, retain_graph=True)[0] for t in (a, b))
        assert torch.equal(ga, gb)


def test_saved_tensor_hooks(problem):
    n, make = problem
    params = torch.tensor([0.8, 1.1], device="cuda", requires_grad=True)
    rhs = torch.randn(n, 3, device="cuda")
    want = torch.autograd.grad(make(params).matmul(rhs).sum(), params)[0]
    with torch.autograd.graph.save_on_cpu():
        out = make(params).matmul(rhs)
    assert torch.equal(torch.autograd.grad(out.sum(), params)[0], want)
