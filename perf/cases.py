"""What a user of kernel_matmul_b200 has it do, as cases to time and compare.

A case is a dict of plain values with a ``"kind"``:

``product``   ``KernelMatmulOperator.matmul`` on a kept operator, with ``grad`` also the gradient of
              the result with respect to the kernel parameters (``matmul`` / ``matmul_bwd``)
``train``     one training step of a kernel module: parameters -> band -> operator -> product ->
              gradients of the raw parameters
``predict``   a kernel module called on test and training points (a rectangular matrix), its
              product with a few weight columns, and the transposed product
``bilinear``  ``KernelMatmulOperator.bilinear_derivative``
``dense``     ``KernelMatmulOperator.to_dense`` and its gradient
``gather``    ``KernelMatmulOperator.get_indices`` and its gradient
``solve``     band, row-sharded operator over a sum of spectral components and a CG solve
``mll``       ``gp.mll_gradient``: value and gradient of the marginal likelihood

Inputs are uniform points, sorted where there is a cutoff, at 50 to 250 points per unit (the density of the benchmark
configurations), lengthscales around one and a cutoff of about four lengthscales, as in the
repository's workloads and tests.  All values are fp32: the library has no other type.
"""
from __future__ import annotations

import math

import torch

from kernel_matmul_b200 import gp, kernels, ranges
from kernel_matmul_b200.cg import ShardedOperator, conjugate_gradient
from kernel_matmul_b200.linear_operator import KernelMatmulOperator

BLOCK = 128
MODULES = {
    "rbf": kernels.RBFKernelMatmulModule,
    "spectral": kernels.SpectralKernelMatmulModule,
    "locally_periodic": kernels.LocallyPeriodicKernelMatmulModule,
}


def listed():
    return [
        # One vector through a small banded RBF kernel: the step of any iterative method on a data set
        # of a few thousand points.  Launch and host time are all there is.
        dict(name="product_small", kind="product", kernel="rbf", batch=0, n=4096, k=1, per_unit=102.4, ell=0.5, ell_ratio=1.0,
             cutoff=4.0, grad=False),
        # A training step of a two-component spectral module on 3000 points, the size of the module tests,
        # with the cutoff that follows the learnt lengthscale.
        dict(name="train_small", kind="train", kernel="spectral", batch=2, n=3000, k=16, per_unit=30.0, ell=1.0, epsilon=1e-4),
        # A training step of one kernel on 20 000 points with 1 + 10 columns (target and probes): the
        # middle of the range, an odd width.
        dict(name="train_medium", kind="train", kernel="locally_periodic", batch=0, n=20011, k=11, per_unit=100.0, ell=1.5,
             epsilon=1e-4),
        # Predictive mean and its adjoint at 5003 test points from 50 021 training points: rectangular,
        # ragged, two columns.
        dict(name="predict", kind="predict", kernel="spectral", batch=3, m=5003, n=50021, k=2, per_unit=100.0, ell=1.0, cutoff=4.0),
        # Spectral mixture with 16 components of their own lengthscales and bands: product and gradient.
        dict(name="spectral_mixture", kind="product", kernel="spectral", batch=16, n=65536, k=16, per_unit=131.072, ell=0.5,
             ell_ratio=10.0, cutoff=4.0, grad=True),
        # The same for a wide odd number of columns and an RBF batch of three.
        dict(name="product_wide_ragged", kind="product", kernel="rbf", batch=3, n=50021, k=65, per_unit=100.0, ell=1.0, ell_ratio=2.0,
             cutoff=4.0, grad=True),
        # Every entry of a large RBF kernel (no cutoff) against 128 columns.
        dict(name="product_unbanded", kind="product", kernel="rbf", batch=0, n=131072, k=128, per_unit=1310.72, ell=2.0,
             ell_ratio=1.0, cutoff=0.0, grad=False),
        # Gradient of a quadratic form from solved vectors, 32 columns, four locally periodic kernels.
        dict(name="bilinear", kind="bilinear", kernel="locally_periodic", batch=4, n=262144, k=32, per_unit=131.072, ell=3.0,
             cutoff=4.0),
        # The matrix itself, as preconditioners, diagnostics and exact small-scale solves take it.
        dict(name="dense", kind="dense", kernel="spectral", batch=3, m=6007, n=6007, per_unit=100.0, ell=1.0, cutoff=4.0),
        # Single entries by index, as pivoted Cholesky and sampling take them, and the gradient of a sum of them.
        dict(name="gather", kind="gather", kernel="rbf", batch=0, n=131072, lookups=1 << 24, per_unit=1310.72, ell=2.0, cutoff=0.0),
        # Marginal likelihood and gradient of a Gaussian process with 20 000 points: 15 probes, 100 CG steps.
        dict(name="mll", kind="mll", kernel="rbf", n=20000, probes=15, iterations=100, per_unit=100.0, ell=0.5, sigma2=0.2,
             cutoff=4.0),
        # CG steps of a sum of 64 spectral components on 4 million points, 8 right-hand sides: the largest.
        dict(name="solve", kind="solve", batch=64, n=1 << 22, k=8, iterations=20, per_unit=209.7152, ell=1.5, sigma2=0.01, cutoff=4.0),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["product", "product", "train", "predict", "bilinear", "dense", "gather", "mll", "solve"])
    kernel = rng.choice(["rbf", "spectral", "locally_periodic"])
    per_unit = round(rng.uniform(50.0, 250.0), 3)
    ell = round(math.exp(rng.uniform(math.log(0.5), math.log(3.0))), 4)
    batch = rng.choice([0, 0, 2, 3, 4, 8, 16])
    if kind == "product":
        if rng.random() < 0.2:  # every entry, no cutoff
            return dict(kind=kind, kernel=kernel, batch=0, n=_log_int(rng, 1000, 60000), k=_log_int(rng, 1, 128),
                        per_unit=round(per_unit * 4, 3), ell=ell, ell_ratio=1.0, cutoff=0.0, grad=rng.random() < 0.5)
        return dict(kind=kind, kernel=kernel, batch=batch, n=_log_int(rng, 1000, 131072), k=_log_int(rng, 1, 128), per_unit=per_unit,
                    ell=ell, ell_ratio=rng.choice([1.0, 2.0]), cutoff=4.0, grad=rng.random() < 0.6)
    if kind == "train":
        return dict(kind=kind, kernel=kernel, batch=rng.choice([0, 2, 3]), n=_log_int(rng, 1000, 50000), k=_log_int(rng, 1, 32),
                    per_unit=per_unit, ell=ell, epsilon=1e-4)
    if kind == "predict":
        return dict(kind=kind, kernel=kernel, batch=rng.choice([0, 2, 3]), m=_log_int(rng, 300, 20000), n=_log_int(rng, 2000, 131072),
                    k=rng.choice([1, 2, 3]), per_unit=per_unit, ell=ell, cutoff=4.0)
    if kind == "bilinear":
        return dict(kind=kind, kernel=kernel, batch=rng.choice([0, 2, 4]), n=_log_int(rng, 4000, 262144), k=_log_int(rng, 4, 64),
                    per_unit=per_unit, ell=ell, cutoff=4.0)
    if kind == "dense":
        return dict(kind=kind, kernel=kernel, batch=rng.choice([0, 2, 3]), m=_log_int(rng, 500, 8000), n=_log_int(rng, 500, 8000),
                    per_unit=per_unit, ell=ell, cutoff=4.0)
    if kind == "gather":
        return dict(kind=kind, kernel=kernel, batch=rng.choice([0, 3]), n=_log_int(rng, 2000, 131072), lookups=_log_int(rng, 1 << 12, 1 << 24),
                    per_unit=per_unit, ell=ell, cutoff=rng.choice([0.0, 4.0]))
    if kind == "mll":
        return dict(kind=kind, kernel=rng.choice(["rbf", "spectral"]), n=_log_int(rng, 2000, 60000), probes=rng.choice([7, 10, 15]),
                    iterations=rng.choice([50, 100]), per_unit=round(rng.uniform(50.0, 120.0), 3), ell=round(rng.uniform(0.4, 0.8), 4),
                    sigma2=0.2, cutoff=4.0)
    return dict(kind=kind, batch=rng.choice([4, 16, 64]), n=_log_int(rng, 100000, 1 << 22), k=rng.choice([1, 4, 8, 11]), iterations=10,
                per_unit=per_unit, ell=1.5, sigma2=0.01, cutoff=4.0)


def _points(g, n, per_unit, ordered=True):
    x = torch.rand(n, generator=g, device="cuda") * (n / per_unit)
    return torch.sort(x)[0] if ordered else x


def _spread(g, batch, lo, hi):
    shape = (batch,) if batch else ()
    return lo + (hi - lo) * torch.rand(shape, generator=g, device="cuda")


def _values(g, kernel, batch, ell, ratio=1.0):
    """Kernel parameters in native order, by name: lengthscales in [ell, ell * ratio]."""
    first = ell * ratio ** _spread(g, batch, 0.0, 1.0)
    if kernel == "rbf":
        return dict(lengthscale=first, outputscale=_spread(g, batch, 0.8, 1.2))
    if kernel == "spectral":
        return dict(lengthscale=first, frequency=_spread(g, batch, 0.0, 2.0), outputscale=_spread(g, batch, 0.8, 1.2))
    return dict(lengthscale_rbf=first, lengthscale_periodic=_spread(g, batch, 0.8, 1.6), period_length=_spread(g, batch, 1.2, 1.9),
                outputscale=_spread(g, batch, 0.8, 1.2))


def _operator(g, case, x):
    """A kept operator on the points ``x``: parameters, band of four lengthscales per component."""
    batch = case["batch"]
    values = list(_values(g, case["kernel"], batch, case["ell"], case.get("ell_ratio", 1.0)).values())
    params = torch.stack(values, dim=-1)
    if case["cutoff"] == 0.0:
        start, end = ranges.make_ranges(None, x)
        if batch:
            start, end = start.expand(batch, -1), end.expand(batch, -1)
    elif batch:
        start, end = ranges.make_ranges_symmetric_cutoffs(case["cutoff"] * values[0], x)
    else:
        start, end = ranges.make_ranges(case["cutoff"] * float(values[0]), x)
    params.requires_grad_(bool(case.get("grad", True)))
    xs = x.unsqueeze(-1)
    return KernelMatmulOperator(xs, xs, params, start, end, kernel_type=case["kernel"], symmetric=True), params


def prepare(case, seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    kind = case["kind"]
    normal = lambda *shape: torch.randn(*shape, generator=g, device="cuda")  # noqa: E731
    lead = (case["batch"],) if case.get("batch") else ()
    s = dict(case)
    if kind in ("product", "bilinear", "dense", "gather"):
        n = case["n"]
        if kind == "dense" and case["m"] != n:
            x1 = torch.sort(torch.rand(case["m"], generator=g, device="cuda") * (n / case["per_unit"]))[0]
            x2 = _points(g, n, case["per_unit"])
            values = list(_values(g, case["kernel"], case["batch"], case["ell"]).values())
            s["params"] = torch.stack(values, dim=-1).requires_grad_(True)
            start, end = ranges.make_ranges(case["cutoff"] * case["ell"], x1, x2, align=True)
            s["op"] = KernelMatmulOperator(x1.unsqueeze(-1), x2.unsqueeze(-1), s["params"], start, end, kernel_type=case["kernel"],
                                           symmetric=False)
        else:
            s["op"], s["params"] = _operator(g, case, _points(g, n, case["per_unit"], case["cutoff"] != 0.0))
    if kind == "product":
        s["rhs"] = normal(n, case["k"])  # one right-hand side for all components
        if case["grad"]:
            s["out_grad"] = normal(*lead, n, case["k"])
    elif kind == "bilinear":
        s["params"].requires_grad_(False)
        s["left"], s["right"] = normal(*lead, n, case["k"]), normal(*lead, n, case["k"])
    elif kind == "dense":
        s["out_grad"] = normal(*lead, case["m"], n)
    elif kind == "gather":
        count = case["lookups"]
        whole = lambda top: torch.randint(0, top, (count,), generator=g, device="cuda", dtype=torch.int32)  # noqa: E731
        s["row"] = whole(n)
        # with a band, lookups near the diagonal (elsewhere the matrix is zero)
        s["col"] = whole(n) if case["cutoff"] == 0.0 else ((s["row"] + whole(2 * BLOCK + 1) - BLOCK).clamp_(0, n - 1))
        s["which"] = (whole(case["batch"]),) if case["batch"] else ()
        s["out_grad"] = normal(count)
    elif kind == "train":
        module = MODULES[case["kernel"]](epsilon=case["epsilon"], batch_shape=lead).cuda()
        s["module"] = module.initialize(**_values(g, case["kernel"], case["batch"], case["ell"]))
        s["x"] = _points(g, case["n"], case["per_unit"]).unsqueeze(-1)
        s["rhs"] = normal(case["n"], case["k"])
        s["out_grad"] = normal(*lead, case["n"], case["k"])
    elif kind == "predict":
        module = MODULES[case["kernel"]](cutoff=case["cutoff"] * case["ell"], batch_shape=lead).cuda()
        s["module"] = module.initialize(**_values(g, case["kernel"], case["batch"], case["ell"]))
        s["x"] = _points(g, case["n"], case["per_unit"]).unsqueeze(-1)
        s["x_test"] = torch.sort(torch.rand(case["m"], generator=g, device="cuda") * (case["n"] / case["per_unit"]))[0].unsqueeze(-1)
        s["weights"], s["back"] = normal(case["n"], case["k"]), normal(case["m"], case["k"])
    elif kind == "mll":
        s["x"] = _points(g, case["n"], case["per_unit"])
        v = _values(g, case["kernel"], 0, case["ell"])
        s["params"] = torch.stack(list(v.values()))
        s["y"] = torch.sin(2.0 * s["x"]) + math.sqrt(case["sigma2"]) * normal(case["n"])
        s["signs"] = torch.randint(0, 2, (case["n"], case["probes"]), generator=g, device="cuda").float() * 2.0 - 1.0
    elif kind == "solve":
        B = case["batch"]
        s["x"] = _points(g, case["n"], case["per_unit"])
        f = torch.rand(B, generator=g, device="cuda")
        f[0] = 0.0  # the plain RBF term
        s["params"] = torch.stack([torch.full_like(f, case["ell"]), f, torch.full_like(f, 1.0 / B)], dim=-1)
        s["y"] = normal(case["n"], case["k"])
    return s


def run(s):
    kind = s["kind"]
    if kind == "product":
        out = s["op"].matmul(s["rhs"])
        if not s["grad"]:
            return out
        return out.detach(), torch.autograd.grad(out, s["params"], s["out_grad"])[0]
    if kind == "train":
        op = s["module"](s["x"], s["x"])
        out = op.matmul(s["rhs"])
        grads = torch.autograd.grad(out, list(s["module"].parameters()), s["out_grad"])
        return (out.detach(), *grads)
    if kind == "predict":
        with torch.no_grad():
            op = s["module"](s["x_test"], s["x"])
            return op.matmul(s["weights"]), op.transpose().matmul(s["back"])
    if kind == "bilinear":
        return s["op"].bilinear_derivative(s["left"], s["right"])
    if kind == "dense":
        out = s["op"].to_dense()
        return out.detach(), torch.autograd.grad(out, s["params"], s["out_grad"])[0]
    if kind == "gather":
        out = s["op"].get_indices(s["row"], s["col"], *s["which"])
        return out.detach(), torch.autograd.grad(out, s["params"], s["out_grad"])[0]
    if kind == "mll":
        r = gp.mll_gradient(s["kernel"], s["x"], s["params"], s["sigma2"], s["y"], cutoff=s["cutoff"] * s["ell"], probes=s["signs"],
                            cg_iterations=s["iterations"])
        return r.grad_params, r.grad_sigma2, r.inv_quad, r.logdet, r.nll, r.solve, r.probe_solves, r.residual_norms
    start, end = ranges.make_ranges(s["cutoff"] * s["ell"], s["x"])
    op = ShardedOperator.from_kernel("spectral", s["x"], s["params"], start, end, s["sigma2"])
    r = conjugate_gradient(op, s["y"], s["iterations"])
    return r.solution, r.residual_norms


def _entries(case):
    """Kernel entries inside the bands of all components: per row block its own extent, the cutoff
    on both sides and, as ends are rounded to blocks, about a block."""
    m, n = case.get("m", case["n"]), case["n"]
    components = max(1, case.get("batch", 0))
    if case.get("cutoff") == 0.0:
        return float(components) * m * n
    ratio = case.get("ell_ratio", 1.0)
    ell = case["ell"] * ((ratio - 1.0) / math.log(ratio) if ratio > 1.0 else 1.0)  # mean of the log-uniform lengthscales
    reach = case.get("cutoff", 3.89)  # epsilon 1e-4: sqrt(2) erfinv(1 - epsilon) lengthscales
    rows_extent = BLOCK * n / m  # columns beside the rows of one block
    return float(components) * m * min(float(n), 2.0 * reach * ell * case["per_unit"] + rows_extent + BLOCK)


def work(case):
    kind = case["kind"]
    entries, components = _entries(case), max(1, case.get("batch", 0))
    n, k = case["n"], case.get("k", 1)
    m = case.get("m", n)
    if kind in ("product", "train"):
        passes = 2 if case.get("grad", True) else 1  # the gradient reads out_grad and rhs, and writes a few values
        return {"bytes": 4.0 * (n * (1 + k) + passes * components * m * k), "flops": passes * entries * (2.0 * k + 8.0)}
    if kind == "predict":
        return {"bytes": 4.0 * ((n + m) * (1 + k) + components * (n + m) * k), "flops": 2.0 * entries * (2.0 * k + 8.0)}
    if kind == "bilinear":
        return {"bytes": 4.0 * (n + 2.0 * components * n * k), "flops": entries * (2.0 * k + 8.0)}
    if kind == "dense":  # the matrix is written; of its gradient only the band is read
        return {"bytes": 4.0 * (components * m * n + entries + m + n), "flops": 24.0 * entries}
    if kind == "gather":  # indices read and values written, indices and the gradient read
        index = 4.0 * (3 if case["batch"] else 2)
        return {"bytes": case["lookups"] * 2.0 * (index + 4.0) + 4.0 * n, "flops": 24.0 * case["lookups"]}
    if kind == "mll":  # each step: products with the directions, three vectors read and written; then the gradient
        k = 1 + case["probes"]
        steps = case["iterations"]
        return {"bytes": 4.0 * n * (steps * 7.0 * k + 3.0 * k), "flops": (steps + 1.0) * entries * (2.0 * k + 8.0)}
    # solve: the entries of the sum of all components; x, r, p and K p once each per step
    return {"bytes": case["iterations"] * 4.0 * n * 7.0 * k, "flops": case["iterations"] * (entries * 4.0 + entries / components * 2.0 * k)}


def tolerance(case):
    if case["kind"] in ("mll", "solve"):
        # tens of CG steps on a system of condition number about a thousand: a relative error of 1e-6
        # in the products, or in the right-hand side, comes back up to thirty times larger
        return {"rel": 2e-4, "max": 5e-3}
    # sums of fp32 products; the gradients among the outputs are sums of terms of either sign that
    # largely cancel (a sum of N of them is about sqrt(N) terms large)
    return {"rel": 2e-5, "max": 5e-4}
