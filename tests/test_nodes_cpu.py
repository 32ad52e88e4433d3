"""The rule by which blockwise interpolation chooses its nodes (``csrc/km_nodes.cuh``), restated in fp64: what
error it leaves, without the rounding of the kernels."""
import math

import pytest
import torch


def nodes_needed(kt, theta, half, eps=3e-8):
    """Smallest number of nodes the rule allows for kernel parameters ``theta`` on intervals of half-length ``half``."""
    rho = 1.1 * 2.0 ** (0.17 * torch.arange(32, dtype=torch.float64))
    b = 0.5 * half * (rho - 1 / rho)
    be = (b / theta[0]) ** 2
    log_m = 0.5 * be + torch.log1p(be)
    if kt == "spectral":
        log_m = log_m + 2 * math.pi * abs(theta[1]) * b
    if kt == "locally_periodic":
        log_m = log_m + (torch.cosh((2 * math.pi * b / theta[2]).clamp(max=300)) - 1) / theta[1]
    return math.ceil(((log_m + torch.log(4 / (rho - 1)) - math.log(eps)) / torch.log(rho)).min().item())


def nodes_by_level(kt, params, longest, unit, cap, classes=8):
    """The plan of ``csrc/km_nodes.cu``: nodes of every kernel at the four half-lengths, after each level has kept its
    largest classes and merged the others into them."""
    out = []
    for level in range(4):
        need = [max(4, -(-nodes_needed(kt, theta, longest / 1.15**level) // unit) * unit) for theta in params.double().tolist()]
        kept = []
        for p in sorted(set(need), reverse=True):
            if len(kept) == classes or sum(kept) + p > cap:
                break
            kept.append(p)
        out.append([min(q for q in kept if q >= p) for p in need])
    return torch.tensor(out).T


def _factors(kt, theta, tau):
    """kappa and the factors of its gradients."""
    ell = theta[0]
    envelope = torch.exp(-0.5 * (tau / ell) ** 2)
    if kt == "rbf":
        return envelope, [envelope * tau**2 / ell**3]
    if kt == "spectral":
        w = 2 * math.pi * theta[1]
        k = envelope * torch.cos(w * tau)
        return k, [k * tau**2 / ell**3, -envelope * torch.sin(w * tau) * 2 * math.pi * tau]
    u = math.pi * tau / theta[2]
    k = envelope * torch.exp(-2 * torch.sin(u) ** 2 / theta[1])
    return k, [k * tau**2 / ell**3, k * 2 * torch.sin(u) ** 2 / theta[1] ** 2, k * 4 * torch.sin(u) * torch.cos(u) / theta[1] * u / theta[2]]


def _lagrange(nodes, half, x):
    angle = math.pi * (2 * torch.arange(nodes, dtype=torch.float64) + 1) / (2 * nodes)
    at = half * torch.cos(angle)
    z = (-1.0) ** torch.arange(nodes) * torch.sin(angle) / (x[:, None] - at)
    return at, z / z.sum(dim=1, keepdim=True)


@pytest.mark.parametrize("kt", ["rbf", "spectral", "locally_periodic"])
def test_error_that_the_rule_leaves(kt):
    """Up to 3e-8 of kappa's maximum for an entry, 2.5e-7 of its own maximum for a factor of a gradient."""
    entry = factor = 0.0
    for _ in range(120):
        u = torch.rand(5, dtype=torch.float64).tolist()
        ell = 0.5 * 6 ** u[0]
        theta = {"rbf": [ell], "spectral": [ell, 2 * u[1]], "locally_periodic": [ell, 0.8 + 0.8 * u[1], 1.2 + 0.7 * u[2]]}[kt]
        half = 64 / (50 * 5 ** u[3]) * (1 + 0.4 * u[4])  # blocks of 128 points, 50 to 250 of them per unit
        nodes = max(4, -(-nodes_needed(kt, theta, half) // 2) * 2)
        if nodes > 80:
            continue
        x = (torch.rand(30, dtype=torch.float64) * 2 - 1) * half
        at, lam = _lagrange(nodes, half, x)
        worst, largest = [0.0] * 4, [0.0] * 4
        for distance in torch.arange(0, 4 * ell, 1.4 * half, dtype=torch.float64):
            k, grads = _factors(kt, theta, distance + x[:, None] - x[None, :])
            k_nodes, grads_nodes = _factors(kt, theta, distance + at[:, None] - at[None, :])
            for i, (f, g) in enumerate(zip([k, *grads], [k_nodes, *grads_nodes])):
                worst[i] = max(worst[i], float((f - lam @ g @ lam.T).abs().max()))
                largest[i] = max(largest[i], float(f.abs().max()))
        entry = max(entry, worst[0])
        factor = max(factor, *(w / m for w, m in zip(worst[1:], largest[1:]) if m > 0))
    assert entry <= 3e-8 and factor <= 2.5e-7, (entry, factor)
