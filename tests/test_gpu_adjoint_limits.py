"""Adjoint solves at the two limits of its extrapolation: tolerances near the
rounding of lambda, and sweep caps near what the plain iteration needs. What
the plain iteration solves has to be solved, and what it refuses refused."""
from __future__ import annotations

import numpy as np
import pytest

import knappnet_b200 as K
from test_gpu_adjoint import dense_pagerank
from test_gpu_rows import hub_graph

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")


def gradient(solve, w, target):
    v = torch.tensor(w, dtype=torch.float64, device="cuda", requires_grad=True)
    ((solve(v) - target) ** 2).sum().backward()
    return v.grad


@pytest.mark.parametrize("directed", [True, False])
@pytest.mark.parametrize("tol", [1e-14, 1e-13, 1e-12])
def test_tolerances_near_rounding(directed, tol):
    """Undirected, lambda's L1 size is about 1000, one unit in the last place of
    every node 2e-13: above the smallest tolerance."""
    from knappnet_b200 import autograd as A
    n, s, t, w = hub_graph(3, False)
    g = K.Graph(n, s, t, w, directed)
    gen = torch.Generator(device="cuda").manual_seed(1)
    for trial in range(12):
        target = torch.rand(n, dtype=torch.float64, device="cuda", generator=gen) / n
        ours = gradient(lambda v: A.pagerank(v, g, tol=tol), w, target)
        if trial < 2:
            dense = gradient(lambda v: dense_pagerank(v, s, t, n, 0.85, directed,
                                                      1.0 if directed else 2.0), w, target)
            # 12,000 terms a row within 12,000 eps = 1.3e-12, their difference
            # to lambda up to 100 times smaller, twice (forward and adjoint)
            assert float((ours - dense).abs().max()) <= 1e-9 * float(dense.abs().max())


@pytest.mark.parametrize("damping", [0.5, 0.85, 0.95])
def test_caps_near_the_plain_iteration(damping):
    from knappnet_b200 import autograd as A
    n, s, t, w = hub_graph(3, False)
    m = np.zeros((n, n))
    np.add.at(m, (s, t), np.where(s == t, 2.0, 1.0) * w)
    np.add.at(m, (t[s != t], s[s != t]), w[s != t])
    p = m / m.sum(1, keepdims=True)
    g = K.Graph(n, s, t, w, False)
    target = torch.zeros(n, dtype=torch.float64, device="cuda")
    x = A.pagerank(torch.tensor(w, dtype=torch.float64, device="cuda"), g, damping=damping,
                   tol=1e-14).cpu().numpy()
    grad_x = 2.0 * x
    lam, count, tol = grad_x, 0, 1e-9 * max(1.0, np.abs(grad_x).sum())
    while True:
        new = grad_x + damping * (p @ lam)
        count += 1
        change, lam = np.abs(new - lam).sum(), new
        if change <= tol:
            break

    def solve(cap):
        v = torch.tensor(w, dtype=torch.float64, device="cuda", requires_grad=True)
        y = A.pagerank(v, g, damping=damping, tol=1e-9, max_iter=cap)
        (y ** 2).sum().backward()

    solve(count + 1)  # x to 1e-9 instead of 1e-14 moves the count by one at most
    with pytest.raises(K.EngineError, match="adjoint did not converge"):
        solve(count - 2)
