"""Set-up passes over an adjacency (strengths, arc values with loop factors,
out-strengths, edge gradients) at the row lengths where their work is split
differently: one thread per row up to 64 arcs, a CTA per row above."""
from __future__ import annotations

import numpy as np
import pytest

import knappnet_b200 as K
from oracle import oracle as O
from test_gpu_adjoint import dense_pagerank

pytestmark = pytest.mark.gpu

LENGTHS = [0, 1, 2, 63, 64, 65, 127, 128, 129, 511, 5000]


def hub_graph(seed, f32):
    """Node k has LENGTHS[k] out-arcs, a few of them loops, to random nodes of
    300 (parallel arcs among them); lognormal strengths."""
    rng = np.random.default_rng(seed)
    src = np.repeat(np.arange(len(LENGTHS)), LENGTHS)
    tgt = rng.integers(0, 300, len(src))
    loop = rng.random(len(src)) < 0.05
    tgt[loop] = src[loop]
    back = rng.integers(0, 300, 900)  # most other nodes get short rows
    src = np.concatenate([src, back])
    tgt = np.concatenate([tgt, rng.integers(0, len(LENGTHS), 900)])
    order = rng.permutation(len(src))
    w = rng.lognormal(size=len(src))
    if f32:
        w = w.astype(np.float32).astype(np.float64)
    return 300, src[order], tgt[order], w


@pytest.mark.parametrize("directed", [True, False])
def test_degrees_at_row_length_edges(directed):
    n, s, t, w = hub_graph(1, False)
    kg, og = K.Graph(n, s, t, w, directed), O.Graph(n, s, t, w, directed)
    for mode in (1, 2, 3):
        for loops in (False, True):
            assert np.array_equal(kg.degree(mode, loops, False), og.degree(mode, loops, False))
            a, b = kg.degree(mode, loops, True), og.degree(mode, loops, True)
            # two sums of at most 12,000 positive terms, each within 12,000 eps
            assert np.allclose(a, b, rtol=2 * 12_000 * 2.0 ** -53, atol=0)


@pytest.mark.parametrize("f32", [True, False])
@pytest.mark.parametrize("loops", [0, 1, 2])
@pytest.mark.parametrize("directed", [True, False])
def test_pagerank_with_hubs_and_loop_factors(directed, loops, f32):
    n, s, t, w = hub_graph(2, f32)
    kg, og = K.Graph(n, s, t, w, directed), O.Graph(n, s, t, w, directed)
    for d in (True, False):
        kw = dict(directed=d, weighted=True, loops=loops)
        assert np.abs(kg.pagerank(**kw) - og.pagerank(**kw)).sum() <= 1e-12
        a = kg.pagerank(precision=K.PREC_MIXED, **kw)
        assert np.abs(a - og.pagerank(**kw)).sum() <= 1e-9


@pytest.mark.parametrize("directed", [True, False])
def test_edge_gradients_with_hubs_and_loops(directed):
    torch = pytest.importorskip("torch")
    from knappnet_b200 import autograd as A
    n, s, t, w = hub_graph(3, False)
    g = K.Graph(n, s, t, w, directed)
    target = torch.rand(n, dtype=torch.float64, device="cuda") / n
    grads = []
    for solve in (lambda v: A.pagerank(v, g, tol=1e-14),
                  lambda v: dense_pagerank(v, s, t, n, 0.85, directed, 1.0 if directed else 2.0)):
        v = torch.tensor(w, dtype=torch.float64, device="cuda", requires_grad=True)
        ((solve(v) - target) ** 2).sum().backward()
        grads.append(v.grad)
    assert (grads[0] - grads[1]).abs().max().item() <= 1e-9 * grads[1].abs().max().item()
