"""The device radix sort at the edges of its 2048-element tiles, through the
arcs of a graph: parallel edges keep their input order, so a row's arcs and
the edge indices beside them are those of a stable sort, and whole numbers."""
from __future__ import annotations

import numpy as np
import pytest

import knappnet_b200 as K
from oracle import oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("m", [2, 31, 33, 255, 257, 2047, 2048, 2049, 4096, 4097, 300_001])
@pytest.mark.parametrize("n", [2, 300, 70_000])
def test_simplify_sizes(n, m):
    """Keys of one digit, of three, and with bits left over in the last."""
    rng = np.random.default_rng(m + n)
    src, tgt = rng.integers(0, n, m), rng.integers(0, n, m)
    w = rng.uniform(0.1, 5.0, m)
    for undirected, keep in ((False, 0), (True, 1)):
        a = K.Graph(n, src, tgt, w, True).simplify(undirected, keep).edges()
        b = O.Graph(n, src, tgt, w, True).simplify(undirected, keep).edges()
        for x, y in zip(a, b):
            assert np.array_equal(x, y)


@pytest.mark.parametrize("m", [2047, 2048, 2049, 70_001])
def test_parallel_edges_keep_their_order(m):
    """Weights that come after the build reach the arcs by the edge index that
    was sorted along: one that went astray hands an arc another edge's weight."""
    torch = pytest.importorskip("torch")
    from knappnet_b200 import autograd as A
    n = 5
    rng = np.random.default_rng(m)
    src, tgt = rng.integers(0, n, m), rng.integers(0, n, m)
    w = rng.uniform(0.1, 5.0, m)
    g = K.Graph(n, src, tgt, np.ones(m), True)
    x = A.pagerank(torch.tensor(w, dtype=torch.float64, device="cuda"), g, tol=1e-13)
    want = O.Graph(n, src, tgt, w, True)
    ref = want.pagerank(weighted=True, tol=1e-14)
    # both sides stop within their tolerance of a fixed point that contracts
    # by 0.85, and sum up to m terms a row one after the other at worst
    assert np.abs(x.cpu().numpy() - ref).max() <= (2 * 1e-13 + m * 2.0 ** -53) / 0.15
