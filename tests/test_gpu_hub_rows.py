"""HITS and symmetric eigenvector centrality of graphs with rows at and above
the length that a CTA instead of a warp sums and copies (2048), against the
oracle, with the bounds that hold for the other graphs of both: eigenvalues
to 1e-9 and vectors to 1e-8 (the two directions' simple leading pair)."""
from __future__ import annotations

import numpy as np
import pytest

import knappnet_b200 as K
from oracle import oracle as O

pytestmark = pytest.mark.gpu

N = 6000


def hubs(length, values, seed):
    """A hub with `length` arcs in a row and one in a column, parallel ones
    among them (one run crosses every part of the row), random arcs besides."""
    rng = np.random.default_rng(seed)
    far = rng.integers(0, N, length)
    far[: length // 3] = 17
    src = np.concatenate([np.full(length, 5), rng.integers(0, N, length), rng.integers(0, N, 20000)])
    tgt = np.concatenate([far, np.full(length, 9), rng.integers(0, N, 20000)])
    w = None
    if values:
        w = rng.uniform(0.1, 2.0, len(src))
        w[rng.random(len(src)) < 0.1] = 0.0  # left out of the blocks' matrices
    return src, tgt, w


@pytest.mark.parametrize("length", [2000, 2047, 2048, 2049, 2560, 70_001])
@pytest.mark.parametrize("values", [False, True])
def test_hub_rows(length, values):
    src, tgt, w = hubs(length, values, length)
    kg, og = K.Graph(N, src, tgt, w, True), O.Graph(N, src, tgt, w, True)
    a, b = kg.hits(weighted=values), og.hits(weighted=values)
    assert abs(a[2] - b[2]) <= 1e-9 * b[2] and a[3] == b[3]
    for x, y in zip(a[:2], b[:2]):
        assert np.abs(x - y).max() <= 1e-8 * np.abs(y).max()
    kg, og = K.Graph(N, src, tgt, w, False), O.Graph(N, src, tgt, w, False)
    x, lam, conn = kg.eigenvector(weighted=values)
    y, mu, oconn = og.eigenvector(weighted=values)[:3]
    assert abs(lam - mu) <= 1e-9 * mu and conn == oconn
    assert np.abs(x - y).max() <= 1e-8 * np.abs(y).max()
