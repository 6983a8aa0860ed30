"""Strong components over several rounds of colouring, against the oracle's
Tarjan: after a round the arcs between unassigned nodes are copied out when
at most 2^22 of more than 2^20 are left, else the next round tries again.
Labels, counts and sizes are whole numbers and must be the same."""
from __future__ import annotations

import numpy as np
import pytest

import knappnet_b200 as K
from oracle import oracle as O

pytestmark = pytest.mark.gpu

KEEP = 1 << 22


def layers(sizes, seed):
    """Strong components (a cycle and random arcs each) of (nodes, arcs), each
    reaching the next by arcs from it. The first holds the largest ids, so a
    round of colours by largest ancestor assigns one component at a time."""
    rng = np.random.default_rng(seed)
    n = sum(k for k, _ in sizes)
    src, tgt, top = [], [], n
    for k, m in sizes:
        ids = np.arange(top - k, top)
        src += [ids, rng.integers(top - k, top, m - k)]
        tgt += [np.roll(ids, 1), rng.integers(top - k, top, m - k)]
        top -= k
        if top:  # one arc into the next component's largest node
            src.append(ids[:1])
            tgt.append(np.array([top - 1]))
    return n, np.concatenate(src), np.concatenate(tgt)


@pytest.mark.parametrize("sizes", [
    # at most 2^20 arcs: nothing is copied out
    [(500, 2000), (900, 4000), (33, 100)],
    # more, and what is left after the first round fits
    [(2000, KEEP // 4 + 1), (1000, 5000), (257, 700), (31, 40)],
    # nothing but single nodes and short cycles is left
    [(5000, KEEP // 4 + 5000), (2, 2), (2, 3)],
    # too many are left after the first round, few after the second
    [(300, 1000), (40000, KEEP + 4096), (700, 3000), (2, 2)],
])
def test_rounds(sizes):
    n, src, tgt = layers(sizes, 5)
    got, count = K.Graph(n, src, tgt, None, True).components(strong=True)
    want, wcount = O.Graph(n, src, tgt, None, True).components(strong=True)
    assert count == wcount == len(sizes)
    assert np.array_equal(got.astype(np.int64), want.astype(np.int64))


@pytest.mark.parametrize("n", [1, 31, 32, 33, 255, 257])
@pytest.mark.parametrize("strong", [False, True])
def test_label_warps(n, strong):
    """Sizes at the edges of a warp and a block, in one component and in n."""
    a = np.arange(n)
    for src, tgt, k in ((a, (a + 1) % n, 1), (a, a, n)):
        got, count = K.Graph(n, src, tgt, None, True).components(strong=strong)
        assert count == k
        assert np.array_equal(got, np.zeros(n) if k == 1 else a)
