"""Packed-graph PageRank where its launch changes: one CTA or a cluster, all of
a graph in shared memory, its vectors only, or none of it; hub rows taken by
whole warps; 1, 4 and 8 bytes of arc value. Against the oracle: L1 within 1e-12
(plus the oracle's own normalisation residual) and the same iteration count."""
from __future__ import annotations

import numpy as np
import pytest

import knappnet_b200 as K
from oracle import oracle as O

pytestmark = pytest.mark.gpu


def graph(n, degree, seed, weights, hubs):
    rng = np.random.default_rng(seed)
    m = max(1, n * degree // 2)
    src = rng.integers(0, n, m)
    tgt = rng.integers(0, n, m)
    if hubs:  # a few nodes hold most arcs; the last tenth has no out-arcs
        tgt = np.minimum(tgt, rng.integers(0, n, m) // 7)
        src = np.where(src >= n - n // 10, src - n // 10, src)
    w = None
    if weights:
        w = rng.lognormal(size=m)
        if weights == "f32":
            w = w.astype(np.float32).astype(np.float64)
    return src, tgt, w


def check(x, its, n, s, t, w, directed, **kw):
    og = O.Graph(n, s, t, w, directed)
    ref = og.pagerank(directed=directed, weighted=w is not None, **kw)
    assert np.abs(x - ref).sum() <= 1e-12 + abs(1.0 - ref.sum()), n
    # the sweep path stops on the oracle's sweep (tests/test_gpu_parity.py)
    g = K.Graph(n, s, t, w, directed)
    try:
        K.set_tuning(K.TUNE_SMALL_EDGES, 0)
        _, info = g.pagerank_ex(directed=directed, weighted=w is not None, **kw)
    finally:
        K.set_tuning(K.TUNE_SMALL_EDGES, 1 << 18)
    assert its == info.iterations


# one CTA below 400 nodes; a cluster of 8 while z fits every CTA's shared
# memory (about 11,000 nodes without values, 5,000 with FP64 values and 20
# arcs a node); columns of more than 16 bits above 65,536
@pytest.mark.parametrize("n,degree", [(1, 2), (2, 2), (31, 4), (33, 60), (399, 6), (400, 6),
                                      (1025, 40), (5000, 20), (11000, 10), (12500, 10),
                                      (65536, 4), (65537, 4)])
@pytest.mark.parametrize("weights", [None, "f32", "f64"])
def test_single_graph(n, degree, weights):
    for k, directed in enumerate((True, False)):
        s, t, w = graph(n, degree, n + k, weights, hubs=k == 0)
        g = K.Graph(n, s, t, w, directed)
        pers = None if k else np.arange(n) % 3 + 1.0
        # (the oracle's sequential sums over 65,537 nodes stall above 1e-12)
        kw = dict(personalization=pers, dangling=n % 2, tol=1e-12 if n < 65536 else 1e-11)
        x, info = g.pagerank_ex(directed=directed, weighted=w is not None, **kw)
        assert info.kernel_launches == 1
        check(x, info.iterations, n, s, t, w, directed, **kw)
        again, _ = g.pagerank_ex(directed=directed, weighted=w is not None, **kw)
        assert np.array_equal(x, again)


@pytest.mark.parametrize("weights", [None, "f32", "f64"])
def test_batch_of_mixed_sizes(weights):
    sizes = [1, 40, 0, 580, 700, 1300, 4095, 4096, 9000, 300, 2, 15000]
    off = np.concatenate([[0], np.cumsum(sizes)])
    parts = [graph(n, 12, 7 + k, weights, k % 2 == 0) if n > 1 else
             (np.zeros(0, np.int64),) * 2 + (np.zeros(0),) for k, n in enumerate(sizes)]
    src = np.concatenate([p[0] + o for p, o in zip(parts, off)])
    tgt = np.concatenate([p[1] + o for p, o in zip(parts, off)])
    w = np.concatenate([p[2] for p in parts]) if weights else None
    g = K.Graph(int(off[-1]), src, tgt, w, True)
    pers = np.arange(off[-1]) % 5 + 0.5
    for p in (None, pers):
        x, its, _ = g.pagerank_graphs(off, weighted=w is not None, personalization=p)
        for k, n in enumerate(sizes):
            if n == 0:
                assert its[k] == 0
                continue
            s, t, wk = parts[k]
            check(x[off[k]:off[k + 1]], its[k], n, s, t, wk if weights else None, True,
                  personalization=None if p is None else p[off[k]:off[k + 1]])
