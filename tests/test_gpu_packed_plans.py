"""The kept launch of a packed batch follows what it depends on: the tuning keys
and the teleport vector of the call, not those of an earlier one."""
from __future__ import annotations

import numpy as np
import pytest

import knappnet_b200 as K
from oracle import oracle as O

pytestmark = pytest.mark.gpu


def packed(sizes, degree, seed):
    rng = np.random.default_rng(seed)
    off = np.concatenate([[0], np.cumsum(sizes)])
    which = np.repeat(np.arange(len(sizes)), np.maximum(1, np.asarray(sizes) * degree // 2))
    a, b = (off[which] + (rng.random(len(which)) * np.asarray(sizes)[which]).astype(np.int64)
            for _ in range(2))
    return K.Graph(int(off[-1]), a, b, None, False), off


def test_the_large_graph_threshold_of_the_call():
    sizes = [6000, 3000, 1500, 700, 300]
    g, off = packed(sizes, 8, 1)
    try:
        for big, split in ((0, 1), (1000, 3), (500, 4), (0, 1)):
            K.set_tuning(K.TUNE_EGO_BIG_NODES, big)
            _, _, info = g.pagerank_graphs(off)
            assert info.iterations_fp32 == split  # graphs split over a cluster
    finally:
        K.set_tuning(K.TUNE_EGO_BIG_NODES, 0)


def test_a_pinned_shape_does_not_outlive_its_pins():
    rng = np.random.default_rng(2)
    sizes = np.concatenate([[30_000], rng.integers(50, 400, 1500)])
    fresh = set()
    for _ in range(3):  # timed on the batch itself
        g, off = packed(sizes, 12, 3)
        _, _, info = g.pagerank_graphs(off)
        fresh.add((info.sweep_kernel, info.hot_columns))
    g, off = packed(sizes, 12, 3)
    try:
        for threads, cluster in ((128, 4), (128, 0), (0, 4)):
            K.set_tuning(K.TUNE_EGO_THREADS, threads)
            K.set_tuning(K.TUNE_EGO_CLUSTER, cluster)
            _, _, info = g.pagerank_graphs(off)
            assert threads in (0, info.sweep_kernel) and cluster in (0, info.hot_columns)
    finally:
        K.set_tuning(K.TUNE_EGO_THREADS, 0)
        K.set_tuning(K.TUNE_EGO_CLUSTER, 0)
    _, _, info = g.pagerank_graphs(off)
    assert (info.sweep_kernel, info.hot_columns) in fresh


# 10,000 nodes and arcs fit a cluster of 8 without a teleport vector only
def test_a_single_graphs_shape_follows_its_own_teleport():
    n = 10_000
    rng = np.random.default_rng(4)
    g = K.Graph(n, rng.integers(0, n, n), rng.integers(0, n, n), None, True)
    pers = rng.random(n)
    for p, cluster in ((pers, 16), (None, 8), (pers, 16), (None, 8)):
        _, _, info = g.pagerank_graphs([0, n], personalization=p)
        assert info.hot_columns == cluster


# On both sides of what a cluster of 8 holds (about 9,600 nodes of 10 arcs without
# values), and a row whose CTA cannot hold its arcs (its graph's vectors stay in
# shared memory, the arcs do not): scores of the oracle, and the cluster that says
# which side a graph is on.
@pytest.mark.parametrize("n,m,hub,weighted,cluster",
                         [(9000, 90_000, 0, False, 8), (10_000, 100_000, 0, False, 16),
                          (3000, 90_000, 45_000, True, 8)])
def test_scores_on_both_sides_of_the_shared_memory(n, m, hub, weighted, cluster):
    rng = np.random.default_rng(n)
    src, tgt = rng.integers(0, n, m), rng.integers(0, n, m)
    tgt[:hub] = 17
    w = rng.lognormal(size=m) if weighted else None
    g, o = K.Graph(n, src, tgt, w, True), O.Graph(n, src, tgt, w, True)
    for pers in (None, rng.random(n)):
        x, its, info = g.pagerank_graphs([0, n], weighted=weighted, personalization=pers,
                                         tol=1e-12)
        if pers is None:
            assert info.hot_columns == cluster
        y = o.pagerank(weighted=weighted, personalization=pers, tol=1e-12)
        assert np.abs(x - y).sum() <= 1e-12 + abs(1.0 - y.sum())
