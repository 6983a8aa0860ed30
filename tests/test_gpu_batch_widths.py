"""Batched PageRank at the widths where a sweep's work is split differently
(several rows per warp up to 16 columns, whole warps above), with columns that
stop at very different sweeps, so that the running ones are packed into ever
narrower iterates on the way."""
from __future__ import annotations

import numpy as np
import pytest

import knappnet_b200 as K
from oracle import oracle as O

pytestmark = pytest.mark.gpu

N = 700


def graph(weights):
    """A random digraph with dangling nodes, a hub of 1,500 in-arcs (a row cut
    into chunks) and a closed pair {0, 1}: teleport vectors that reach the
    pair converge as slowly as the damping allows."""
    rng = np.random.default_rng(3)
    src = rng.integers(2, N, 5000)
    tgt = rng.integers(0, N, 5000)
    src = np.where(src >= N - 60, src - 60, src)
    src = np.concatenate([src, rng.integers(2, N - 60, 1500), [0, 1]])
    tgt = np.concatenate([tgt, np.full(1500, 5), [1, 0]])
    w = None
    if weights:
        w = rng.lognormal(size=len(src))
        if weights == "f32":
            w = w.astype(np.float32).astype(np.float64)
    return src, tgt, w


def teleport(width, dense):
    """Sparse seed sets (or dense vectors); a few put all their mass on the
    closed pair, some on nodes without out-arcs."""
    rng = np.random.default_rng(width)
    P = np.zeros((width, N))
    for c in range(width):
        if dense:
            P[c] = rng.random(N)
        elif c % 7 == 3:
            P[c, c % 2] = 1.0
        elif c % 7 == 5:
            P[c, N - 1 - c % 50] = 1.0
        else:
            P[c, rng.choice(N, rng.integers(1, 20), replace=False)] = 1.0
    return P


@pytest.mark.parametrize("width", [1, 2, 3, 4, 5, 8, 9, 16, 17, 32, 33, 65, 129, 256, 261])
@pytest.mark.parametrize("precision,bar", [(K.PREC_FP64, 1e-12), (K.PREC_MIXED, 1e-9)])
def test_every_column_matches_the_oracle(width, precision, bar):
    weights = [None, "f32", "f64"][width % 3]
    src, tgt, w = graph(weights)
    kg, og = K.Graph(N, src, tgt, w, True), O.Graph(N, src, tgt, w, True)
    # a column with half its mass on one node cannot settle below about 1e-11
    # once its correction is held in FP32
    tol = 1e-12 if precision == K.PREC_FP64 else 1e-10
    for dense in (False, True):
        P = teleport(width, dense)
        kw = dict(weighted=w is not None, dangling=width % 2, tol=tol)
        X, info = kg.pagerank_batch(P, precision=precision, **kw)
        again, _ = kg.pagerank_batch(P, precision=precision, **kw)
        assert np.array_equal(X, again)
        pick = sorted({0, 3, 5, width - 1} & set(range(width)))
        for c in pick:
            ref = og.pagerank(personalization=P[c], **kw)
            assert np.abs(X[c] - ref).sum() <= bar, (width, dense, c)
        assert np.abs(X.sum(1) - 1).max() <= 1e-12
        assert info.column_iterations <= info.max_column_iterations * width


def test_a_slow_column_still_reaches_the_cap():
    src, tgt, _ = graph(None)
    g = K.Graph(N, src, tgt, None, True)
    P = teleport(40, False)
    for precision in (K.PREC_FP64, K.PREC_MIXED):
        with pytest.raises(K.EngineError, match="did not converge .* within 60 iterations"):
            g.pagerank_batch(P, tol=1e-12, max_iter=60, precision=precision)


def test_plain_fp64_phase_after_fp32_sweeps():
    src, tgt, w = graph("f64")
    kg, og = K.Graph(N, src, tgt, w, True), O.Graph(N, src, tgt, w, True)
    P = teleport(37, False)
    try:
        K.set_tuning(K.TUNE_REFINE, 0)
        X, _ = kg.pagerank_batch(P, weighted=True, precision=K.PREC_MIXED, tol=1e-12)
    finally:
        K.set_tuning(K.TUNE_REFINE, 1)
    for c in (0, 3, 5, 36):
        assert np.abs(X[c] - og.pagerank(weighted=True, personalization=P[c], tol=1e-12)).sum() <= 1e-9
