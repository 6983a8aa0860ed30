"""The sweep a packed graph stops on is decided by the iteration that divides by
the total in every sweep, to the bit: tolerances at a change of that iteration,
and one unit below it. The sizes and the damping are powers of two, so numpy
gives its products without rounding and its sums in the stated order."""
from __future__ import annotations

import numpy as np
import pytest

import knappnet_b200 as K

pytestmark = pytest.mark.gpu

DAMPING = 0.5
SWEEPS = 44


def total(v, threads, split):
    """Every threads-th value added in order, then a warp's 32 sums by halves, then
    the warps in order; from `split` values on each eighth by itself, then these."""
    n = len(v)
    t = 0.0
    for part in v.reshape(8, -1) if n >= split else v[None]:
        lanes = np.zeros(threads)
        for lo in range(0, len(part), threads):
            row = part[lo:lo + threads]
            lanes[:len(row)] += row
        w = lanes.reshape(-1, 32)
        for o in (16, 8, 4, 2, 1):
            w = w + w[:, np.arange(32) ^ o]
        s = 0.0
        for x in w[:, 0]:
            s += x
        t += s
    return t


def iterate(n, src, tgt, threads, split=4096):
    """Changes and iterates of SWEEPS sweeps."""
    order = np.lexsort((src, tgt))
    src, tgt = src[order], tgt[order]
    out = np.bincount(src, minlength=n).astype(np.float64)
    x = np.full(n, 1.0 / n)
    changes, xs = [], []
    for _ in range(SWEEPS):
        z = np.divide(x, out, out=np.zeros(n), where=out > 0)
        stuck = total(np.where(out > 0, 0.0, x), threads, split)
        y = DAMPING * (np.bincount(tgt, z[src], minlength=n) + stuck / n) + (1 - DAMPING) / n
        y = y / total(y, threads, split)
        changes.append(total(np.abs(y - x), threads, split))
        xs.append(y)
        x = y
    return np.array(changes), xs


def edges(n, seed):
    rng = np.random.default_rng(seed)
    m = int(n * rng.uniform(2, 8))
    tgt = rng.integers(0, n, m)
    if seed % 3 == 0:  # a hub row and its neighbours
        tgt[: m // 3] //= max(1, n // 4)
    return rng.integers(0, n - n // 8 * (seed % 2), m), tgt


# one row a thread; several; eight shares of the rows
@pytest.mark.parametrize("n,graphs", [(64, 24), (256, 24), (2048, 6), (4096, 6), (16384, 3)])
def test_single_graphs_stop_where_the_change_says(n, graphs):
    for seed in range(graphs):
        src, tgt = edges(n, seed)
        c, xs = iterate(n, src, tgt, 1024)
        g = K.Graph(n, src, tgt, None, True)
        for k in (4, 11, 19, 28, 37):
            for tol in (c[k], np.nextafter(c[k], 0)):
                if tol <= 0 or not (c <= tol).any():
                    continue
                first = int(np.argmax(c <= tol))
                x, info = g.pagerank_ex(damping=DAMPING, directed=True, tol=float(tol))
                assert info.kernel_launches == 1
                assert info.iterations == first + 1, (seed, k)
                assert info.change == c[first]
                assert np.array_equal(x, xs[first])


def test_a_batch_stops_where_the_changes_say():
    sizes = [64, 128, 256] * 20
    off = np.concatenate([[0], np.cumsum(sizes)])
    parts = [edges(n, k) for k, n in enumerate(sizes)]
    every = [iterate(n, s, t, 256)[0] for n, (s, t) in zip(sizes, parts)]
    g = K.Graph(int(off[-1]), np.concatenate([p[0] + o for p, o in zip(parts, off)]),
                np.concatenate([p[1] + o for p, o in zip(parts, off)]), None, True)
    for k in range(len(sizes)):
        tol = every[k][8 + k % 24]
        if tol <= 0 or not all((c <= tol).any() for c in every):
            continue
        _, its, _ = g.pagerank_graphs(off, damping=DAMPING, directed=True, tol=float(tol))
        assert its.tolist() == [int(np.argmax(c <= tol)) + 1 for c in every]


# at or below a unit of rounding the other iteration is not begun at all
def test_tolerances_of_a_rounding():
    seen = 0
    for seed in range(40):
        src, tgt = edges(64, 100 + seed)
        c, xs = iterate(64, src, tgt, 1024)
        tol = 2.0 ** -53
        if not (c <= tol).any():
            continue
        first = int(np.argmax(c <= tol))
        x, info = K.Graph(64, src, tgt, None, True).pagerank_ex(damping=DAMPING, directed=True,
                                                               tol=tol)
        assert info.iterations == first + 1 and np.array_equal(x, xs[first])
        seen += 1
    assert seen
