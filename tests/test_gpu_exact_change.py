"""Stopping where the cheap bounds of the L1 change cannot tell it from the
tolerance: the tolerance of the second solve is the change that the first one
stopped with, to the bit, so that the exact change decides. It has to stop
there, or one sweep later if the first one's change was a rounding off."""
from __future__ import annotations

import numpy as np
import pytest

import knappnet_b200 as K
from oracle import oracle as O

pytestmark = pytest.mark.gpu

TOL = 1e-7


# packed (one cluster), the sweeps' sizes, and rows long enough to be split
@pytest.mark.parametrize("n,m,hub", [(33, 200, 0), (1500, 9000, 0), (9001, 70_000, 0),
                                     (40_000, 300_000, 20_000), (70_001, 700_003, 0)])
@pytest.mark.parametrize("precision", [K.PREC_FP64, K.PREC_MIXED])
@pytest.mark.parametrize("dangling", [0, 1])
def test_tolerance_at_a_change(n, m, hub, precision, dangling):
    rng = np.random.default_rng(n + hub)
    src, tgt = rng.integers(0, n, m), rng.integers(0, n, m)
    tgt[:hub] = 3
    w = rng.lognormal(size=m)
    g, o = K.Graph(n, src, tgt, w, True), O.Graph(n, src, tgt, w, True)
    kw = dict(weighted=True, dangling=dangling, precision=precision)
    _, first = g.pagerank_ex(tol=TOL, **kw)
    assert 0 < first.change <= TOL
    x, info = g.pagerank_ex(tol=first.change, **kw)
    assert info.converged and info.change <= first.change
    # FP32 sweeps before the FP64 ones switch on a multiple of the tolerance
    if precision == K.PREC_FP64:
        assert info.iterations in (first.iterations, first.iterations + 1)
    # the map contracts by 0.85 in L1: within change * 0.85 / 0.15 of the fixed
    # point, and the oracle as well
    y = o.pagerank(weighted=True, dangling=dangling, tol=1e-12)
    assert np.abs(x - y).sum() <= (first.change + 1e-12) * 0.85 / 0.15 + n * 2.0 ** -52
    again, _ = g.pagerank_ex(tol=first.change, **kw)
    assert np.array_equal(x, again)
    # below the change of this iterate it must go on
    _, less = g.pagerank_ex(tol=info.change * (1 - 1e-6), **kw)
    assert less.change <= info.change * (1 - 1e-6)
    if precision == K.PREC_FP64:
        assert less.iterations > info.iterations
