"""Work that ends early does so: columns of a batch that stop before the others
count their own sweeps only, and an extrapolated adjoint runs fewer sweeps than
its cap counts."""
from __future__ import annotations

import numpy as np
import pytest

import knappnet_b200 as K
from test_gpu_adjoint import adjoint_vector
from test_gpu_batch_widths import graph, teleport

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")

N = 700


@pytest.mark.parametrize("width", [7, 40, 129])
def test_columns_count_their_own_sweeps(width):
    src, tgt, _ = graph(None)
    g = K.Graph(N, src, tgt, None, True)
    P = teleport(width, False)
    _, info = g.pagerank_batch(P, tol=1e-12, precision=K.PREC_FP64)
    alone = [g.pagerank_batch(p[None], tol=1e-12, precision=K.PREC_FP64)[1].column_iterations
             for p in P]
    # a sum of another order may move a column by a sweep
    assert abs(info.column_iterations - sum(alone)) <= width
    assert abs(info.max_column_iterations - max(alone)) <= 1
    assert len(set(alone)) > 1


def test_an_extrapolated_adjoint_runs_fewer_sweeps_than_its_cap_counts():
    g = K.generate_rmat(10, 16, seed=8, clean=True, lognormal=True, wseed=9)
    w = torch.tensor(g.edges()[2], device="cuda")
    x = torch.tensor(g.pagerank(weighted=True), device="cuda")
    gx = torch.rand(g.n, dtype=torch.float64, device="cuda")
    _, _, info = adjoint_vector(g, w, x, gx, max_iter=400)
    assert info.iterations < 100  # the plain iteration needs about 170
