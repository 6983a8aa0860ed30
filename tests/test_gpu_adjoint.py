"""Differentiable PageRank: the hand-written adjoint against dense torch
autograd (FP64) and central finite differences."""
from __future__ import annotations

import numpy as np
import pytest

import knappnet_b200 as K

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")


def dense_pagerank(w, src, tgt, n, d, directed, loops_factor=1.0):
    """PageRank by a dense solve: M[i, j] = sum of w over arcs j -> i / s_j,
    x = solve(I - d M - d jump 1_D^T, (1 - d) p), uniform p and jump."""
    A = torch.zeros((n, n), dtype=torch.float64, device=w.device)
    s_ = torch.as_tensor(src, device=w.device)
    t_ = torch.as_tensor(tgt, device=w.device)
    f = torch.where(s_ == t_, torch.as_tensor(loops_factor, dtype=torch.float64, device=w.device),
                    torch.ones((), dtype=torch.float64, device=w.device))
    A = A.index_put((t_, s_), w * f, accumulate=True)
    if not directed:
        off = s_ != t_
        A = A.index_put((s_[off], t_[off]), w[off], accumulate=True)
    out = A.sum(dim=0)
    dang = out == 0
    M = A / torch.where(dang, torch.ones_like(out), out)
    jump = torch.full((n,), 1.0 / n, dtype=torch.float64, device=w.device)
    G = M + torch.outer(jump, dang.to(torch.float64))
    I = torch.eye(n, dtype=torch.float64, device=w.device)
    x = torch.linalg.solve(I - d * G, (1 - d) * jump)
    return x / x.sum()


def random_weighted(n, m, seed, directed=True):
    rng = np.random.default_rng(seed)
    src = rng.integers(0, n, m)
    tgt = rng.integers(0, n, m)
    # some dangling nodes: no arcs out of the last tenth
    src = np.where(src >= n - n // 10, src - n // 10, src)
    w = rng.lognormal(size=m)
    return src, tgt, w


@pytest.mark.parametrize("directed", [True, False])
def test_adjoint_matches_dense_autograd(directed):
    from knappnet_b200 import autograd as A
    n, m = 300, 2400
    src, tgt, w = random_weighted(n, m, 3, directed)
    g = K.Graph(n, src, tgt, w, directed)
    wt = torch.tensor(w, dtype=torch.float64, device="cuda", requires_grad=True)
    target = torch.rand(n, dtype=torch.float64, device="cuda") / n
    x = A.pagerank(wt, g, tol=1e-14)
    loss = ((x - target) ** 2).sum()
    loss.backward()
    ours = wt.grad.detach().clone()
    wd = torch.tensor(w, dtype=torch.float64, device="cuda", requires_grad=True)
    xd = dense_pagerank(wd, src, tgt, n, 0.85, directed, 1.0 if directed else 2.0)
    assert torch.abs(x.detach() - xd.detach()).sum().item() <= 1e-12
    ld = ((xd - target) ** 2).sum()
    ld.backward()
    ref = wd.grad.detach()
    err = torch.abs(ours - ref).max().item()
    scale = torch.abs(ref).max().item()
    assert err <= 1e-9 * scale, (err, scale)


def test_adjoint_finite_differences_on_rmat_subgraph():
    from knappnet_b200 import autograd as A
    # 1,000-node induced subgraph of an R-MAT graph: the 1,000 nodes of
    # highest total degree
    big = K.generate_rmat(12, 16, seed=4, clean=True, lognormal=True, wseed=5)
    s, t, w = big.edges()
    deg = np.bincount(s, minlength=big.n) + np.bincount(t, minlength=big.n)
    keep = np.argsort(-deg, kind="stable")[:1000]
    idx = -np.ones(big.n, dtype=np.int64)
    idx[keep] = np.arange(1000)
    sel = (idx[s] >= 0) & (idx[t] >= 0)
    src, tgt, w = idx[s[sel]], idx[t[sel]], w[sel]
    g = K.Graph(1000, src, tgt, w, True)
    rng = np.random.default_rng(7)
    wt = torch.tensor(w, dtype=torch.float64, device="cuda", requires_grad=True)
    # target: PageRank with weights perturbed by 10%
    wp = torch.tensor(w * np.maximum(1 + 0.1 * rng.standard_normal(len(w)), 1e-3),
                      dtype=torch.float64, device="cuda")
    target = A.pagerank(wp, g, tol=1e-15).detach()
    x = A.pagerank(wt, g, tol=1e-15)
    loss = ((x - target) ** 2).sum()
    loss.backward()
    grad = wt.grad.detach().cpu().numpy()
    picks = rng.choice(len(w), 25, replace=False)
    for e in picks:
        h = 1e-4 * w[e]
        wa = w.copy()
        wa[e] += h
        wb = w.copy()
        wb[e] -= h
        la = ((A.pagerank(torch.tensor(wa, device="cuda"), g, tol=1e-15) - target) ** 2).sum()
        lb = ((A.pagerank(torch.tensor(wb, device="cuda"), g, tol=1e-15) - target) ** 2).sum()
        fd = (la - lb).item() / (2 * h)
        assert abs(fd - grad[e]) <= 1e-5 * max(abs(fd), 1e-3 * np.abs(grad).max()), (e, fd, grad[e])


def test_weights_forward_matches_graph_weights():
    kg = K.generate_rmat(11, 16, seed=8, clean=True, lognormal=True, wseed=9)
    _, _, w = kg.edges()
    a = kg.pagerank(weighted=True)
    out = torch.empty(kg.n, dtype=torch.float64, device="cuda")
    wt = torch.tensor(w, device="cuda")
    import ctypes
    info = K.NetSolveInfo()
    err = ctypes.create_string_buffer(K.ERR_LEN)
    K._check(K.lib().net_pagerank_weights_device(kg.h, ctypes.c_void_p(wt.data_ptr()), 0.85, 1,
                                                 None, 0, 0, 0.0, 0, 0,
                                                 ctypes.c_void_p(out.data_ptr()),
                                                 ctypes.byref(info), err, K.ERR_LEN), err)
    assert np.abs(out.cpu().numpy() - a).sum() <= 1e-12


def adjoint_vector(g, w, x, gx, tol=0.0, max_iter=0, pers=None, dangling=0):
    """net_pagerank_grad_device with the adjoint vector: (grad, lambda, info)."""
    import ctypes
    grad = torch.empty(g.m, dtype=torch.float64, device="cuda")
    lam = torch.empty(g.n, dtype=torch.float64, device="cuda")
    info = K.NetSolveInfo()
    err = ctypes.create_string_buffer(K.ERR_LEN)
    p = lambda t: None if t is None else ctypes.c_void_p(t.data_ptr())
    torch.cuda.synchronize()
    K._check(K.lib().net_pagerank_grad_device(g.h, p(w), p(x), p(gx), 0.85, int(g.directed),
                                              p(pers), dangling, 0, tol, max_iter, p(grad), p(lam),
                                              ctypes.byref(info), err, K.ERR_LEN), err)
    return grad, lam, info


@pytest.mark.parametrize("shape", ["mixing", "two closed halves", "cycle"])
@pytest.mark.parametrize("personalized", [False, True])
def test_adjoint_vector_solves_its_equation(shape, personalized):
    """lambda = g + d G lambda, whether one closed class holds all that shrinks
    slowly (mixing), two do (two closed halves), or no part of the change
    shrinks faster than d (a cycle)."""
    from knappnet_b200 import autograd as A
    n = 400
    rng = np.random.default_rng(11)
    if shape == "cycle":
        src, tgt = np.arange(n), (np.arange(n) + 1) % n
    else:
        src, tgt = rng.integers(0, n, 4000), rng.integers(0, n, 4000)
        if shape == "two closed halves":
            tgt = tgt % (n // 2) + np.where(src < n // 2, 0, n // 2)
        else:  # dangling nodes
            src = np.where(src >= n - 40, src - 40, src)
    w = rng.lognormal(size=len(src))
    g = K.Graph(n, src, tgt, w, True)
    wt = torch.tensor(w, device="cuda")
    pers = torch.rand(n, dtype=torch.float64, device="cuda") if personalized else None
    x = A.pagerank(wt, g, personalization=pers, tol=1e-14).detach()
    gx = torch.randn(n, dtype=torch.float64, device="cuda")
    _, lam, info = adjoint_vector(g, wt, x, gx, pers=pers)
    G = torch.zeros((n, n), dtype=torch.float64, device="cuda")
    G.index_put_((torch.as_tensor(src, device="cuda"), torch.as_tensor(tgt, device="cuda")), wt,
                 accumulate=True)
    out = G.sum(1, keepdim=True)
    jump = torch.full((n,), 1.0 / n, dtype=torch.float64, device="cuda")
    if personalized:
        jump = pers / pers.sum()
    G = torch.where(out > 0, G / torch.where(out > 0, out, torch.ones_like(out)), jump)
    ref = torch.linalg.solve(torch.eye(n, dtype=torch.float64, device="cuda") - 0.85 * G, gx)
    # a change of at most tol max(1, ||g||_1) leaves an L1 error of at most
    # n d / (1 - d) times it, and the dense solve one of its condition number
    bound = n * 0.85 / 0.15 * 1e-12 * max(1.0, gx.abs().sum().item())
    assert (lam - ref).abs().sum().item() <= bound + 1e-12 * ref.abs().sum().item()
    if shape != "cycle":
        assert info.iterations < 100  # 0.85^k alone would need 170


def test_adjoint_iteration_cap_means_the_same_sweeps():
    """The cap counts the sweeps the tolerance needs (the constant part shrinks
    by d = 0.85: about ln(1e-12) / ln(0.85) = 170 here), though fewer run."""
    g = K.generate_rmat(10, 16, seed=8, clean=True, lognormal=True, wseed=9)
    w = torch.tensor(g.edges()[2], device="cuda")
    x = torch.tensor(g.pagerank(weighted=True), device="cuda")
    gx = torch.rand(g.n, dtype=torch.float64, device="cuda")
    with pytest.raises(K.EngineError, match="did not converge within 100 iterations"):
        adjoint_vector(g, w, x, gx, max_iter=100)
    _, _, info = adjoint_vector(g, w, x, gx, max_iter=400)
    assert info.iterations <= 400
