"""Workloads of the library's public entry points, as user programs call them.

Each case is a dict of plain values; `prepare` makes what a program holds
before the call (a graph handle, weights, teleport vectors) from a seed
alone, `run` is one pass through the public API, `exact` restates the result
in 64-bit torch / numpy, and `work` counts what a pass cannot do without.

Kinds: "pagerank" (one solve), "batch" (many teleport vectors), "egos" (many
packed graphs), "eigenvector", "hits", "katz", "gradient" (differentiable
PageRank, forward and backward), "components" and "build" (an edge table in
host memory to a graph, its CSR and its strengths).
"""
import ctypes
import math

import numpy as np
import torch

import knappnet_b200 as K
from knappnet_b200 import autograd as AG

DAMPING = 0.85
DEV = "cuda"


# ------------------------------------------------------------------ inputs
def _generator(seed):
    return torch.Generator(device=DEV).manual_seed(seed)


def _rmat_draws(n, m, gen):
    """m endpoint pairs of an R-MAT graph (0.57 / 0.19 / 0.19 / 0.05) scaled to n nodes."""
    levels = max(1, (n - 1).bit_length())
    src = torch.empty(m, dtype=torch.int64, device=DEV)
    tgt = torch.empty(m, dtype=torch.int64, device=DEV)
    step = 1 << 25
    for lo in range(0, m, step):
        k = min(step, m - lo)
        s = torch.zeros(k, dtype=torch.int64, device=DEV)
        t = torch.zeros(k, dtype=torch.int64, device=DEV)
        for _ in range(levels):
            u = torch.rand(k, device=DEV, generator=gen)
            s.mul_(2).add_(u >= 0.76)
            t.mul_(2).add_(((u >= 0.57) & (u < 0.76)) | (u >= 0.95))
        src[lo:lo + k] = (s * n) >> levels
        tgt[lo:lo + k] = (t * n) >> levels
    return src, tgt


def _draw_keys(case, m, gen):
    """m drawn edges as src * n + tgt, loops left out."""
    n = case["n"]
    if case["graph"] == "er":
        src = torch.randint(0, n, (m,), device=DEV, generator=gen)
        tgt = torch.randint(0, n, (m,), device=DEV, generator=gen)
    else:
        src, tgt = _rmat_draws(n, m, gen)
    if not case["directed"]:
        src, tgt = torch.minimum(src, tgt), torch.maximum(src, tgt)
    return (src * n + tgt)[src != tgt]


def _edges(case, gen):
    """Distinct edges without loops, sorted: (src, tgt) int64 on the GPU. Those that are left
    of `edges` draws, or, where every edge has a parameter of its own, exactly `edges`."""
    n, m = case["n"], case["edges"]
    key = torch.unique(_draw_keys(case, m, gen))
    if case["kind"] == "gradient":
        while len(key) < m:
            key = torch.unique(torch.cat([key, _draw_keys(case, m // 4 + 64, gen)]))
        key = key[torch.randperm(len(key), device=DEV, generator=gen)[:m].sort()[0]]
    return key // n, key % n


def _weights(case, m, gen):
    """Lognormal(0, 1) tie strengths, in FP32 or FP64; None for an unweighted graph."""
    if case["weights"] == "none":
        return None
    dt = torch.float32 if case["weights"] == "f32" else torch.float64
    return torch.empty(m, dtype=dt, device=DEV).log_normal_(generator=gen)


def _device_graph(n, src, tgt, w, directed):
    """A graph handle from edge arrays on the GPU (net_graph_new_device)."""
    s, t = src.to(torch.int32), tgt.to(torch.int32)
    torch.cuda.synchronize()
    h = ctypes.c_void_p()
    err = ctypes.create_string_buffer(K.ERR_LEN)
    ptr = lambda x: None if x is None else ctypes.c_void_p(x.data_ptr())  # noqa: E731
    w32 = w if w is not None and w.dtype == torch.float32 else None
    w64 = w if w is not None and w.dtype == torch.float64 else None
    if K.lib().net_graph_new_device(n, ptr(s), ptr(t), ptr(w32), ptr(w64), s.numel(),
                                    int(directed), ctypes.byref(h), err, K.ERR_LEN):
        raise K.EngineError(err.value.decode())
    return K.Graph(n, directed=directed, _handle=h, _m=s.numel(), _weighted=w is not None)


def _teleport(n, k, gen):
    """k teleport vectors, each uniform over 1 to 64 random seed nodes."""
    P = torch.zeros(k, n, dtype=torch.float64, device=DEV)
    count = torch.randint(1, 65, (k, 1), device=DEV, generator=gen)
    pick = torch.randint(0, n, (k, 64), device=DEV, generator=gen)
    P.scatter_add_(1, pick, (torch.arange(64, device=DEV) < count).to(torch.float64))
    return P / P.sum(1, keepdim=True)


def _pers_vector(n, gen):
    """A teleport vector over all nodes: positive interest, a third of the nodes without any."""
    p = torch.empty(n, dtype=torch.float64, device=DEV).log_normal_(generator=gen)
    p = torch.where(torch.rand(n, device=DEV, generator=gen) < 1 / 3, torch.zeros_like(p), p)
    p[0] = 1.0
    return p


def _egos(case, gen):
    """Undirected G(n, 6 n) graphs with power-law sizes (exponent 2.1), packed:
    (node offsets on the host, src, tgt)."""
    # the law's quantiles in random order: the packed size does not depend on the seed
    u = torch.randperm(case["graphs"], device=DEV, generator=gen).double()
    u = (u + 0.5) / case["graphs"]
    a, lo, hi = 1.1, 50.0, float(case["largest"])
    size = (lo ** -a - u * (lo ** -a - hi ** -a)) ** (-1 / a)
    size = size.floor().to(torch.int64).clamp_(50, case["largest"])
    size[int(u.argmax())] = case["largest"]
    off = torch.cat([size.new_zeros(1), size.cumsum(0)])
    g = torch.repeat_interleave(torch.arange(len(size), device=DEV), 6 * size)
    r = torch.rand(2, len(g), device=DEV, generator=gen, dtype=torch.float64)
    a, b = ((r * size[g]).floor().to(torch.int64) + off[g])
    n = int(off[-1])
    key = torch.minimum(a, b) * n + torch.maximum(a, b)
    key = torch.unique(key[a != b])
    return off.cpu().numpy(), key // n, key % n


def _katz_alpha(n, src, tgt, w):
    """0.5 / lambda_max of the weighted adjacency matrix, to six digits, by power iteration."""
    x = torch.ones(n, dtype=torch.float64, device=DEV)
    lam = 1.0
    wd = 1.0 if w is None else w.double()
    for _ in range(15):
        y = torch.zeros_like(x).index_add_(0, tgt, wd * x[src])
        lam = float(y.norm() / x.norm()) or 1.0
        x = y / lam + 1e-30
    return float("%.5e" % (0.5 / lam))


def _inputs(case, seed):
    """Everything the case draws from its seed."""
    gen = _generator(seed)
    kind = case["kind"]
    if kind == "egos":
        off, s, t = _egos(case, gen)
        return {"off": off, "src": s, "tgt": t, "w": None, "n": int(off[-1])}
    if kind == "build":  # an edge table as read: any order, repeats and (if directed) loops kept
        s, t = _rmat_draws(case["n"], case["edges"], gen)
        if not case["directed"]:
            t = torch.where(s == t, (t + 1) % case["n"], t)
        relabel = torch.randperm(case["n"], device=DEV, generator=gen)
        return {"src": relabel[s], "tgt": relabel[t], "w": _weights(case, len(s), gen),
                "n": case["n"]}
    s, t = _edges(case, gen)
    d = {"src": s, "tgt": t, "w": _weights(case, len(s), gen), "n": case["n"]}
    if kind == "pagerank" and case["personalized"]:
        d["pers"] = _pers_vector(case["n"], gen)
    if kind == "batch":
        d["pers"] = _teleport(case["n"], case["batch"], gen)
    if kind == "katz":
        d["alpha"] = _katz_alpha(case["n"], s, t, d["w"])
    if kind == "gradient":
        x = torch.empty(case["n"], dtype=torch.float64, device=DEV).log_normal_(generator=gen)
        d["target"] = x / x.sum()
    return d


# ------------------------------------------------------------------ cases
def _case(kind, name=None, **kw):
    base = {"kind": kind, "graph": "rmat", "directed": True, "weights": "none"}
    base.update(kw)
    if name is not None:
        base["name"] = name
    return base


def _pagerank(n, edges, name=None, **kw):
    d = dict(precision="fp64", tol=1e-12, personalized=False, dangling=0, host=True)
    d.update(kw)
    return _case("pagerank", name, n=n, edges=edges, **d)


def listed():
    return [
        # one survey or classroom network, solved by itself: latency is all
        _pagerank(500, 2500, "pagerank_tiny", graph="er", weights="f64", personalized=True),
        # plain PageRank of an Erdos-Renyi graph of 10,000 nodes and mean degree 10
        _pagerank(10_000, 50_000, "pagerank_small", graph="er", directed=False),
        # a mid-sized weighted network, personalised, host arrays in and out
        _pagerank(300_007, 3_600_000, "pagerank_medium", weights="f64", personalized=True,
                  dangling=1),
        # the headline workload: R-MAT 24, FP32 strengths, mixed precision, in device memory
        _pagerank(1 << 24, 16 << 24, "pagerank_large", weights="f32", precision="mixed",
                  tol=1e-9, host=False),
        # a hundred personalised rankings of one graph at once (recommendation)
        _case("batch", "batch_100", n=1 << 20, edges=16 << 20, batch=100, tol=1e-10),
        # every ego network of a survey in one call
        _case("egos", "egos_2000", graphs=2000, largest=50_000, directed=False),
        # eigenvector centrality of a symmetric network
        _case("eigenvector", "eigenvector", n=1 << 20, edges=16 << 20, directed=False, tol=1e-10,
              precision=0),
        # hubs and authorities of a directed network
        _case("hits", "hits", n=1 << 20, edges=16 << 20),
        # Katz centrality at half of the convergence limit
        _case("katz", "katz", n=1 << 20, edges=16 << 20, weights="f32"),
        # one step of a fit of tie strengths: forward, adjoint and edge gradients
        _case("gradient", "gradient", n=1 << 20, edges=16 << 20, weights="f64"),
        # strong components
        _case("components", "components_strong", n=1 << 21, edges=16 << 21, strong=True),
        # an edge table in host memory to a graph, its rows and its strengths
        _case("build", "build", n=1 << 18, edges=16 << 18, weights="f64"),
    ]


def _spread(rng, lo, hi):
    """A whole number spread over the logarithm of [lo, hi], odd ones among them."""
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["pagerank", "pagerank", "batch", "egos", "eigenvector", "hits", "katz",
                       "gradient", "components", "build"])
    if kind == "pagerank":
        n = _spread(rng, 200, 1 << 23)
        mixed = rng.random() < 0.4
        return _pagerank(n, int(n * rng.uniform(4, 16)),
                         graph="er" if n < 50_000 and rng.random() < 0.5 else "rmat",
                         directed=rng.random() < 0.7,
                         weights=rng.choice(["none", "f32", "f64"]),
                         precision="mixed" if mixed else "fp64",
                         tol=rng.choice([1e-9, 1e-10, 1e-12]),
                         personalized=rng.random() < 0.4, dangling=rng.choice([0, 1]),
                         host=rng.random() < 0.5)
    if kind == "egos":
        return _case(kind, graphs=_spread(rng, 20, 4000), largest=_spread(rng, 100, 50_000),
                     directed=False)
    n = _spread(rng, 500, (1 << 21) if kind == "components" else
                (1 << 18) if kind == "build" else 1 << 20)
    edges = int(n * rng.uniform(4, 16))
    w = rng.choice(["none", "f32", "f64"])
    if kind == "batch":
        return _case(kind, n=n, edges=edges, batch=_spread(rng, 2, 100), tol=1e-10)
    if kind == "eigenvector":
        return _case(kind, n=n, edges=edges, directed=False, weights=w, tol=1e-10,
                     precision=rng.choice([0, 1]))
    if kind == "hits":
        return _case(kind, n=n, edges=edges, weights=w)
    if kind == "katz":
        return _case(kind, n=n, edges=edges, weights=w)
    if kind == "gradient":
        return _case(kind, n=n, edges=edges, weights="f64", directed=rng.random() < 0.7)
    if kind == "components":
        return _case(kind, n=n, edges=edges, strong=rng.random() < 0.6)
    return _case("build", n=n, edges=edges, weights=rng.choice(["none", "f64"]),
                 directed=rng.random() < 0.7)


# ------------------------------------------------------------------ one pass
def prepare(case, seed):
    d = _inputs(case, seed)
    st = {"case": case}
    kind = case["kind"]
    if kind == "build":
        st["src"], st["tgt"] = d["src"].cpu().numpy(), d["tgt"].cpu().numpy()
        st["w"] = None if d["w"] is None else d["w"].double().cpu().numpy()
        return st
    st["g"] = _device_graph(d["n"], d["src"], d["tgt"], d["w"], case["directed"])
    if kind == "pagerank":
        p = d.get("pers")
        if case["host"]:
            st["p"] = None if p is None else p.cpu().numpy()
        else:
            st["p"] = p
            st["out"] = torch.empty(case["n"], dtype=torch.float64, device=DEV)
    elif kind == "batch":
        st["p"] = d["pers"]
        st["out"] = torch.empty_like(d["pers"])
    elif kind == "egos":
        st["off"] = d["off"]
    elif kind == "katz":
        st["alpha"] = d["alpha"]
    elif kind == "gradient":
        st["w"] = d["w"].double().requires_grad_(True)
        st["target"] = d["target"]
    del d
    if case.get("edges", 0) > 1 << 26:
        torch.cuda.empty_cache()
    torch.cuda.synchronize()
    return st


def run(st):
    c = st["case"]
    kind = c["kind"]
    if kind == "build":
        g = K.Graph(c["n"], st["src"], st["tgt"], st["w"], c["directed"])
        off, tgt, w = g.csr(0)
        out = {"off": off.astype(np.int64), "tgt": tgt.astype(np.int64),
               "degree": g.degree(mode=3, weighted=w is not None)}
        if w is not None:
            out["w"] = w
        return out
    g = st["g"]
    if kind == "pagerank":
        kw = dict(damping=DAMPING, directed=c["directed"], weighted=c["weights"] != "none",
                  dangling=c["dangling"], tol=c["tol"],
                  precision=K.PREC_MIXED if c["precision"] == "mixed" else K.PREC_FP64)
        if c["host"]:
            return g.pagerank(personalization=st["p"], **kw)
        p = st["p"]
        g.pagerank_device(st["out"].data_ptr(),
                          personalization_ptr=None if p is None else p.data_ptr(), **kw)
        return st["out"]
    if kind == "batch":
        g.pagerank_batch_device(st["p"].data_ptr(), c["batch"], st["out"].data_ptr(),
                                damping=DAMPING, precision=K.PREC_MIXED, tol=c["tol"])
        return st["out"]
    if kind == "egos":
        x, its, _ = g.pagerank_graphs(st["off"], damping=DAMPING, tol=1e-12)
        return {"scores": x, "iterations": its}
    if kind == "eigenvector":
        x, value, connected = g.eigenvector(mode=3, weighted=c["weights"] != "none", tol=c["tol"],
                                            precision=c["precision"])
        return {"scores": x, "value": value, "connected": connected}
    if kind == "hits":
        h, a, value, unique = g.hits(weighted=c["weights"] != "none")
        return {"hubs": h, "authorities": a, "value": value, "unique": unique}
    if kind == "katz":
        return g.katz(alpha=st["alpha"], beta=1.0, mode=2, weighted=c["weights"] != "none")
    if kind == "gradient":
        w = st["w"]
        w.grad = None
        x = AG.pagerank(w, g, damping=DAMPING, directed=c["directed"], tol=1e-12)
        ((x - st["target"]) ** 2).sum().backward()
        return {"scores": x, "grad": w.grad}
    label, count = g.components(strong=c["strong"])
    return {"membership": label, "count": count}


# ------------------------------------------------------------------ 64-bit results
def _csr(n, row, col, val):
    """A sparse n x n matrix in 64 bits with val at (row, col), repeated entries kept."""
    order = torch.argsort(row, stable=True)
    crow = torch.zeros(n + 1, dtype=torch.int64, device=DEV)
    crow[1:] = torch.bincount(row, minlength=n).cumsum(0)
    v = torch.ones(len(row), dtype=torch.float64, device=DEV) if val is None else val.double()
    return torch.sparse_csr_tensor(crow, col[order], v[order], (n, n), check_invariants=False)


def _pull(d, directed):
    """PageRank's pull matrix (row = target) and the nodes' out-strengths."""
    s, t, w, n = d["src"], d["tgt"], d["w"], d["n"]
    if not directed:
        s, t = torch.cat([s, t]), torch.cat([t, s])
        w = None if w is None else torch.cat([w, w])
    out = torch.bincount(s, weights=None if w is None else w.double(), minlength=n).double()
    return _csr(n, t, s, w), out


def _iterate(A, out, jump, p, tol):
    """PageRank of the columns of p (n x k), each stopped by the L1 change of its own iterate."""
    n, k = p.shape
    x = torch.full((n, k), 1.0 / n, dtype=torch.float64, device=DEV)
    live = torch.ones(k, dtype=torch.bool, device=DEV)
    inv = torch.where(out > 0, 1.0 / out, torch.zeros_like(out))[:, None]
    for _ in range(10_000):
        stuck = x[out == 0].sum(0)
        y = A @ (x * inv) if k > 1 else (A @ (x * inv)[:, 0])[:, None]
        y = DAMPING * (y + stuck * jump) + (1 - DAMPING) * p
        y = y / y.sum(0)
        change = (y - x).abs().sum(0)
        x = torch.where(live, y, x)
        live &= change > tol
        if not bool(live.any()):
            break
    return x


def _exact_egos(d):
    """Every packed graph's own iteration, all at once, each stopped by its own change."""
    off = torch.from_numpy(d["off"]).to(DEV)
    n, k = d["n"], len(off) - 1
    size = off[1:] - off[:-1]
    of = torch.repeat_interleave(torch.arange(k, device=DEV), size)
    A, out = _pull(d, False)
    total = lambda v: torch.zeros(k, dtype=torch.float64, device=DEV).index_add_(0, of, v)  # noqa: E731
    p = 1.0 / size[of].double()
    x = p.clone()
    inv = torch.where(out > 0, 1.0 / out, torch.zeros_like(out))
    live = torch.ones(k, dtype=torch.bool, device=DEV)
    for _ in range(10_000):
        stuck = total(torch.where(out == 0, x, torch.zeros_like(x)))
        y = DAMPING * (A @ (x * inv) + stuck[of] * p) + (1 - DAMPING) * p
        y = y / total(y)[of]
        change = total((y - x).abs())
        x = torch.where(live[of], y, x)
        live &= change > 1e-12
        if not bool(live.any()):
            break
    return {"scores": x, "iterations": None}


def _leading(apply, x):
    """Leading eigenvector (length 1) and eigenvalue of a symmetric non-negative operator;
    None where power iteration does not settle (a leading pair too close to the next)."""
    for k in range(6000):
        y = apply(x)
        y = y / y.norm()
        if k % 20 == 0 and float((y - x).abs().max()) < 1e-15:
            return y, float(y @ apply(y))
        x = y
    return None


def exact(case, seed):
    d = _inputs(case, seed)
    kind, n = case["kind"], d["n"]
    if kind == "components":
        return None  # labels are whole numbers
    if kind == "egos":
        return _exact_egos(d)
    if kind == "build":
        s, t = d["src"].cpu().numpy(), d["tgt"].cpu().numpy()
        w = None if d["w"] is None else d["w"].double().cpu().numpy()
        deg = np.bincount(s, weights=w, minlength=n) + np.bincount(t, weights=w, minlength=n)
        res = {"off": None, "tgt": None, "degree": deg.astype(np.float64)}
        if w is not None:
            if not case["directed"]:  # both directions of every edge, edge by edge
                w = np.repeat(w, 2)
                s, t = np.stack([s, t], 1).ravel(), np.stack([t, s], 1).ravel()
            res["w"] = w[np.lexsort((t, s))]
        return res
    if kind in ("pagerank", "batch", "gradient"):
        A, out = _pull(d, case["directed"])
        uniform = torch.full((n, 1), 1.0 / n, dtype=torch.float64, device=DEV)
        if kind == "gradient":
            x = _iterate(A, out, uniform, uniform, 1e-12)[:, 0]
            return _exact_gradient(case, d, A, out, x)
        p = d.get("pers")
        p = uniform if p is None else p.reshape(-1, n).t().contiguous()
        p = p / p.sum(0)
        jump = uniform if case.get("dangling") == 1 else p
        del d
        x = _iterate(A, out, jump, p, case["tol"])
        return x.t().contiguous() if kind == "batch" else x[:, 0]
    s, t, w = d["src"], d["tgt"], d["w"]
    if kind == "katz":
        A = _csr(n, t, s, w)
        x = torch.ones(n, dtype=torch.float64, device=DEV)
        for _ in range(10_000):
            y = 1.0 + d["alpha"] * (A @ x)
            step = float(((y - x).abs() / y.abs().max()).max())
            x = y
            if step < 1e-16:
                break
        return x / x.norm()
    one = torch.ones(n, dtype=torch.float64, device=DEV)
    if kind == "eigenvector":
        A = _csr(n, torch.cat([s, t]), torch.cat([t, s]), None if w is None else torch.cat([w, w]))
        lead = _leading(lambda v: A @ v + v, one / one.norm())
        if lead is None:
            return None
        x, value = lead
        return {"scores": x / x.max(), "value": value - 1.0, "connected": None}
    A, At = _csr(n, s, t, w), _csr(n, t, s, w)
    lead = _leading(lambda v: At @ (A @ v), one / one.norm())
    if lead is None:
        return None
    a, value = lead
    h = A @ a
    return {"hubs": h / h.max(), "authorities": a / a.max(), "value": value, "unique": None}


def _exact_gradient(case, d, A, out, x):
    """dL/dw of L = |x - target|^2 through the adjoint equation, by autograd-free 64-bit torch."""
    s, t, n = d["src"], d["tgt"], d["n"]
    w = d["w"].double()
    g = 2.0 * (x - d["target"])
    inv = torch.where(out > 0, 1.0 / out, torch.zeros_like(out))
    arcs = [(s, t)] if case["directed"] else [(s, t), (t, s)]
    At = _csr(n, torch.cat([a for a, _ in arcs]), torch.cat([b for _, b in arcs]),
              torch.cat([w] * len(arcs)))
    lam = g.clone()
    for _ in range(10_000):
        new = g + DAMPING * torch.where(out > 0, (At @ lam) * inv, lam.sum() / n)
        step = float((new - lam).abs().sum())
        lam = new
        if step < 1e-17 * max(1.0, float(g.abs().sum())):
            break
    mt = (At @ lam) * inv
    grad = torch.zeros_like(w)
    for a, b in arcs:
        grad += DAMPING * (x * inv)[a] * (lam[b] - mt[a])
    return {"scores": x, "grad": grad}


# ------------------------------------------------------------------ unavoidable work
def work(case):
    kind = case["kind"]
    if kind == "egos":
        # sizes of the power law: mean about 50 (a / (a - 1)) capped at the largest
        mean = 11.0 * 50.0 * (1 - (50.0 / case["largest"]) ** 0.1)
        n = case["graphs"] * mean + case["largest"]
        m = 6.0 * n
        return {"bytes": 36 * (8.0 * m + 40.0 * n), "flops": 36 * (4.0 * m + 6.0 * n)}
    n, m = float(case["n"]), float(case["edges"])
    if kind == "build":
        wb = 0.0 if case["weights"] == "none" else 8.0
        # the table once, the CSR once, the degrees
        return {"bytes": (16.0 + wb) * m + (8.0 + wb) * m + 16.0 * n, "flops": m}
    arcs = m if case["directed"] else 2.0 * m
    wb = {"none": 0.0, "f32": 4.0, "f64": 8.0}[case["weights"]]
    if kind == "components":
        return {"bytes": 8.0 * m + 4.0 * n, "flops": 0.0}
    if kind == "gradient":
        # about 36 sweeps forward and 36 back, and one pass for the gradients
        return {"bytes": 73 * (12.0 * arcs + 32.0 * n), "flops": 73 * (2.0 * arcs + 6.0 * n)}
    # iterations: an operator read and a vector read and written in each
    if kind == "batch":
        k = case["batch"]
        return {"bytes": 30 * (4.0 * arcs + 12.0 * n * k), "flops": 30.0 * k * (2 * arcs + 6 * n)}
    if kind == "pagerank":
        its = 28 if case["tol"] == 1e-9 else 36
        vb = 4.0 if case["precision"] == "mixed" else 8.0
        return {"bytes": its * ((4.0 + wb) * arcs + 5 * vb * n), "flops": its * (2 * arcs + 6 * n)}
    its = {"eigenvector": 14, "hits": 24, "katz": 40}[kind]
    return {"bytes": its * ((4.0 + wb) * arcs + 24.0 * n), "flops": its * (2.0 * arcs + 4.0 * n)}
