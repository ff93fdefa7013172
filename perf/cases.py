"""Performance cases of the local push solvers: what users have the library do, over its range of sizes.

A case is a dict of plain values; `family` says which entry point it calls and on which graph:

* ``call``    one drop-in ``ppr_solver.ppr_gd`` call on host arrays (the reference's own call);
* ``solve``   one batched ``gde.api.solve`` (PPR / Katz / heat kernel, every method, FP64 and FP32);
* ``mixed``   ``gde.api.serve_mixed``: PPR, Katz and heat-kernel queries through shared slots;
* ``sor``     ``gde.api.sor``: LocalSOR in multicolour order;
* ``push``    ``gde.api.feature_push``: the initial InstantGNN propagation of every feature column;
* ``update``  ``gde.api.feature_update``: one snapshot (edge batch, repair, incremental push).

Graphs are synthetic, of the shapes that the benchmark and the tests use: Chung-Lu graphs with power-law
degrees and an R-MAT graph.  A graph stays resident between passes, as in a program that serves it; the
queries (seeds, tolerances), the features and the edge batches come from the seed.
"""
from __future__ import annotations

import functools
import math
import os
import sys

import numpy as np
import torch

_PKG = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "faster-local-solver-for-gdes_gb300")
if _PKG not in sys.path:
    sys.path.insert(0, _PKG)

import ppr_solver  # noqa: E402
from gde import _lib as L  # noqa: E402
from gde import api  # noqa: E402

DEV = "cuda:0"
KINDS = {"ppr": L.PPR, "katz": L.KATZ, "hk": L.HK}
METHODS = {"local_gd": L.LOCAL_GD, "global_gd": L.GLOBAL_GD, "local_cheby": L.LOCAL_CHEBY,
           "global_cheby": L.GLOBAL_CHEBY, "hk_local": L.HK_LOCAL, "hk_global": L.HK_GLOBAL, "hk_taylor": L.HK_TAYLOR}
ALPHA = 0.1   # PPR teleport probability of every configuration
TAU = 5.0     # heat-kernel temperature
BETA = 0.5    # InstantGNN exponent

# graph name -> generator arguments
GRAPHS = {
    "cl3k": ("chung_lu", 3_000, 2.1, 8.0, 300.0),            # the smoke test's graph
    "cl100k": ("chung_lu", 100_000, 2.1, 10.0, 2_000.0),     # 87k nodes, 0.7M entries
    "cl2m": ("chung_lu", 5_650_000, 2.1, 1.92, 100_000.0),   # the wiki-talk shape: 2.36M nodes, 9.4M entries
    "rmat20": ("rmat", 20, 16),                              # R-MAT, 0.5M nodes, 16M entries
    "rmat17": ("rmat", 17, 16),
    "cl169k": ("chung_lu", 169_343, 2.3, 14.5, 20_000.0),    # the ogbn-arxiv shape: 2.3M entries
}


def listed():
    return [
        # the smallest call: one seed on a graph of a few thousand nodes, host arrays in and out
        {"name": "call_tiny", "family": "call", "graph": "cl3k", "eps": 1e-5},
        # a reference user's loop over seeds: one drop-in call on the 100k-node graph
        {"name": "call_100k", "family": "call", "graph": "cl100k", "eps": 1e-6},
        # one interactive query on the large graph, FP32, row left on the device
        {"name": "one_query_2m", "family": "solve", "graph": "cl2m", "kind": "ppr", "method": "local_gd",
         "prec": "fp32", "nq": 1, "eps_lo": 1e-7, "eps_hi": 1e-7, "tile_w": 0, "slots": 0},
        # 50 seeds in FP64 with solutions and residuals: the reference's experiment on its mid-size graphs
        {"name": "gd_fp64_100k", "family": "solve", "graph": "cl100k", "kind": "ppr", "method": "local_gd",
         "prec": "fp64", "nq": 50, "eps_lo": 1e-6, "eps_hi": 1e-6, "tile_w": 0, "slots": 0, "want_r": True},
        # throughput serving on the large graph: the benchmark's default workload at half its batch
        {"name": "served_2m", "family": "solve", "graph": "cl2m", "kind": "ppr", "method": "local_gd",
         "prec": "fp32", "nq": 512, "eps_lo": 1e-7, "eps_hi": 1e-7, "tile_w": 0, "slots": 64},
        # many seeds of uneven tolerance in node x seed tiles
        {"name": "tiles_100k", "family": "solve", "graph": "cl100k", "kind": "ppr", "method": "local_gd",
         "prec": "fp64", "nq": 256, "eps_lo": 1e-8, "eps_hi": 1e-5, "tile_w": 8, "slots": 0},
        # local Chebyshev, FP64, a handful of seeds
        {"name": "cheby_2m", "family": "solve", "graph": "cl2m", "kind": "ppr", "method": "local_cheby",
         "prec": "fp64", "nq": 12, "eps_lo": 1e-7, "eps_hi": 1e-7, "tile_w": 0, "slots": 0},
        # the global method (every node each round), FP32
        {"name": "global_2m", "family": "solve", "graph": "cl2m", "kind": "ppr", "method": "global_gd",
         "prec": "fp32", "nq": 8, "eps_lo": 1e-7, "eps_hi": 1e-7, "tile_w": 0, "slots": 0},
        # a request mix: 60% PPR, 25% Katz, 15% heat kernel through shared slots, FP64
        {"name": "mixed_rmat", "family": "mixed", "graph": "rmat20", "prec": "fp64", "nq": 128, "eps_lo": 1e-8,
         "eps_hi": 1e-5, "slots": 64},
        # LocalSOR (omega > 1), FP64
        {"name": "sor_100k", "family": "sor", "graph": "cl100k", "kind": "ppr", "nq": 6, "eps": 1e-6, "omega": 1.3},
        # InstantGNN: initial propagation of all feature columns, FP64 (the drop-in's precision)
        {"name": "push_169k", "family": "push", "graph": "cl169k", "cols": 128, "eps": 1e-6},
        # InstantGNN: one snapshot with edges arriving and leaving, FP64
        {"name": "update_169k", "family": "update", "graph": "cl169k", "cols": 64, "edges": 8_000, "eps": 1e-6},
    ]


def _log(rng, lo, hi):
    return float(math.exp(rng.uniform(math.log(lo), math.log(hi))))


def draw(rng):
    family = rng.choice(["call", "solve", "solve", "solve", "batch", "mixed", "sor", "push", "update"])
    if family == "call":
        graph = rng.choice(["cl3k", "cl100k", "rmat17"])
        return {"family": "call", "graph": graph, "eps": _log(rng, 1e-6, 1e-4)}
    if family == "batch":  # served local GD, FP32, the graphs and batch sizes of the serving workloads
        graph = rng.choice(["cl100k", "cl2m", "rmat20"])
        lo = _log(rng, 1e-7, 1e-6)
        return {"family": "solve", "graph": graph, "kind": "ppr", "method": "local_gd", "prec": "fp32",
                "nq": int(_log(rng, 8, 256)), "eps_lo": lo, "eps_hi": lo * rng.choice([1.0, 10.0]), "tile_w": 0,
                "slots": rng.choice([0, 32, 64])}
    if family == "solve":
        graph = rng.choice(["cl3k", "cl100k", "cl2m", "rmat17"])
        kind, method = rng.choice([("ppr", "local_gd"), ("ppr", "global_gd"), ("ppr", "local_cheby"),
                                   ("ppr", "global_cheby"), ("katz", "local_gd"), ("katz", "global_gd"),
                                   ("hk", "hk_local"), ("hk", "hk_global"), ("hk", "hk_taylor")])
        nq = int(_log(rng, 1, 9 if graph == "cl2m" else 70))
        lo = _log(rng, 1e-7, 1e-5)
        return {"family": "solve", "graph": graph, "kind": kind, "method": method, "prec": "fp64", "nq": nq,
                "eps_lo": lo, "eps_hi": lo, "tile_w": rng.choice([0, 0, 2, 4, 8, 16]), "slots": 0,
                "want_r": rng.choice([True, False])}
    if family == "mixed":
        return {"family": "mixed", "graph": rng.choice(["cl100k", "rmat17", "rmat20"]),
                "prec": rng.choice(["fp32", "fp64"]), "nq": int(_log(rng, 8, 100)), "eps_lo": _log(rng, 1e-8, 1e-6),
                "eps_hi": 1e-5, "slots": rng.choice([16, 32, 64])}
    if family == "sor":
        return {"family": "sor", "graph": rng.choice(["cl3k", "cl100k"]), "kind": "ppr", "nq": int(_log(rng, 1, 8)),
                "eps": _log(rng, 1e-6, 1e-4), "omega": round(rng.uniform(0.9, 1.5), 3)}
    if family == "push":
        return {"family": "push", "graph": "cl169k", "cols": int(_log(rng, 1, 128)), "eps": _log(rng, 1e-6, 1e-4)}
    return {"family": "update", "graph": "cl169k", "cols": int(_log(rng, 1, 64)), "edges": int(_log(rng, 100, 20_000)),
            "eps": _log(rng, 1e-6, 1e-4)}


# ---------------------------------------------------------------------------
# Graphs
# ---------------------------------------------------------------------------
def _csr(n, a, b, drop_isolated):
    """Symmetric CSR of an undirected edge list: no self-loops, no repeats, degree-0 nodes dropped on request."""
    keep = a != b
    key = torch.unique(torch.minimum(a, b)[keep] * n + torch.maximum(a, b)[keep])
    lo, hi = key // n, key % n
    if drop_isolated:
        alive = (torch.bincount(lo, minlength=n) + torch.bincount(hi, minlength=n)) > 0
        new = torch.cumsum(alive.long(), 0) - 1
        lo, hi, n = new[lo], new[hi], int(alive.sum())
    both = torch.sort(torch.cat([lo * n + hi, hi * n + lo])).values
    indptr = torch.zeros(n + 1, dtype=torch.int64, device=both.device)
    indptr[1:] = torch.cumsum(torch.bincount(both // n, minlength=n), 0)
    return indptr.cpu().numpy(), (both % n).int().cpu().numpy()


@functools.lru_cache(maxsize=None)
def _arrays(name):
    """Host CSR arrays (indptr int64, indices int32) of a named graph."""
    what, *args = GRAPHS[name]
    if what == "rmat":  # a = 0.57, b = c = 0.19
        scale, factor = args
        gen = torch.Generator(device=DEV).manual_seed(0)
        m = factor * (1 << scale) // 2
        s = torch.zeros(m, dtype=torch.int64, device=DEV)
        d = torch.zeros(m, dtype=torch.int64, device=DEV)
        for _ in range(scale):
            r = torch.rand(m, generator=gen, device=DEV, dtype=torch.float64)
            s = 2 * s + (r >= 0.76)
            d = 2 * d + (((r >= 0.57) & (r < 0.76)) | (r >= 0.95))
        return _csr(1 << scale, s, d, True)
    n, exponent, mean, most = args
    rng = np.random.default_rng(0)
    w = (1.0 - rng.random(n)) ** (-1.0 / (exponent - 1.0))
    w *= mean / w.mean()
    np.minimum(w, most, out=w)
    cdf = torch.from_numpy(np.cumsum(w / w.sum())).to(DEV)
    m = int(round(w.sum() / 2.0))
    a, b = (torch.searchsorted(cdf, torch.from_numpy(rng.random(m)).to(DEV), right=True).clamp_(max=n - 1)
            for _ in range(2))
    return _csr(n, a, b, name != "cl169k")


@functools.lru_cache(maxsize=None)
def _resident(name):
    return api.Graph(*_arrays(name))


@functools.lru_cache(maxsize=None)
def _degree(name):
    return np.diff(_arrays(name)[0])


def _seeds(name, count, rng):
    return rng.choice(np.flatnonzero(_degree(name) > 0), size=count).astype(np.int32)


def _eps(case, rng, degree):
    lo, hi = case["eps_lo"], case["eps_hi"]
    e = np.exp(rng.uniform(math.log(lo), math.log(hi), case["nq"])) if hi > lo else np.full(case["nq"], lo)
    return np.minimum(e, 1.0 / degree)  # the solvers' precondition eps * degree[s] <= 1


def _katz_alpha(name):
    return 0.5 / float(_degree(name).max())


def _queries(case, seed):
    rng = np.random.default_rng([seed, 1])
    name = case["graph"]
    if case["family"] == "mixed":
        # heat-kernel queries keep every residual in the slots' precision: in FP32 a rounding at a hub's threshold
        # shows in the row, so the FP32 mix leaves them out
        share = [0.60, 0.25, 0.15] if case["prec"] == "fp64" else [0.70, 0.30, 0.0]
        kinds = rng.choice(np.array([L.PPR, L.KATZ, L.HK], np.int32), size=case["nq"], p=share)
        seeds = _seeds(name, case["nq"], rng)
        return kinds, seeds, _eps(case, rng, _degree(name)[seeds]), np.where(kinds == L.KATZ, _katz_alpha(name), ALPHA)
    nq = case.get("nq", 1)
    seeds = _seeds(name, nq, rng)
    eps = _eps(case, rng, _degree(name)[seeds]) if case["family"] == "solve" else np.full(nq, case["eps"])
    return seeds, np.minimum(eps, 1.0 / _degree(name)[seeds])


def _snapshot(case, seed):
    """A padded CSR and an edge batch: half of the batch's edges are in the graph (they leave), half are not."""
    indptr, indices = _arrays(case["graph"])
    n = indptr.shape[0] - 1
    src = np.repeat(np.arange(n), np.diff(indptr))
    up = np.flatnonzero(src < indices)
    rng = np.random.default_rng([seed, 2])
    pick = rng.permutation(up)[:2 * (case["edges"] // 2)]
    lost = np.bincount(np.concatenate([src[pick], indices[pick]]), minlength=n)
    keep = np.diff(indptr) - lost >= 2  # both endpoints keep neighbours whatever order the batch runs in
    pick = pick[keep[src[pick]] & keep[indices[pick]]]
    leave, arrive = pick[: pick.size // 2], pick[pick.size // 2:]
    key = np.minimum(src, indices).astype(np.int64) * n + np.maximum(src, indices)
    out = np.isin(key, src[arrive].astype(np.int64) * n + indices[arrive])
    degree = np.diff(indptr) - np.bincount(src[out], minlength=n)
    order = np.lexsort((out, src))  # live entries first in each row, then slack
    col = np.where(out[order], n, indices[order]).astype(np.int32)
    both = rng.permutation(np.concatenate([leave, arrive]))
    return (indptr, col, degree.astype(np.int64), src[both].astype(np.int32), indices[both].astype(np.int32),
            src[leave], indices[leave], src[arrive], indices[arrive])


def _features(case, seed, n):
    gen = torch.Generator(device=DEV).manual_seed(seed)
    return torch.randn(n, case["cols"], generator=gen, device=DEV, dtype=torch.float64)


@functools.lru_cache(maxsize=None)
def _padded(name):
    """The whole graph in the padded layout (every slot live)."""
    indptr, indices = _arrays(name)
    deg = np.diff(indptr).astype(np.int64)
    return api.Graph(indptr, indices, row_len=deg, degree=deg.astype(np.float64))


# ---------------------------------------------------------------------------
# The cases
# ---------------------------------------------------------------------------
def prepare(case, seed):
    family = case["family"]
    if family == "call":
        seeds, eps = _queries(case, seed)
        return {"case": case, "arrays": _arrays(case["graph"]), "degree": _degree(case["graph"]),
                "seed": int(seeds[0]), "eps": float(eps[0])}
    if family == "push":
        G = _padded(case["graph"])
        X = _features(case, seed, G.n)
        return {"case": case, "G": G, "X": X, "P": torch.zeros_like(X), "R": torch.zeros_like(X)}
    if family == "update":
        indptr, col, degree, us, vs = _snapshot(case, seed)[:5]
        G = api.Graph(indptr, col, row_len=degree, degree=degree.astype(np.float64))
        X = _features(case, seed, G.n)
        P, R = torch.zeros_like(X), X.clone()
        torch.cuda.synchronize()
        api.feature_push(G, L.IGN, P, R, case["eps"], alpha=ALPHA, beta=BETA, prec="fp64")
        return {"case": case, "G": G, "col": col, "degree": degree, "us": us, "vs": vs, "X": X, "P": P, "R": R}
    G = _resident(case["graph"])
    if family == "sor":
        return {"case": case, "G": G, "queries": _queries(case, seed)}
    out = torch.float32 if case["prec"] == "fp32" else torch.float64
    x = torch.empty((case["nq"], G.n), dtype=out, device=DEV)
    return {"case": case, "G": G, "queries": _queries(case, seed), "x": x}


def run(state):
    case, family = state["case"], state["case"]["family"]
    if family == "call":
        indptr, indices = state["arrays"]
        x, r, oper, _ = ppr_solver.ppr_gd(indptr.shape[0] - 1, indptr, indices, state["degree"], state["seed"], ALPHA,
                                          state["eps"], True)
        return {"x": x, "r": r, "oper": oper}
    G = state["G"]
    if family == "push":
        # a program propagates fresh features: r = x, p = 0 (the library's stream starts after the copies)
        state["P"].zero_()
        state["R"].copy_(state["X"])
        torch.cuda.current_stream().synchronize()
        api.feature_push(G, L.IGN, state["P"], state["R"], case["eps"], alpha=ALPHA, beta=BETA, prec="fp64")
        return {"p": state["P"], "r": state["R"]}
    if family == "update":
        api.feature_update(G, L.IGN, state["col"], state["degree"], state["us"], state["vs"], False, state["P"],
                           state["R"], state["X"], case["eps"], alpha=ALPHA, beta=BETA, prec="fp64")
        return {"p": state["P"], "r": state["R"], "col": state["col"], "degree": state["degree"]}
    if family == "mixed":
        kinds, seeds, eps, alphas = state["queries"]
        api.serve_mixed(G, kinds, seeds, eps, alphas=alphas, tau=TAU, prec=case["prec"], x_out=state["x"],
                        device_out=True, slots=case["slots"])
        return {"x": state["x"]}
    seeds, eps = state["queries"]
    if family == "sor":
        res = api.sor(G, KINDS[case["kind"]], seeds, eps, omega=case["omega"], alpha=ALPHA, prec="fp64",
                      device_out=True)
        return {"x": res["x"], "r": res["r"], "oper": res["oper"]}
    kind = KINDS[case["kind"]]
    res = api.solve(G, kind, METHODS[case["method"]], seeds, eps, prec=case["prec"], x_out=state["x"],
                    want_r=case.get("want_r", False), device_out=True, tile_w=case["tile_w"],
                    alpha=0.0 if kind == L.HK else ALPHA if kind == L.PPR else _katz_alpha(case["graph"]),
                    tau=TAU if kind == L.HK else 0.0, tuning={"slots": case["slots"]} if case["slots"] else None)
    out = {"x": res["x"]}
    if case.get("want_r", False):
        out["r"] = res["r"]
    if case["prec"] == "fp64":
        out["oper"] = res["oper"]
    return out


def work(case):
    """The graph read once, the seeds or features read once, every output row written once; one multiply and one add
    per graph entry and column."""
    indptr, indices = _arrays(case["graph"])
    n, nnz = indptr.shape[0] - 1, indices.shape[0]
    graph = 4 * nnz + 8 * n
    if case["family"] in ("push", "update"):
        moved = (3 if case["family"] == "push" else 5) * 8 * n * case["cols"]
        return {"bytes": graph + moved, "flops": 2 * nnz * case["cols"]}
    nq = case.get("nq", 1)
    es = 4 if case.get("prec") == "fp32" else 8
    rows = 2 if case["family"] in ("call", "sor") or case.get("want_r", False) else 1
    if rows == 2 and case.get("method") in ("hk_local", "hk_global"):
        rows = 3  # the residual is two level buffers
    return {"bytes": graph + rows * nq * n * es, "flops": 2 * nnz * nq}


# ---------------------------------------------------------------------------
# The same results in 64 bits, with torch
# ---------------------------------------------------------------------------
class _Adj:
    """Adjacency of a CSR graph on the device: its rows, and its product with a dense [n, k] matrix."""

    def __init__(self, indptr, indices):
        self.indptr = torch.from_numpy(np.asarray(indptr, dtype=np.int64)).to(DEV)
        self.indices = torch.from_numpy(np.asarray(indices, dtype=np.int64)).to(DEV)
        self.n = self.indptr.shape[0] - 1
        self.len = self.indptr[1:] - self.indptr[:-1]
        self.deg = self.len.double()
        self._m = torch.sparse_csr_tensor(self.indptr, self.indices,
                                          torch.ones(self.indices.shape[0], dtype=torch.float64, device=DEV),
                                          size=(self.n, self.n))

    def mm(self, y):
        return self._m @ y

    def edges(self, u):
        """Every neighbour of the nodes u, and the position in u that it belongs to."""
        k = self.len[u]
        at = torch.repeat_interleave(torch.arange(u.shape[0], device=DEV), k)
        first = torch.cumsum(k, 0) - k
        return self.indices[self.indptr[u][at] + torch.arange(at.shape[0], device=DEV) - first[at]], at


def _local_gd(A, seeds, r0, theta, katz_alpha=None):
    """Synchronous local push over a list of active (query, node) pairs -> x, r [q, n], operation counts."""
    q, n = seeds.shape[0], A.n
    X = torch.zeros(q * n, dtype=torch.float64, device=DEV)
    R = torch.zeros(q * n, dtype=torch.float64, device=DEV)
    oper = torch.zeros(q, dtype=torch.float64, device=DEV)
    act = torch.arange(q, device=DEV) * n + seeds
    R[act] = r0
    act = act[R[act] >= theta * A.deg[seeds]]
    while act.numel():
        r = R[act]
        R[act] = 0.0
        X[act] += r
        u, row = act % n, act // n
        oper.index_add_(0, row, A.deg[u])
        p = katz_alpha * r if katz_alpha is not None else (1.0 - ALPHA) * r / A.deg[u]
        cuts = torch.cumsum(A.len[u], 0) // 50_000_000  # bounded pieces of the round's edges
        found = []
        for c in range(int(cuts[-1]) + 1):
            part = slice(None) if int(cuts[-1]) == 0 else cuts == c
            v, at = A.edges(u[part])
            flat = row[part][at] * n + v
            R.index_add_(0, flat, p[part][at])
            found.append(flat)
        hit = torch.cat([f[R[f] >= theta[f // n] * A.deg[f % n]] for f in found])
        act = torch.unique(hit)
    return X.view(q, n), R.view(q, n), oper


def _dense(A, method, seeds, theta, alpha, katz):
    """Chebyshev (synchronous frontier) and gradient descent, local or global, on dense [n, k] columns."""
    k, n = seeds.shape[0], A.n
    deg = A.deg[:, None]
    cols = torch.arange(k, device=DEV)
    X, R, D = (torch.zeros(n, k, dtype=torch.float64, device=DEV) for _ in range(3))
    oper = torch.zeros(k, dtype=torch.float64, device=DEV)
    cheby, local = "cheby" in method, method.startswith("local")
    if cheby:
        X[seeds, cols] = alpha
        D[seeds, cols] = alpha
        Y = torch.zeros_like(R)
        Y[seeds, cols] = (1.0 - alpha) * alpha / A.deg[seeds]
        R = A.mm(Y)
    else:
        R[seeds, cols] = 1.0 if katz else alpha
    delta = 1.0 - alpha
    while True:
        above = R.abs() >= theta * deg
        live = above.any(0)
        if not bool(live.any()):
            return X.T, R.T, oper
        if cheby:
            delta = 1.0 / (2.0 / (1.0 - alpha) - delta)
            c = 2.0 * delta / (1.0 - alpha)
            step = c * R + (c - 1.0) * D
            act = above if local else live.expand_as(above)
            step = torch.where(act, step, 0.0)
            D = torch.where(act, step, D)
        else:
            step = torch.where(above if local else live, R, 0.0)
        R = R - step
        X += step
        oper += (above * deg).sum(0) if local else live * float(n + A.deg.sum())
        R += A.mm(alpha * step if katz else (1.0 - alpha) * step / deg)


def _estimate_n(tau, eps):
    k = math.ceil(tau - 1)
    t = tau
    for i in range(k):
        t *= tau / (i + 2)
    cur = t * ((k + 2.0) / (k + 2.0 - tau))
    limit = eps * math.exp(tau)
    for i in range(k, 1000 * (k + 1)):
        if cur < limit:
            return i
        cur *= ((k + 2.0 - tau) * tau / (k + 2.0) ** 2) * ((k + 3.0) / (k + 3.0 - tau))
    return 1000 * (k + 1)


def _heat(A, method, seeds, eps):
    """Heat-kernel levels for queries of one eps -> x [k, n], operation counts."""
    k, n = seeds.shape[0], A.n
    deg = A.deg[:, None]
    taylor = method == "hk_taylor"
    N = _estimate_n(TAU, eps if taylor else 0.5 * eps)
    psi = [1.0] * (N + 2)
    for i in range(N - 1, -1, -1):
        psi[i] = psi[i + 1] * TAU / (i + 1.0) + 1.0
    X = torch.zeros(n, k, dtype=torch.float64, device=DEV)
    R = torch.zeros_like(X)
    R[seeds, torch.arange(k, device=DEV)] = 1.0
    oper = torch.zeros(k, dtype=torch.float64, device=DEV)
    for j in range(N + 1 if taylor else N):
        act = R != 0 if method != "hk_local" else R.abs() >= ((math.exp(TAU) * eps * deg) / N) / psi[j]
        if not bool(act.any()):
            break
        moved = torch.where(act, R, 0.0)
        X += moved
        oper += (act * deg).sum(0) if method == "hk_local" else float(A.deg.sum() + n)
        if taylor and j == N:
            break
        last = not taylor and j + 1 == N
        if last:
            X += A.mm(moved / deg)
        else:
            R = A.mm((TAU / (j + 1.0)) * moved / deg)
    return X.T / math.exp(TAU), oper


def _features_push(deg, mm, P, R, eps):
    """Synchronous InstantGNN push on dense [n, F] columns; nodes without neighbours absorb their residual."""
    lone = deg == 0
    P[lone] = torch.where(R[lone] != 0, R[lone], P[lone])
    R[lone] = 0.0
    d = deg.clamp(min=1.0)[:, None]
    thr = torch.where(lone[:, None], math.inf, d ** (1.0 - BETA) * eps)
    while True:
        act = R.abs() >= thr
        if not bool(act.any()):
            return P, R
        moved = torch.where(act, R, 0.0)
        P += ALPHA * moved
        R = R - moved + mm((1.0 - ALPHA) * moved / d ** (1.0 - BETA)) / d ** BETA


def _exact_update(case, seed):
    indptr, col, degree, us, vs, lu, lv, au, av = _snapshot(case, seed)
    n = indptr.shape[0] - 1

    def csr(live):
        src = np.repeat(np.arange(n), np.diff(indptr))
        u, v = src[live], live_col[live]
        o = np.lexsort((v, u))
        ptr = np.concatenate([[0], np.cumsum(np.bincount(u, minlength=n))])
        return _Adj(ptr, v[o])

    live_col = col.astype(np.int64)
    A0 = csr(col != n)
    X = _features(case, seed, n)
    P, R = _features_push(A0.deg, A0.mm, torch.zeros_like(X), X.clone(), case["eps"])
    key = lambda u, v: np.minimum(u, v).astype(np.int64) * n + np.maximum(u, v)  # noqa: E731
    base_ptr, base = _arrays(case["graph"])
    src = np.repeat(np.arange(n), np.diff(base_ptr))
    live_col = base.astype(np.int64)
    A1 = csr(~np.isin(key(src, base), key(lu, lv)))
    iu, iv = (torch.from_numpy(np.concatenate(p).astype(np.int64)).to(DEV) for p in ((au, av), (av, au)))
    du, dv = (torch.from_numpy(np.concatenate(p).astype(np.int64)).to(DEV) for p in ((lu, lv), (lv, lu)))
    touched = torch.zeros(n, dtype=torch.bool, device=DEV)
    touched[iu] = True  # only nodes that gained an edge are repaired
    t = touched[:, None]
    od, d = A0.deg.clamp(min=1.0)[:, None], A1.deg.clamp(min=1.0)[:, None]
    P = torch.where(t, P * (d / od) ** (1 - BETA), P)
    R = torch.where(t, R + P * (od ** (1 - BETA) - d ** (1 - BETA)) / d ** (1 - BETA) / ALPHA, R)
    dr = (P + ALPHA * R - ALPHA * X) * (od ** BETA - d ** BETA) / d ** BETA
    share = (1.0 - ALPHA) * P / d ** (1 - BETA)
    gain = torch.zeros_like(P).index_add_(0, iu, share[iv]).index_add_(0, du, share[dv], alpha=-1.0)
    R = torch.where(t, R + (dr + gain / d ** BETA) / ALPHA, R)
    P, _ = _features_push(A1.deg, A1.mm, P, R, case["eps"])
    # a node whose threshold fell with its degree keeps its residual until a push reaches it, so r has no such value
    return {"p": P, "r": None, "col": None, "degree": None}


@functools.lru_cache(maxsize=1)
def _adjacency(name):
    return _Adj(*_arrays(name))


def exact(case, seed):
    family = case["family"]
    if family == "sor":
        return None  # its order is that of a colouring the library makes
    if family == "update":
        return _exact_update(case, seed)
    A = _adjacency(case["graph"])
    if family == "push":
        X = _features(case, seed, A.n)
        P, R = _features_push(A.deg, A.mm, torch.zeros_like(X), X.clone(), case["eps"])
        return {"p": P, "r": R}
    q = _queries(case, seed)
    kinds, alphas = (q[0], q[3]) if family == "mixed" else (None, None)
    seeds, eps = (q[1], q[2]) if family == "mixed" else q
    nq, n = seeds.shape[0], A.n
    kind_of = np.full(nq, L.PPR if family == "call" else KINDS.get(case.get("kind"), L.PPR)) if kinds is None else kinds
    method = case.get("method", "local_gd")
    x = torch.zeros(nq, n, dtype=torch.float64, device=DEV)
    want_r = family == "call" or case.get("want_r", False)
    hk_levels = family == "solve" and method in ("hk_local", "hk_global")
    r = torch.zeros(nq, n, dtype=torch.float64, device=DEV) if want_r and not hk_levels else None
    oper = torch.zeros(nq, dtype=torch.float64, device=DEV)
    for kind in (L.PPR, L.KATZ, L.HK):
        mine = np.flatnonzero(kind_of == kind)
        sparse = method == "local_gd" and n > 1_000_000  # its frontiers are a small part of such a graph
        step = 256 if sparse else 32
        groups = [mine[i:i + step] for i in range(0, mine.size, step)]
        if kind == L.HK:
            groups = [np.array([i]) for i in mine] if family == "mixed" else groups
        for g in groups:
            at = torch.from_numpy(g).to(DEV)
            s = torch.from_numpy(seeds[g].astype(np.int64)).to(DEV)
            e = torch.from_numpy(eps[g]).to(DEV)
            if kind == L.HK:
                parts = [np.flatnonzero(eps[g] == v) for v in np.unique(eps[g])]
                for p in parts:
                    xi, oi = _heat(A, "hk_local" if family == "mixed" else method, s[p], float(eps[g][p[0]]))
                    x[at[p]], oper[at[p]] = xi, oi
                continue
            katz = kind == L.KATZ
            alpha = _katz_alpha(case["graph"]) if katz else ALPHA
            theta = e if katz else e * ALPHA
            if sparse:
                xi, ri, oi = _local_gd(A, s, 1.0 if katz else ALPHA, theta, alpha if katz else None)
            else:
                xi, ri, oi = _dense(A, method, s, theta, alpha, katz)
            if katz:
                xi = xi.clone()
                xi[torch.arange(g.size, device=DEV), s] -= 1.0
            x[at], oper[at] = xi, oi
            if r is not None:
                r[at] = ri
    if family == "call":
        return {"x": x[0], "r": r[0], "oper": None}
    out = {"x": x}
    if want_r:
        out["r"] = r
    if family == "solve" and case["prec"] == "fp64":
        out["oper"] = None if method == "hk_taylor" else oper
    return out
