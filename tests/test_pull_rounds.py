"""Pull rounds, and the row items of push rounds: rows gather their neighbours' push values once a frontier holds a good part of the graph.

Row lengths sit on both sides of every class boundary of the pull plan (16, 64, 256-edge chunks), frontiers
cover the whole graph within a few rounds, and FP64 operation counts must stay those of the oracle's pushes.
"""
import numpy as np
import pytest

from gde import _lib as L
from gde import api, graphs
from oracle import oracle as O

pytestmark = pytest.mark.gpu

FP64_L1 = 1e-12
OPER_RTOL = 1e-12


def _csr(n, a, b):
    return graphs._csr_from_undirected(n, np.asarray(a), np.asarray(b), False)[0]


def _hubs():
    """Hubs whose degrees lie around the row classes' limits, over a ring of 701 nodes."""
    want = [1, 2, 15, 16, 17, 63, 64, 65, 255, 256, 257, 511, 512, 513]
    ring = 701
    a = [np.arange(ring)]
    b = [(np.arange(ring) + 1) % ring]
    rng = np.random.default_rng(5)
    for i, d in enumerate(want):
        a.append(np.full(d, ring + i))
        b.append(rng.permutation(ring)[:d])
    return _csr(ring + len(want), np.concatenate(a), np.concatenate(b))


def _dense():
    """333 nodes of about 100 neighbours: single-column solves pull as well, every node is a hub."""
    rng = np.random.default_rng(6)
    i, j = np.triu_indices(333, 1)
    keep = rng.random(i.size) < 0.3
    return _csr(333, i[keep], j[keep])


GRAPHS = {"hubs": _hubs, "dense": _dense}


def rel_l1(a, b):
    return np.abs(np.asarray(a, np.float64) - b).sum() / max(np.abs(b).sum(), 1e-300)


@pytest.mark.parametrize("graph", list(GRAPHS))
@pytest.mark.parametrize("W", [1, 2, 8, 32])
@pytest.mark.parametrize("method", [L.LOCAL_GD, L.GLOBAL_GD])
def test_gd_counts_and_rows(graph, W, method):
    g = GRAPHS[graph]()
    G = api.Graph(g.indptr, g.indices)
    deg = g.degree.astype(np.float64)
    seeds = graphs.uniform_seeds(g, 9, seed=3)
    eps = np.geomspace(1e-7, 1e-5, 9)
    katz = 0.5 / deg.max()
    for kind, alpha, fn in ((L.PPR, 0.1, O.ppr_gd), (L.KATZ, katz, O.katz_gd)):
        res = api.solve(G, kind, method, seeds, eps, prec="fp64", alpha=alpha, tile_w=W)
        r32 = api.solve(G, kind, method, seeds, eps, prec="fp32", alpha=alpha, tile_w=W)
        for i, s in enumerate(seeds):
            xo, ro, oo = fn(g.n, g.indptr, g.indices, deg, int(s), alpha, eps[i], method == L.LOCAL_GD)
            assert res["oper"][i] == pytest.approx(oo, rel=OPER_RTOL)
            assert rel_l1(res["x"][i], xo) < FP64_L1
            assert np.abs(res["r"][i] - ro).sum() < 1e-12
            # an FP32 rounding at a threshold moves about 2 theta d of l1: a few of those at the largest degree
            theta = eps[i] * (alpha if kind == L.PPR else 1.0)
            assert rel_l1(r32["x"][i], xo) < 2e-6 + 6 * theta * deg.max() / max(np.abs(xo).sum(), 1e-300)


@pytest.mark.parametrize("graph", list(GRAPHS))
@pytest.mark.parametrize("W", [1, 4])
def test_cheby_and_heat_kernel(graph, W):
    g = GRAPHS[graph]()
    G = api.Graph(g.indptr, g.indices)
    deg = g.degree.astype(np.float64)
    seeds = graphs.uniform_seeds(g, 5, seed=4)
    for local in (True, False):
        res = api.solve(G, L.PPR, L.LOCAL_CHEBY if local else L.GLOBAL_CHEBY, seeds, 1e-7, prec="fp64", alpha=0.1,
                        tile_w=W)
        hk = api.solve(G, L.HK, L.HK_LOCAL if local else L.HK_GLOBAL, seeds, 1e-7, prec="fp64", tau=5.0, tile_w=W)
        for i, s in enumerate(seeds):
            xo, _, oo = O.cheby(g.n, g.indptr, g.indices, deg, int(s), 0.1, 1e-7, local, sync=True)
            assert res["oper"][i] == pytest.approx(oo, rel=OPER_RTOL)
            assert rel_l1(res["x"][i], xo) < FP64_L1
            _, xh, _, oh = O.hk_sor_queue(g.n, g.indptr, g.indices, deg, int(s), 5.0, 1e-7, 1.0, local, sync=True)[:4]
            assert hk["oper"][i] == pytest.approx(oh, rel=OPER_RTOL)
            assert rel_l1(hk["x"][i], xh) < FP64_L1


@pytest.mark.parametrize("graph", list(GRAPHS))
@pytest.mark.parametrize("F", [1, 6, 16])
def test_feature_push_on_padded_rows(graph, F):
    """Padded rows (live entries shorter than their capacity), nodes that absorb, every column from the start."""
    import torch
    g = GRAPHS[graph]()
    n = g.n + 3  # three nodes without neighbours
    deg = np.concatenate([g.degree, [0, 0, 0]])
    indptr = np.concatenate([[0], np.cumsum(deg + 1 + np.arange(n) % 5)])
    col = np.full(indptr[-1], n, np.int32)
    for u in range(g.n):
        col[indptr[u]:indptr[u] + deg[u]] = g.indices[g.indptr[u]:g.indptr[u + 1]]
    X = np.random.default_rng(8).standard_normal((n, F))
    P, R = np.zeros_like(X), X.copy()
    want = O.ign_sync(n, indptr, col, deg, 0.1, 1e-6, 0.5, P, R)
    G = api.Graph(indptr, col, row_len=deg, degree=deg.astype(np.float64))
    Pd, Rd = torch.zeros(n, F, dtype=torch.float64, device="cuda"), torch.from_numpy(X).cuda()
    torch.cuda.synchronize()
    res = api.feature_push(G, L.IGN, Pd, Rd, 1e-6, alpha=0.1, beta=0.5, prec="fp64")
    assert np.array_equal(res["oper"], want)
    assert rel_l1(Pd.cpu().numpy(), P) < FP64_L1
    assert np.abs(Rd.cpu().numpy() - R).max() < 1e-12


@pytest.mark.parametrize("W", [1, 8])
def test_rows_that_do_not_match_are_pushed(W):
    """A directed adjacency (row u holds v without row v holding u) never pulls."""
    rng = np.random.default_rng(9)
    n = 400
    rows = [np.sort(rng.choice(n, size=30 + u % 50, replace=False)) for u in range(n)]
    indptr = np.concatenate([[0], np.cumsum([r.size for r in rows])])
    indices = np.concatenate(rows).astype(np.int32)
    deg = np.diff(indptr).astype(np.float64)
    G = api.Graph(indptr, indices)
    seeds = np.array([0, 7, 399, 250], np.int32)
    res = api.solve(G, L.PPR, L.LOCAL_GD, seeds, 1e-6, prec="fp64", alpha=0.1, tile_w=W)
    for i, s in enumerate(seeds):
        xo, _, oo = O.ppr_gd(n, indptr, indices, deg, int(s), 0.1, 1e-6, True)
        assert res["oper"][i] == pytest.approx(oo, rel=OPER_RTOL)
        assert rel_l1(res["x"][i], xo) < FP64_L1


@pytest.mark.parametrize("tuning", [None, {"small_max": 3, "med_max": 70, "chunk": 100},
                                    {"small_max": 16, "med_max": 1000, "chunk": 1000}])
@pytest.mark.parametrize("W", [1, 8])
def test_row_items_and_their_pieces(tuning, W):
    """Rows around every class limit, whole and cut into pieces, pushed by warps of one and of several columns."""
    g = _hubs()
    G = api.Graph(g.indptr, g.indices)
    deg = g.degree.astype(np.float64)
    seeds = np.arange(g.n - 14, g.n, 2, dtype=np.int32)  # the hubs push first
    for eps in (1e-3, 1e-5):
        e = np.minimum(eps, 1.0 / deg[seeds])
        res = api.solve(G, L.PPR, L.LOCAL_GD, seeds, e, prec="fp64", alpha=0.1, tile_w=W, tuning=tuning)
        for i, s in enumerate(seeds):
            xo, _, oo = O.ppr_gd(g.n, g.indptr, g.indices, deg, int(s), 0.1, e[i], True)
            assert res["oper"][i] == pytest.approx(oo, rel=OPER_RTOL)
            assert rel_l1(res["x"][i], xo) < FP64_L1
