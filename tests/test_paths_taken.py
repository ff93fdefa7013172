"""Which way a launch went: rounds that pulled and the nodes it ran on, where each is expected and where it must not be."""
import numpy as np
import pytest

from gde import _lib as L
from gde import api, graphs

pytestmark = pytest.mark.gpu


def _dense():
    """333 nodes of about 100 neighbours: frontiers cover the graph at once, in one column too."""
    i, j = np.triu_indices(333, 1)
    keep = np.random.default_rng(6).random(i.size) < 0.3
    return graphs._csr_from_undirected(333, i[keep], j[keep], False)[0]


def _leafy():
    """A ring of 40 nodes with 10 leaves each: 440 nodes, 80 once each node's leaves are one."""
    ring = np.arange(40)
    a = np.concatenate([ring, np.repeat(ring, 10)])
    b = np.concatenate([(ring + 1) % 40, np.arange(40, 440)])
    return graphs._csr_from_undirected(440, a, b, False)[0]


def _taken(G, kind, method, prec, W):
    seeds = np.array([0, 5, 20, 39], np.int32)
    alpha = {L.PPR: 0.1, L.KATZ: 1e-3, L.HK: 0.0}[kind]
    api.solve(G, kind, method, seeds, 1e-6, prec=prec, alpha=alpha, tau=5.0 if kind == L.HK else 0.0, tile_w=W)
    return G.ctx.last_push()


@pytest.mark.parametrize("W", [1, 4])
@pytest.mark.parametrize("kind, method", [(L.PPR, L.LOCAL_GD), (L.PPR, L.GLOBAL_GD), (L.PPR, L.LOCAL_CHEBY),
                                          (L.HK, L.HK_LOCAL), (L.HK, L.HK_GLOBAL)])
def test_pull_rounds(kind, method, W):
    g = _dense()
    G = api.Graph(g.indptr, g.indices)
    assert _taken(G, kind, method, "fp64", W)["pull_rounds"] > 0
    whole = method in (L.GLOBAL_GD, L.HK_GLOBAL)
    assert (_taken(G, kind, method, "fp32", W)["pull_rounds"] > 0) == (not whole)
    # an entry taken out of one row only: that row's neighbour is no longer matched
    cut = int(g.indptr[7])
    indptr = g.indptr - (np.arange(g.n + 1) > 7)
    D = api.Graph(indptr, np.delete(g.indices, cut))
    assert _taken(D, kind, method, "fp64", W)["pull_rounds"] == 0


@pytest.mark.parametrize("prec", ["fp64", "fp32"])
def test_merged_leaves(prec):
    g = _leafy()
    G = api.Graph(g.indptr, g.indices)
    for kind, method, W in ((L.PPR, L.LOCAL_GD, 1), (L.PPR, L.LOCAL_GD, 4), (L.KATZ, L.LOCAL_GD, 1),
                            (L.HK, L.HK_LOCAL, 4)):
        assert _taken(G, kind, method, prec, W)["nodes"] == 80
    for kind, method in ((L.PPR, L.GLOBAL_GD), (L.HK, L.HK_TAYLOR)):
        assert _taken(G, kind, method, prec, 4)["nodes"] == (80 if prec == "fp64" else 440)
    assert _taken(G, L.PPR, L.LOCAL_CHEBY, prec, 4)["nodes"] == 440


def test_feature_pushes_pull():
    import torch
    g = _dense()
    deg = g.degree.astype(np.int64)
    G = api.Graph(g.indptr, g.indices, row_len=deg, degree=deg.astype(np.float64))
    P = torch.zeros(g.n, 8, dtype=torch.float64, device="cuda")
    R = torch.ones(g.n, 8, dtype=torch.float64, device="cuda")
    torch.cuda.synchronize()
    api.feature_push(G, L.IGN, P, R, 1e-6, alpha=0.1, beta=0.5, prec="fp64")
    assert G.ctx.last_push()["pull_rounds"] > 0
