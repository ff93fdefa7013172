"""One graph, several contexts: what a solve makes of it on first use (pull plan, symmetry, reciprocals) serves the others."""
import numpy as np
import pytest

from gde import _lib as L
from gde import api, graphs
from oracle import oracle as O

pytestmark = pytest.mark.gpu


def _view(G, ctx):
    """The same resident graph, solved on through another context."""
    V = object.__new__(api.Graph)
    V.ctx, V.ptr, V.n, V.cap, V.vol = ctx, G.ptr, G.n, G.cap, G.vol
    return V


def test_contexts_solve_on_a_graph_one_after_another():
    """(One after another: launches that fill the device each do not run side by side.)"""
    i, j = np.triu_indices(333, 1)
    keep = np.random.default_rng(6).random(i.size) < 0.3
    g = graphs._csr_from_undirected(333, i[keep], j[keep], False)[0]
    deg = g.degree.astype(np.float64)
    seeds, eps = np.array([0, 9, 100, 332], np.int32), 1e-6
    want = [O.ppr_gd(g.n, g.indptr, g.indices, deg, int(s), 0.1, eps, True) for s in seeds]
    own, other = api.Context(0), api.Context(0)
    for order in ((own, other), (other, own)):
        G = api.Graph(g.indptr, g.indices, ctx=own)
        for ctx in order:
            res = api.solve(_view(G, ctx), L.PPR, L.LOCAL_GD, seeds, eps, prec="fp64", alpha=0.1, tile_w=4)
            for q, (xo, _, oo) in enumerate(want):
                assert res["oper"][q] == oo
                assert np.abs(res["x"][q] - xo).sum() < 1e-12
        G.free()
