"""LocalSOR in block groups: a query per group, several queries in turn per group, rows around the 64-edge pieces."""
import numpy as np
import pytest

from gde import _lib as L
from gde import api, graphs
from oracle import oracle as O
from test_pull_rounds import _hubs

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nq", [1, 3, 170])
@pytest.mark.parametrize("local", [True, False])
def test_every_query_equals_the_oracles(nq, local):
    """170 queries are more than the launch has groups (a group keeps four blocks)."""
    g = _hubs()
    G = api.Graph(g.indptr, g.indices)
    deg = g.degree.astype(np.float64)
    colors = api.graph_colors(G)
    seeds = np.concatenate([np.arange(g.n - 3, g.n), np.arange(nq)])[:nq].astype(np.int32)
    eps = np.minimum(np.geomspace(1e-3, 1e-5, nq), 1.0 / deg[seeds])
    for kind, alpha, katz in ((L.PPR, 0.1, False), (L.KATZ, 0.5 / deg.max(), True)):
        res = api.sor(G, kind, seeds, eps, omega=1.2, local=local, alpha=alpha)
        for i, s in enumerate(seeds):
            xo, _, oo, _ = O.sor_color(g.n, g.indptr, g.indices, deg, int(s), alpha, eps[i], 1.2, local, colors,
                                         katz=katz)
            assert res["oper"][i] == pytest.approx(oo, rel=1e-12)
            # (sweeps are not compared: with omega > 1 additions have both signs, and whether a node passes its
            # threshold between two of them, and so waits in one more sweep unrelaxed, depends on their order)
            assert np.abs(res["x"][i] - xo).sum() <= 1e-10 * max(1.0, np.abs(xo).sum())
