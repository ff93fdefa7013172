"""Solves on the graph with merged leaves: seeds with and without twins, every method that uses it, against the oracle."""
import numpy as np
import pytest

from gde import _lib as L
from gde import api, graphs
from oracle import oracle as O

pytestmark = pytest.mark.gpu

FP64_L1 = 1e-12
OPER_RTOL = 1e-12


def _tree_like():
    """40 hubs in a dense core, hub i with 3 i leaves (0, 3, ..., 117), and two nodes joined only to each other."""
    rng = np.random.default_rng(2)
    a, b = np.triu_indices(40, 1)
    keep = rng.random(a.size) < 0.4
    a, b, n = [a[keep]], [b[keep]], 40
    for i in range(40):
        a.append(np.full(3 * i, i))
        b.append(np.arange(n, n + 3 * i))
        n += 3 * i
    a.append(np.array([n]))
    b.append(np.array([n + 1]))
    return graphs._csr_from_undirected(n + 2, np.concatenate(a), np.concatenate(b), False)[0]


def rel_l1(a, b):
    return np.abs(np.asarray(a, np.float64) - b).sum() / max(np.abs(b).sum(), 1e-300)


@pytest.fixture(scope="module")
def graph():
    g = _tree_like()
    # a hub, a hub's leaf among many, a leaf among three, an isolated pair
    return g, api.Graph(g.indptr, g.indices), np.array([39, g.n - 3, 43, g.n - 1, 20], np.int32)


@pytest.mark.parametrize("W", [1, 2, 8])
@pytest.mark.parametrize("method", [L.LOCAL_GD, L.GLOBAL_GD])
@pytest.mark.parametrize("device", [False, True])
def test_gd(graph, W, method, device):
    g, G, seeds = graph
    deg = g.degree.astype(np.float64)
    for kind, alpha, fn in ((L.PPR, 0.1, O.ppr_gd), (L.KATZ, 0.5 / deg.max(), O.katz_gd)):
        for eps in (1e-3, 1e-6):
            e = np.minimum(eps, 1.0 / deg[seeds]) if kind == L.PPR else np.full(seeds.size, eps)
            res = api.solve(G, kind, method, seeds, e, prec="fp64", alpha=alpha, tile_w=W, device_out=device)
            r32 = api.solve(G, kind, method, seeds, e, prec="fp32", alpha=alpha, tile_w=W, device_out=device,
                            want_r=False)
            host = (lambda t: t.cpu().numpy()) if device else np.asarray
            for i, s in enumerate(seeds):
                xo, ro, oo = fn(g.n, g.indptr, g.indices, deg, int(s), alpha, e[i], method == L.LOCAL_GD)
                assert res["oper"][i] == pytest.approx(oo, rel=OPER_RTOL)
                assert np.abs(host(res["x"])[i] - xo).sum() <= FP64_L1 * max(1.0, np.abs(xo).sum())
                assert np.abs(host(res["r"])[i] - ro).sum() < 1e-12
                theta = e[i] * (alpha if kind == L.PPR else 1.0)
                assert np.abs(host(r32["x"])[i] - xo).sum() < 2e-6 + 6 * theta * deg.max()


@pytest.mark.parametrize("W", [1, 8])
@pytest.mark.parametrize("method", [L.LOCAL_GD, L.GLOBAL_GD])
def test_a_seed_below_its_threshold_keeps_its_residual(graph, W, method):
    """Katz with eps * degree > 1: no round runs; the residual is the seed's alone, not its twins'."""
    g, G, seeds = graph
    res = api.solve(G, L.KATZ, method, seeds, 2.0, prec="fp64", alpha=0.5 / g.degree.max(), tile_w=W)
    unit = np.zeros((seeds.size, g.n))
    unit[np.arange(seeds.size), seeds] = 1.0
    assert np.array_equal(res["oper"], np.zeros(seeds.size))
    assert np.array_equal(res["x"], -unit) and np.array_equal(res["r"], unit)


@pytest.mark.parametrize("W", [1, 4])
@pytest.mark.parametrize("method", [L.HK_LOCAL, L.HK_GLOBAL, L.HK_TAYLOR])
def test_heat_kernel(graph, W, method):
    g, G, seeds = graph
    deg = g.degree.astype(np.float64)
    res = api.solve(G, L.HK, method, seeds, 1e-6, prec="fp64", tau=5.0, tile_w=W)
    for i, s in enumerate(seeds):
        if method == L.HK_TAYLOR:
            _, xo = O.hk_taylor(g.n, g.indptr, g.indices, deg, int(s), 5.0, 1e-6)
        else:
            _, xo, _, oo = O.hk_sor_queue(g.n, g.indptr, g.indices, deg, int(s), 5.0, 1e-6, 1.0,
                                          method == L.HK_LOCAL, sync=True)
            assert res["oper"][i] == pytest.approx(oo, rel=OPER_RTOL)
        assert rel_l1(res["x"][i], xo) < FP64_L1


@pytest.mark.parametrize("prec", ["fp64", "fp32"])
def test_served_mix_with_more_queries_than_slots(graph, prec):
    g, G, _ = graph
    deg = g.degree.astype(np.float64)
    rng = np.random.default_rng(7)
    seeds = rng.integers(0, g.n, 60).astype(np.int32)
    kinds = np.array([L.PPR, L.KATZ, L.HK], np.int32)[np.arange(60) % 3]
    alphas = np.where(kinds == L.KATZ, 0.5 / deg.max(), 0.1)
    res = api.serve_mixed(G, kinds, seeds, 1e-6, alphas=alphas, tau=5.0, prec=prec, slots=7)
    for i, s in enumerate(seeds):
        a = (g.n, g.indptr, g.indices, deg, int(s))
        if kinds[i] == L.HK:
            xo = O.hk_sor_queue(*a, 5.0, 1e-6, 1.0, True, sync=True)[1]
        else:
            xo = (O.ppr_gd if kinds[i] == L.PPR else O.katz_gd)(*a, alphas[i], 1e-6, True)[0]
        tol = FP64_L1 if prec == "fp64" else 2e-6 + 6 * 1e-6 * deg.max()
        assert np.abs(res["x"][i] - xo).sum() <= tol * max(1.0, np.abs(xo).sum())
