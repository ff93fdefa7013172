"""Solves with a caller's degree array that is not the row lengths: fractions that FP32 holds exactly, and ones that it does not."""
import numpy as np
import pytest

from gde import _lib as L
from gde import api, graphs
from oracle import oracle as O

pytestmark = pytest.mark.gpu

OPER_RTOL = 1e-12
GRAPHS = {}


def _graph(name):
    """(indptr, indices): 333 nodes of about 100 neighbours each (rounds pull), or a ring with hubs."""
    if name not in GRAPHS:
        rng = np.random.default_rng(6)
        if name == "dense":
            i, j = np.triu_indices(333, 1)
            keep = rng.random(i.size) < 0.3
            g = graphs._csr_from_undirected(333, i[keep], j[keep], False)[0]
        else:
            a, b = [np.arange(701)], [(np.arange(701) + 1) % 701]
            for k, d in enumerate((1, 2, 16, 17, 64, 65, 257, 513)):
                a.append(np.full(d, 701 + k))
                b.append(rng.permutation(701)[:d])
            g = graphs._csr_from_undirected(709, np.concatenate(a), np.concatenate(b), False)[0]
        GRAPHS[name] = g
    return GRAPHS[name]


def _local_gd(A, deg, s, alpha, eps):
    """Synchronous local push on the adjacency matrix A: the sum of the pushing nodes' degrees."""
    r = np.zeros(deg.size)
    r[s] = alpha
    oper, act = 0.0, r >= eps * alpha * deg
    while act.any():
        oper += deg[act].sum()
        moved = np.where(act, r, 0.0)
        r = r - moved + A @ ((1 - alpha) * moved / deg)
        act = r >= eps * alpha * deg
    return oper


def _local_cheby(A, deg, s, alpha, eps):
    """Local Chebyshev with a synchronous frontier (ppr_solver.py:582-661): the same sum."""
    r, dx = np.zeros(deg.size), np.zeros(deg.size)
    dx[s] = alpha
    r = r + A @ ((1 - alpha) * dx / deg)
    oper, delta = 0.0, 1 - alpha
    while True:
        act = np.abs(r) >= eps * alpha * deg
        if not act.any():
            return oper
        oper += deg[act].sum()
        delta = 1.0 / (2.0 / (1 - alpha) - delta)
        c = 2.0 * delta / (1 - alpha)
        step = np.where(act, c * r + (c - 1.0) * dx, 0.0)
        dx = np.where(act, step, dx)
        r = r - step + A @ ((1 - alpha) * step / deg)


def _operations(g, deg, kind, method, s, eps):
    if kind == L.HK:
        return O.hk_sor_queue(g.n, g.indptr, g.indices, deg, int(s), 5.0, eps, 1.0, True, sync=True)[3]
    A = np.zeros((g.n, g.n))
    A[np.repeat(np.arange(g.n), g.degree), g.indices] = 1.0
    return (_local_cheby if method == L.LOCAL_CHEBY else _local_gd)(A, deg, int(s), 0.1, eps)


@pytest.mark.parametrize("name", ["dense", "ring"])
@pytest.mark.parametrize("W", [1, 8])
@pytest.mark.parametrize("kind, method", [(L.PPR, L.LOCAL_GD), (L.PPR, L.LOCAL_CHEBY), (L.HK, L.HK_LOCAL)])
def test_operations_of_fractional_degrees(name, W, kind, method):
    """Degrees of 1.25 times the row length: sums of quarters, exact in FP64."""
    g = _graph(name)
    deg = 1.25 * g.degree
    G = api.Graph(g.indptr, g.indices, degree=deg)
    seeds, eps = np.array([3, 200, 332], np.int32), 1e-6
    args = dict(alpha=0.0 if kind == L.HK else 0.1, tau=5.0 if kind == L.HK else 0.0, tile_w=W)
    res = api.solve(G, kind, method, seeds, eps, prec="fp64", **args)
    r32 = api.solve(G, kind, method, seeds, eps, prec="fp32", **args)
    for i, s in enumerate(seeds):
        if W == 1 and method == L.LOCAL_GD:
            # served queries count whole operations, as the reference's GD does (ppr_solver.py:249-250)
            want = O.ppr_gd(g.n, g.indptr, g.indices, deg, int(s), 0.1, eps, True)[2]
        else:
            want = _operations(g, deg, kind, method, s, eps)
        assert res["oper"][i] == want
        # an FP32 rounding at a threshold moves a node's push by a round: a few nodes of the largest degree
        assert abs(r32["oper"][i] - want) <= 6 * deg.max()


@pytest.mark.parametrize("kind, method", [(L.HK, L.HK_LOCAL), (L.PPR, L.LOCAL_GD), (L.KATZ, L.LOCAL_GD)])
def test_fp32_tiles_of_degrees_that_fp32_does_not_hold(kind, method):
    """Degrees of 1.1 times the row length, one eps for all columns: wide tiles push the nodes that one column pushes."""
    g = _graph("dense")
    deg = 1.1 * g.degree
    G = api.Graph(g.indptr, g.indices, degree=deg)
    seeds, eps = np.array([3, 60, 121, 182, 200, 261, 300, 332], np.int32), 1e-5
    katz = 0.5 / deg.max()
    args = dict(alpha=0.0 if kind == L.HK else katz if kind == L.KATZ else 0.1, tau=5.0 if kind == L.HK else 0.0)
    want = api.solve(G, kind, method, seeds, eps, prec="fp64", tile_w=2, **args)["oper"]
    if kind == L.HK:  # (the oracle's own count, to the rounding of a sum in another order)
        for i, s in enumerate(seeds):
            assert want[i] == pytest.approx(_operations(g, deg, kind, method, s, eps), rel=OPER_RTOL)
    for W in (1, 2, 4, 8):
        got = api.solve(G, kind, method, seeds, eps, prec="fp32", tile_w=W, **args)["oper"]
        # an FP32 rounding at a threshold moves a node's push by a round: a few nodes of the largest degree
        assert np.abs(got - want).max() <= 6 * deg.max()
