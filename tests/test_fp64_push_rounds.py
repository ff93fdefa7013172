"""FP64 tiles of several columns in push rounds: rows around the item classes' limits, every method, whole and fractional
degrees, against the oracle."""
import numpy as np
import pytest

from gde import _lib as L
from gde import api, graphs
from oracle import oracle as O

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def directed():
    """Rows around the limits 8 and 256 of the item classes over a ring of 701 nodes, every seventh entry of them left
    out: rounds on a graph that is not symmetric never pull."""
    a, b = [np.arange(701)], [(np.arange(701) + 1) % 701]
    rng = np.random.default_rng(5)
    for i, d in enumerate([1, 6, 7, 8, 9, 10, 255, 256, 257, 300, 511, 512, 513, 600]):
        a.append(np.full(d, 701 + i))
        b.append(rng.permutation(701)[:d])
    g = graphs._csr_from_undirected(715, np.concatenate(a), np.concatenate(b), False)[0]
    length = np.diff(g.indptr)
    place = np.arange(g.indices.size) - np.repeat(g.indptr[:-1], length)
    keep = (place % 7 != 3) | np.repeat(length < 5, length)
    indptr = np.concatenate([[0], np.cumsum(np.add.reduceat(keep, g.indptr[:-1]))])
    return indptr.astype(np.int64), g.indices[keep]


@pytest.mark.parametrize("W", [2, 4, 8, 16, 32])
@pytest.mark.parametrize("scale", [1.0, 1.25, 1.1])
def test_solves(directed, W, scale):
    indptr, indices = directed
    n, deg = indptr.size - 1, np.diff(indptr) * scale  # (1.1: not exact in FP32)
    ctx = api.Context(0)
    G = api.Graph(indptr, indices, degree=deg, ctx=ctx)
    seeds = np.append(np.random.default_rng(3).integers(0, n, 10), n - 1).astype(np.int32)  # a part-filled tile
    eps, katz = 1e-6, 0.5 / deg.max()
    a = (n, indptr, indices, deg)
    for kind, method, alpha, tau in ((L.PPR, L.LOCAL_GD, 0.1, 0.0), (L.PPR, L.GLOBAL_GD, 0.1, 0.0),
                                     (L.KATZ, L.GLOBAL_GD, katz, 0.0), (L.KATZ, L.LOCAL_GD, katz, 0.0),
                                     (L.HK, L.HK_GLOBAL, 0.0, 5.0), (L.HK, L.HK_LOCAL, 0.0, 5.0),
                                     (L.HK, L.HK_TAYLOR, 0.0, 5.0)):
        res = api.solve(G, kind, method, seeds, eps, prec="fp64", alpha=alpha, tau=tau, tile_w=W)
        assert ctx.last_push()["pull_rounds"] == 0
        for i, s in enumerate(seeds):
            if method == L.HK_TAYLOR:
                xo = O.hk_taylor(*a, int(s), tau, eps)[1]
            elif kind == L.HK:
                xo = O.hk_sor_queue(*a, int(s), tau, eps, 1.0, method == L.HK_LOCAL, sync=True)[1]
            else:
                xo, _, oo = (O.ppr_gd if kind == L.PPR else O.katz_gd)(*a, int(s), alpha, eps, method == L.LOCAL_GD)
                if scale == 1.0:  # (the reference cuts the degrees of fractions)
                    assert abs(res["oper"][i] - oo) <= 1e-9 * oo
            # FP64 sums in another order: a few hundred additions of 2^-53 each
            assert np.abs(res["x"][i] - xo).sum() <= 1e-12 * np.abs(xo).sum()


@pytest.mark.parametrize("F", [2, 4, 8, 24])
def test_feature_push_from_a_list(directed, F):
    """Incremental pushes start sparse; three of the nodes have no neighbours and absorb what they hold."""
    import torch
    rows, indices = directed
    deg = np.concatenate([np.diff(rows), [0, 0, 0]])
    n = deg.size
    indptr = np.concatenate([[0], np.cumsum(deg + 1 + np.arange(n) % 5)])
    col = np.full(indptr[-1], n, np.int32)
    for u in range(n - 3):
        col[indptr[u]:indptr[u] + deg[u]] = indices[rows[u]:rows[u + 1]]
    cand = np.array([0, 5, 100, 705, 714, n - 2], np.int32)
    X = np.zeros((n, F))
    X[cand] = np.random.default_rng(8).standard_normal((cand.size, F))
    P, R = np.zeros_like(X), X.copy()
    O.ign_sync(n, indptr, col, deg, 0.1, 1e-5, 0.5, P, R)
    G = api.Graph(indptr, col, row_len=deg, degree=deg.astype(np.float64))
    Pd, Rd = torch.zeros(n, F, device="cuda", dtype=torch.float64), torch.from_numpy(X).cuda()
    torch.cuda.synchronize()
    api.feature_push(G, L.IGN, Pd, Rd, 1e-5, alpha=0.1, beta=0.5, prec="fp64", cand=cand)
    assert np.abs(Pd.cpu().numpy() - P).sum() <= 1e-12 * np.abs(P).sum()
    assert np.abs(Rd.cpu().numpy() - R).sum() <= 1e-12 * np.abs(P).sum()
