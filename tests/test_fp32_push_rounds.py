"""FP32 tiles of several columns in push rounds: rows around the item classes' limits, every method, against the FP64 oracle."""
import numpy as np
import pytest

from gde import _lib as L
from gde import api, graphs
from oracle import oracle as O

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def hubs():
    """Hubs whose degrees lie around the limits 8 and 256 of the item classes, over a ring of 701 nodes."""
    a, b = [np.arange(701)], [(np.arange(701) + 1) % 701]
    rng = np.random.default_rng(5)
    for i, d in enumerate([1, 6, 7, 8, 9, 255, 256, 257, 511, 512, 513]):
        a.append(np.full(d, 701 + i))
        b.append(rng.permutation(701)[:d])
    return graphs._csr_from_undirected(712, np.concatenate(a), np.concatenate(b), False)[0]


def rel_l1(a, b):
    return np.abs(np.asarray(a, np.float64) - b).sum() / max(np.abs(b).sum(), 1e-300)


@pytest.mark.parametrize("W", [2, 4, 8, 16, 32])
def test_solves(hubs, W):
    g = hubs
    G = api.Graph(g.indptr, g.indices)
    deg = g.degree.astype(np.float64)
    seeds = np.concatenate([graphs.uniform_seeds(g, 10, seed=3), [g.n - 1]]).astype(np.int32)  # a part-filled tile
    eps, katz = 1e-6, 0.5 / deg.max()
    a = (g.n, g.indptr, g.indices, deg)
    for kind, method, alpha, tau in ((L.PPR, L.GLOBAL_GD, 0.1, 0.0), (L.KATZ, L.GLOBAL_GD, katz, 0.0),
                                     (L.KATZ, L.LOCAL_GD, katz, 0.0), (L.HK, L.HK_GLOBAL, 0.0, 5.0),
                                     (L.HK, L.HK_LOCAL, 0.0, 5.0), (L.HK, L.HK_TAYLOR, 0.0, 5.0)):
        x = api.solve(G, kind, method, seeds, eps, prec="fp32", alpha=alpha, tau=tau, tile_w=W)["x"]
        for i, s in enumerate(seeds):
            if method == L.HK_TAYLOR:
                xo = O.hk_taylor(*a, int(s), tau, eps)[1]
            elif kind == L.HK:
                xo = O.hk_sor_queue(*a, int(s), tau, eps, 1.0, method == L.HK_LOCAL, sync=True)[1]
            else:
                xo = (O.ppr_gd if kind == L.PPR else O.katz_gd)(*a, int(s), alpha, eps, method == L.LOCAL_GD)[0]
            # an FP32 rounding at a threshold moves about 2 theta d of l1: a few of those at the largest degree
            theta = eps * (alpha if kind == L.PPR else 1.0)
            assert rel_l1(x[i], xo) < 2e-6 + 6 * theta * deg.max() / np.abs(xo).sum()


@pytest.mark.parametrize("F", [2, 4, 8, 24])
def test_feature_push_from_a_list(hubs, F):
    """Incremental pushes start sparse; three of the nodes have no neighbours and absorb what they hold."""
    import torch
    g, n = hubs, hubs.n + 3
    deg = np.concatenate([g.degree, [0, 0, 0]])
    indptr = np.concatenate([[0], np.cumsum(deg + 1 + np.arange(n) % 5)])
    col = np.full(indptr[-1], n, np.int32)
    for u in range(g.n):
        col[indptr[u]:indptr[u] + deg[u]] = g.indices[g.indptr[u]:g.indptr[u + 1]]
    cand = np.array([0, 5, 100, 705, 711, n - 2], np.int32)
    X = np.zeros((n, F))
    X[cand] = np.random.default_rng(8).standard_normal((cand.size, F))
    P, R = np.zeros_like(X), X.copy()
    O.ign_sync(n, indptr, col, deg, 0.1, 1e-5, 0.5, P, R)
    G = api.Graph(indptr, col, row_len=deg, degree=deg.astype(np.float64))
    Pd, Rd = torch.zeros(n, F, device="cuda"), torch.from_numpy(X).float().cuda()
    torch.cuda.synchronize()
    api.feature_push(G, L.IGN, Pd, Rd, 1e-5, alpha=0.1, beta=0.5, prec="fp32", cand=cand)
    # FP32 rounding, and a few roundings at a threshold: each moves at most 2 eps sqrt(d) of a column
    scale = np.abs(P).sum()
    assert np.abs(Pd.cpu().numpy() - P).sum() < 2e-6 * scale + 6 * F * 2e-5 * np.sqrt(deg.max())
