"""Device memory that a merged copy of the graph holds goes back to a call that needs it."""
import numpy as np
import pytest

from gde import _lib as L
from gde import api

pytestmark = pytest.mark.gpu

RING, LEAVES = 3_000_000, 1_000_000  # a quarter of the nodes merge: the copy holds about 180 MB


@pytest.fixture(scope="module")
def arrays():
    """A ring; node 0 holds the leaves too."""
    n = RING + LEAVES
    deg = np.concatenate([[LEAVES + 2], np.full(RING - 1, 2), np.ones(LEAVES, np.int64)])
    indptr = np.concatenate([[0], np.cumsum(deg)])
    i = np.arange(1, RING)
    ring = np.stack([i - 1, (i + 1) % RING], 1).ravel()
    indices = np.concatenate([[1, RING - 1], np.arange(RING, n), ring, np.zeros(LEAVES, np.int64)])
    return indptr, indices.astype(np.int32)


def _cheby(G):
    """FP64, one column: 60 B a node, 240 MB, on the graph as it was uploaded."""
    return api.solve(G, L.PPR, L.LOCAL_CHEBY, np.array([RING // 2], np.int32), 1e-3, alpha=0.1, want_r=False)


def _global(G):
    """FP64 gradient descent, one column: 156 MB on the merged copy, while there is one, or 208 MB."""
    return api.solve(G, L.PPR, L.GLOBAL_GD, np.array([RING // 2], np.int32), 1e-3, alpha=0.1, want_r=False, tile_w=1)


@pytest.mark.parametrize("solve, left", [(_cheby, 180 << 20), (_global, 120 << 20)])
def test_a_solve_that_would_fit_without_the_copy(arrays, solve, left):
    import torch
    ctx = api.Context(0)
    want = solve(api.Graph(*arrays, ctx=ctx))  # also loads the kernels
    want = {k: np.array(want[k]) for k in ("x", "oper")}
    ctx.close()
    ctx = api.Context(0)
    G = api.Graph(*arrays, ctx=ctx)
    torch.cuda.empty_cache()
    fill = torch.empty(torch.cuda.mem_get_info()[0] - left, dtype=torch.uint8, device="cuda")
    try:
        got = solve(G)
    finally:
        del fill
        torch.cuda.empty_cache()
    assert np.array_equal(got["oper"], want["oper"])
    assert np.abs(got["x"] - want["x"]).sum() < 1e-12


def test_a_solve_through_another_context(arrays):
    """The graph's copy is not among those of the context that runs out."""
    import torch
    own, other = api.Context(0), api.Context(0)
    G = api.Graph(*arrays, ctx=own)
    want = np.array(_cheby(G)["x"])
    view = object.__new__(api.Graph)
    view.ctx, view.ptr, view.n, view.cap, view.vol = other, G.ptr, G.n, G.cap, G.vol
    torch.cuda.empty_cache()
    fill = torch.empty(torch.cuda.mem_get_info()[0] - (180 << 20), dtype=torch.uint8, device="cuda")
    try:
        got = _cheby(view)
    finally:
        del fill
        torch.cuda.empty_cache()
    assert np.abs(got["x"] - want).sum() < 1e-12
