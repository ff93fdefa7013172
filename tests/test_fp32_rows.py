"""FP32 whole-graph solves add every push into a residual by itself: rows against the same additions in numpy float32."""
import numpy as np
import pytest

from gde import _lib as L
from gde import api

pytestmark = pytest.mark.gpu

LEAVES = 20_000
ALPHA, TAU = 0.1, 5.0
f32 = np.float32
# The emulation makes the kernel's own roundings; a contracted or reordered operation would change one of them by 2^-24.
RTOL = 8 * 2.0 ** -24


def _added_up(p):
    """LEAVES additions of p, one after another, from 0."""
    return np.add.accumulate(np.full(LEAVES, p, f32), dtype=f32)[-1]


class _Kahan:
    def __init__(self):
        self.x = self.c = f32(0)

    def add(self, v):
        y = f32(v) - self.c
        s = self.x + y
        self.c = (s - self.x) - y
        self.x = s

    def value(self):
        return float(self.x) - float(self.c)


def _global_gd(eps):
    """PPR from the centre of a star: (x of the centre, x of a leaf)."""
    rc, rl, xc, xl = f32(ALPHA), f32(0), _Kahan(), _Kahan()
    rest, d = f32(1.0 - ALPHA), f32(LEAVES)
    while float(rc) >= eps * ALPHA * LEAVES or float(rl) >= eps * ALPHA:
        xc.add(rc)
        xl.add(rl)
        rc, rl = _added_up(rest * rl / f32(1)), rest * rc / d
    return xc.value(), xl.value()


def _taylor(levels):
    """Heat kernel from the centre of a star, its Taylor levels."""
    rc, rl, xc, xl = f32(1), f32(0), _Kahan(), _Kahan()
    for j in range(levels + 1):
        xc.add(rc)
        xl.add(rl)
        t = f32(TAU / (j + 1.0))
        rc, rl = _added_up(t * rl / f32(1)), t * rc / f32(LEAVES)
    return xc.value() / np.exp(TAU), xl.value() / np.exp(TAU)


@pytest.mark.parametrize("W", [2, 4, 8, 16])
def test_a_hub_of_many_leaves(W):
    n = LEAVES + 1
    indptr = np.concatenate([[0], LEAVES + np.arange(n)])
    indices = np.concatenate([np.arange(1, n), np.zeros(LEAVES, np.int64)]).astype(np.int32)
    G = api.Graph(indptr, indices)
    seeds = np.zeros(W, np.int32)
    # 20,000 additions from 0 and one product are 1e-5 and more apart: the two cannot be taken for each other
    assert abs(float(_added_up(f32(0.3))) / (0.3 * LEAVES) - 1) > 1e-5
    eps = 1e-6
    x = api.solve(G, L.PPR, L.GLOBAL_GD, seeds, eps, prec="fp32", alpha=ALPHA, tile_w=W)["x"].astype(np.float64)
    centre, leaf = _global_gd(eps)
    assert np.allclose(x[:, 0], centre, rtol=RTOL, atol=0) and np.allclose(x[:, 1:], leaf, rtol=RTOL, atol=0)
    levels = L.load().gde_hk_estimate_n(TAU, eps)
    x = api.solve(G, L.HK, L.HK_TAYLOR, seeds, eps, prec="fp32", tau=TAU, tile_w=W)["x"].astype(np.float64)
    centre, leaf = _taylor(levels)
    assert np.allclose(x[:, 0], centre, rtol=RTOL, atol=0) and np.allclose(x[:, 1:], leaf, rtol=RTOL, atol=0)


def _served(eps):
    """A served PPR query from the centre, whose residual is FP64: (residual of the centre, of a leaf, x of the centre)."""
    rc, rl, xc = ALPHA, f32(0), _Kahan()
    while True:
        if rc >= eps * ALPHA * LEAVES:
            xc.add(rc)
            rc, rl = 0.0, rl + f32(((1.0 - ALPHA) * rc) / LEAVES)
        elif float(rl) >= eps * ALPHA:
            rc, rl = rc + LEAVES * float(f32(1.0 - ALPHA) * rl / f32(1)), f32(0)
        else:
            return rc, float(rl), xc.value()


def test_a_served_hub_keeps_every_push_in_fp64():
    indptr = np.concatenate([[0], LEAVES + np.arange(LEAVES + 1)])
    indices = np.concatenate([np.arange(1, LEAVES + 1), np.zeros(LEAVES, np.int64)]).astype(np.int32)
    G = api.Graph(indptr, indices)
    eps = next(e for e in np.geomspace(1e-6, 2e-6, 50) if _served(e)[0] > 0)  # the last push is the leaves'
    res = api.solve(G, L.PPR, L.LOCAL_GD, np.zeros(1, np.int32), eps, prec="fp32", out64=True, alpha=ALPHA)
    rc, rl, xc = _served(eps)
    # the sum of the pushes is exact in FP64 (24 bits times 20,000); rounded to FP32 it would be 2^-25 off
    assert float(f32(rc)) != rc and abs(res["r"][0, 0] / rc - 1) < 2.0 ** -50
    assert np.allclose(res["r"][0, 1:], rl, rtol=RTOL, atol=0) and res["x"][0, 0] == pytest.approx(xc, rel=RTOL)
