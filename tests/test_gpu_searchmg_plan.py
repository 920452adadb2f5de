"""The multigrid search at the edges of its kernels' plans: every remainder of
log2 of the transform lengths modulo 3 and the longest (8192), rectangular
regions that split along one side only, tables wider than one scan block,
widths that leave every remainder of a packed word, last-level regions of all
sizes; against the oracle, whose sums are the same integers.  Only the first
level's correlation is a rounded sum, and only its rounded-up peak is used."""
import numpy as np
import pytest

from oracle import searchmg as S

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("W,H,w,step", [
    (150, 131, 16, 8), (260, 251, 24, 10), (523, 300, 32, 16),   # lengths 256, 512, 1024
    (1100, 120, 12, 10), (120, 1101, 12, 10),                    # 2048 x 256 and the other way round
    (2207, 151, 30, 25), (151, 2203, 30, 25),                    # 8192
    (420, 431, 60, 20), (341, 233, 20, 7)])
@pytest.mark.parametrize("dtype", [np.uint8, np.uint16])
def test_mg_plan_edges(aldic, synth, dtype, W, H, w, step):
    if dtype == np.uint16 and max(W, H) > 2048:
        pytest.skip("the oracle's 64-bit sums overflow")
    f = synth.speckle(W, H, W * H // 40, 31)
    g = synth.warp(f, lambda X, Y: (6.3 + 2.0 * np.sin(2 * np.pi * Y / 200), -4.1 + 1.5 * np.cos(2 * np.pi * X / 170)),
                   2.0, 31)
    if dtype == np.uint16:
        rng = np.random.default_rng(2)
        f, g = ((a.astype(np.uint32) * 256 + rng.integers(0, 256, a.shape)).astype(np.uint16) for a in (f, g))
    ro = S.int_search_mg(f, g, [1, W], [1, H], w, step)
    info = {}
    x, y, u, v, cc = aldic.funIntegerSearchMg(f, g, [1, W], [1, H], w, step, step, info=info)
    np.testing.assert_array_equal(x, ro["x"])
    np.testing.assert_array_equal(y, ro["y"])
    assert (info["level1_u"], info["level1_v"]) == tuple(ro["regions"]["level1"])
    assert info["regions"] == len(ro["regions"]["regions"])
    for got, ref in ((u, ro["u"]), (v, ro["v"]), (cc["max"], ro["ccmax"])):
        np.testing.assert_allclose(got, ref, rtol=0, atol=1e-8)
    for q in (0, 1):
        np.testing.assert_allclose(cc["qfactors"][:, q], ro["q1" if q == 0 else "q2"].T.reshape(-1), rtol=0, atol=1e-8)
