"""A training step at the edges of its kernels' plans: the smallest batch, one of no
whole tile, a row more than a block of the column sums, two splits of the largest
weight gradient; every
parameter block's gradient against the oracle (bf16 roundings reproduced), and
the update of all blocks by one Adam launch with the bf16 copies it keeps."""
import numpy as np
import pytest

from oracle import cnn as N

pytestmark = pytest.mark.gpu


def _blocks(v):
    offs = np.cumsum([0] + [c * k + c for c, k in zip(N.COUT, N.K)])
    return [v[a:b] for a, b in zip(offs[:-1], offs[1:])]


@pytest.mark.parametrize("B", [8, 24, 136, 264])  # a weight gradient needs multiples of 8
def test_gradients_and_update(aldic, B):
    net, twin = aldic.InitNet(0, seed=1), aldic.InitNet(0, seed=9)
    p = net.get_params()
    rng = np.random.default_rng(B)
    x = rng.standard_normal((B, 64, 64, 2)).astype(np.float32)
    tgt = (0.5 * rng.standard_normal((B, 6))).astype(np.float32)
    loss, g, out = net.train_step(x, tgt, 1e-3, grads=True, outputs=True)
    lr, gr, outr = N.backward(p.astype(np.float64), x, tgt, rounding=True)
    # a bf16 feature that rounds the other way moves by 2^-8 of itself and few do, so
    # the outputs as a whole differ by less than that (one near zero may by more)
    assert np.linalg.norm(out - outr) < 2.0 ** -8 * np.linalg.norm(outr)
    assert loss == pytest.approx(lr, rel=2e-2)
    for k, (a, b) in enumerate(zip(_blocks(g), _blocks(gr))):
        assert np.linalg.norm(a - b) < 3e-2 * max(np.linalg.norm(b), 1e-12), k
    # the first step of Adam moves every parameter by lr g / (|g| + eps): its FP32
    # moments and their corrections round a few times 2^-24 of lr
    want = p - 1e-3 * g / (np.abs(g) + 1e-8)
    np.testing.assert_allclose(net.get_params(), want, rtol=2e-7, atol=1e-3 * 2e-5)
    # the copies the products read are the new parameters
    twin.set_params(net.get_params())
    np.testing.assert_array_equal(net.predict(x), twin.predict(x))
    net.close()
    twin.close()
