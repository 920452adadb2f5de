"""Image preparation: the ROI sums over rows with every alignment and shorter
than a word, exact integers; the normalisation of every 8- and 16-bit value,
the bits of the IEEE quotient."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _want(f, roi):
    x0, x1, y0, y1 = roi
    r = f[y0 - 1:y1, x0 - 1:x1].astype(object)
    n = r.size
    s1, s2 = int(r.sum()), int((r * r).sum())
    m = np.float64(s1) / np.float64(n)
    sd = np.sqrt((np.float64(s2) - m * np.float64(s1)) / np.float64(n - 1))
    return (f.astype(np.float64) - m) / sd


@pytest.mark.parametrize("dtype", [np.uint8, np.uint16])
@pytest.mark.parametrize("W,H", [(9, 8), (257, 64), (255, 300), (1031, 70)])
def test_normalise_bits(aldic, dtype, W, H):
    rng = np.random.default_rng(W)
    f = rng.integers(0, np.iinfo(dtype).max + 1, (H, W)).astype(dtype)
    top = min(f.size, np.iinfo(dtype).max + 1)
    f.reshape(-1)[:top] = np.arange(top)          # every value, as far as there is room
    for roi in ((1, W, 1, H), (2, W - 1, 3, H - 2), (3, 5, 2, H), (W - 6, W, 1, 7)):
        got = aldic.funNormalizeImg([f], {"gridx": roi[:2], "gridy": roi[2:]})[0][0]
        np.testing.assert_array_equal(got, _want(f, roi))


@pytest.mark.parametrize("spread", [1, 3, 65535])
def test_normalise_every_16bit_value(aldic, spread):
    f = ((np.arange(65536) * 65535 // spread) % 65536 if spread < 65535 else np.arange(65536))
    f = f.astype(np.uint16).reshape(256, 256)
    if spread < 65535:
        f = (f % (spread + 1) + 60000).astype(np.uint16)
    got = aldic.funNormalizeImg([f], {"gridx": (1, 256), "gridy": (1, 256)})[0][0]
    np.testing.assert_array_equal(got, _want(f, (1, 256, 1, 256)))
