"""ba_interp2 on the GPU: the 32-bit path of points whose taps lie inside the image and
the clamped one of the others in one call, bit for bit against the oracle."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", [np.float64, np.float32])
def test_interp_border_and_inside_agree(aldic, oracle, dtype):
    """Points of every kind in one call: far inside, on the last taps that lie
    inside, one past them, beyond the image, not finite; two planes."""
    rng = np.random.default_rng(5)
    N, M = 37, 41
    F = rng.standard_normal((2, N, M)).astype(dtype)
    edge = np.array([-7, -4, -0.5, 0, 0.5, 1, 1.5, 2 - 1e-6, 2, 2.25, 3, 20.7], dtype)
    hi = np.concatenate([edge, [np.nan, np.inf, -np.inf]]).astype(dtype)
    X = np.concatenate([hi, N + 1 - edge, rng.uniform(0, N, 200).astype(dtype)]).astype(dtype)
    Y = np.concatenate([hi, M + 1 - edge, rng.uniform(0, M, 200).astype(dtype)]).astype(dtype)
    X, Y = (np.ascontiguousarray(a) for a in np.meshgrid(X, Y))
    got = aldic.ba_interp2(F, X, Y)
    for p in range(2):
        np.testing.assert_array_equal(got[p], oracle.ba_interp2(F[p], X, Y))
