"""The finite-element global step at the edges of its products' tiling: grids
solved by one cluster (at most eight 32 x 32 tiles a product), by four launches
of 32 x 32 tiles and by four of 64 x 64 ones, one node less and more than a
tile, thin grids, in both directions; against the same fast diagonalisation in
numpy from scipy's eigenbases.  Both are direct FP64 solves of an operator
whose condition is below 1e3 here, so they agree to 1e3 * 2^-53 * (terms of a
sum) < 1e-10 of the largest value."""
import numpy as np
import pytest
from scipy.linalg import eigh

pytestmark = pytest.mark.gpu


def _solve(M, N, h, beta, mu, U, F, ud, vd):
    def km(n):
        K = (np.diag(np.r_[1.0, np.full(n - 2, 2.0), 1.0]) - np.eye(n, k=1) - np.eye(n, k=-1)) / h
        Mm = (np.diag(np.r_[2.0, np.full(n - 2, 4.0), 2.0]) + np.eye(n, k=1) + np.eye(n, k=-1)) * h / 6
        return K, Mm
    (Kx, Mx), (Ky, My) = km(M), km(N)
    lx, Vx = eigh(Kx, Mx)
    ly, Vy = eigh(Ky, My)
    W = (F - ud).reshape(N, M, 4)
    V = (U - vd).reshape(N, M, 2)
    # sum over a node's elements of +-1: elements to its left count +1, to its right -1
    jl, jr = (np.arange(N) > 0) * 1.0, (np.arange(N) < N - 1) * 1.0
    il, ir = (np.arange(M) > 0) * 1.0, (np.arange(M) < M - 1) * 1.0
    sx = np.outer(jl + jr, il - ir) * h / 2
    sy = np.outer(jl - jr, il + ir) * h / 2
    out = np.empty((N, M, 2))
    for f in range(2):
        # F's slots are [F11 F21 F12 F22]: u takes F11, F12, v takes F21, F22
        b = beta * (sx * W[..., f] + sy * W[..., 2 + f]) + mu * (My @ V[..., f] @ Mx)
        C = Vy.T @ b @ Vx / (beta * (ly[:, None] + lx[None]) + mu)
        out[..., f] = Vy @ C @ Vx.T
    return out.reshape(-1)


@pytest.mark.parametrize("M,N", [(2, 2), (9, 9), (32, 32), (33, 31), (64, 64), (65, 64), (128, 32), (3, 129),
                                 (129, 33), (97, 160), (770, 777), (2, 1000)])
def test_subpb2_tile_edges(aldic, M, N):
    rng = np.random.default_rng(M * 1000 + N)
    n, h = M * N, 8.0
    beta, mu = 1e-2 * h * h * 1e-3, 1e-3
    U, F, ud, vd = (rng.standard_normal(k * n) for k in (2, 4, 4, 2))
    x, y = 20 + h * np.arange(M), 30 + h * np.arange(N)
    mesh = aldic.MeshSetUp(np.tile(x, (N, 1)), np.tile(y[:, None], (1, M)), {"ImgSize": (0, 0)})
    got = aldic.Subpb2(mesh, beta, mu, U, F, ud, vd)
    want = _solve(M, N, h, beta, mu, U, F, ud, vd)
    np.testing.assert_allclose(got, want, rtol=0, atol=1e-10 * np.abs(want).max())
