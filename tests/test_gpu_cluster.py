"""The cluster conjugate gradients at the edges of their plan -- one to four
rows a thread, the last grid they take and the first they leave to the
grid-wide kernel, rows that do not fit in shared memory, unknowns in one
corner, one unknown and none -- through the quadtree entry points on uniform
meshes, against scipy's direct solves.  The solves stop at a residual of
1e-11, so the error is below 1e-11 of the right-hand side times the
condition: under 1e4 for refills of patches some 40 nodes across, under 1e2
for the global step."""
import numpy as np
import pytest
from scipy.linalg import eigh

from oracle import quadtree as Q

pytestmark = pytest.mark.gpu

GRIDS = [(2, 2), (7, 5), (64, 128), (91, 91), (127, 129), (128, 129), (157, 157), (181, 181), (184, 183)]


def _mesh(aldic, M, N, h=8.0):
    x, y = np.meshgrid(20 + h * np.arange(M), 30 + h * np.arange(N))
    c, el = Q.uniform_mesh(x, y, M, N)
    return c, el, aldic.QuadtreeMesh.create(c, el, [])


@pytest.mark.parametrize("M,N", GRIDS)
def test_refill_sizes(aldic, M, N):
    c, el, m = _mesh(aldic, M, N)
    n = M * N
    rng = np.random.default_rng(n)
    vals = np.stack([np.sin(c[:, 0] / 90.0), np.cos(c[:, 1] / 70.0), c[:, 0] * 1e-2, rng.standard_normal(n),
                     c[:, 1] * 1e-2], 1)
    i, j = np.arange(n) % M, np.arange(n) // M
    corner = (i < 0.9 * M) & (j < 36)
    for bad in (rng.random(n) < 0.15, corner, np.arange(n) == n - 1, np.zeros(n, bool)):
        if bad.all():
            continue
        vin = np.where(bad[:, None], 0.0, vals)
        ref = Q.graph_fill(n, Q.mesh_edges(np.c_[el, np.zeros((len(el), 4), int)]), vin, bad)
        out = aldic.quadtree_fill(m, vin, bad.astype(np.uint8)).reshape(n, -1)
        np.testing.assert_allclose(out, ref, rtol=0, atol=1e-7 * np.abs(vals).max())
        np.testing.assert_array_equal(out[~bad], vals[~bad])


@pytest.mark.parametrize("M,N", GRIDS)
def test_global_step_sizes(aldic, M, N):
    h, mu, beta = 8.0, 1e-3, 1e-2 * 64 * 1e-3
    c, el, m = _mesh(aldic, M, N, h)
    U = np.random.default_rng(M).standard_normal(2 * M * N)

    def pencil(n):
        K = (np.diag(np.r_[1.0, np.full(n - 2, 2.0), 1.0]) - np.eye(n, k=1) - np.eye(n, k=-1)) / h
        Mm = (np.diag(np.r_[2.0, np.full(n - 2, 4.0), 2.0]) + np.eye(n, k=1) + np.eye(n, k=-1)) * h / 6
        return (*eigh(K, Mm), Mm)

    (lx, Vx, Mx), (ly, Vy, My) = pencil(M), pencil(N)
    want = np.empty((N, M, 2))
    for f in range(2):
        b = mu * (My @ U.reshape(N, M, 2)[..., f] @ Mx)
        want[..., f] = Vy @ (Vy.T @ b @ Vx / (beta * (ly[:, None] + lx[None]) + mu)) @ Vx.T
    out = aldic.Subpb2Quadtree(m, beta, mu, U, np.zeros(4 * M * N))
    np.testing.assert_allclose(out, want.reshape(-1), rtol=0, atol=1e-8)
