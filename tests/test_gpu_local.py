"""The tiled node-grid solves (k_local.cu) against the oracle: gridfit springs
and spring inpainting at tile edges, with nodes without data scattered, in
clusters a tile can hold, and in regions only the grid-wide solver can take."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SIZES = [(2, 2), (3, 40), (31, 33), (32, 32), (65, 64), (97, 130)]


def _data(M, N, nf, seed):
    r = np.random.default_rng(seed)
    j, i = np.mgrid[:N, :M]
    z = np.stack([np.sin(0.1 * (k + 1) * i) + np.cos(0.13 * j + k) for k in range(nf)])
    return z.reshape(nf, -1) + 0.1 * r.standard_normal((nf, M * N))


def _holes(M, N, kind, seed):
    """Flat mask of missing nodes."""
    r = np.random.default_rng(seed + 100)
    m = np.zeros((N, M), bool)
    if kind == "scattered":
        m = r.random((N, M)) < 0.01
    elif kind == "dense":
        m = r.random((N, M)) < 0.41
    elif kind == "blocks":
        for _ in range(max(1, M * N // 600)):
            x, y = r.integers(0, M), r.integers(0, N)
            m[y:y + 5, x:x + 6] = True
    elif kind == "blob":       # wider than a tile and its halo
        m[N // 8:N - N // 8, M // 8:M - M // 8] = True
    elif kind == "snake":      # one connected path through several tiles
        m[::4, :] = True
        m[:, -1:] = True
    m[0, 0] = m[N // 2, 0] = m[-1, -1] = False
    return m.reshape(-1)


@pytest.mark.parametrize("M,N", SIZES)
@pytest.mark.parametrize("kind", ["none", "scattered", "blocks", "blob"])
def test_gridfit_matches_oracle(aldic, oracle, M, N, kind):
    z = _data(M, N, 2, M + N)
    hole = _holes(M, N, kind, M)
    z[:, hole] = np.nan
    z[1, :M // 2] = np.nan           # the fields' masks differ
    if np.isfinite(z).sum(1).min() < 3:
        pytest.skip("gridfit needs three data")
    ref = oracle.gridfit_springs(M, N, z)
    got = aldic.gridfit_springs(M, N, z)
    # |r| <= 1e-11 |b|; A's smallest eigenvalue is that of springs over the widest
    # gap between data, lam2 (pi / (2 gap))^2 at least
    gap = max(M, N) if kind == "blob" else 12
    lmin = min(1.0, 0.0214 * (np.pi / (2 * gap)) ** 2)
    tol = 1e-11 * np.linalg.norm(np.nan_to_num(z)) / lmin + 1e-12
    np.testing.assert_allclose(got, ref, rtol=0, atol=tol)


@pytest.mark.parametrize("M,N", SIZES)
def test_gridfit_in_place_and_infinite_data(aldic, M, N):
    import torch
    z = torch.from_numpy(_data(M, N, 2, 3)).cuda()
    ref = aldic.gridfit_springs(M, N, z)
    inplace = z.clone()
    ctx = aldic.default_context()
    from importlib import import_module
    lib = import_module("2d_aldic_b200._lib")
    lib.call("aldic_gridfit_springs", ctx.h, M, N, 2, inplace.data_ptr(), inplace.data_ptr())
    torch.testing.assert_close(inplace, ref, rtol=0, atol=0)
    z[0, M * N // 2] = float("inf")  # no finite residual: the fields come back as they were
    out = aldic.gridfit_springs(M, N, z)
    torch.testing.assert_close(out[0], z[0], rtol=0, atol=0)
    np.testing.assert_allclose(out[1].cpu(), ref[1].cpu(), rtol=0, atol=1e-9)


@pytest.mark.parametrize("M,N", SIZES + [(243, 61)])
@pytest.mark.parametrize("kind", ["none", "scattered", "dense", "blocks", "blob", "snake"])
def test_inpaint_matches_oracle(aldic, oracle, M, N, kind):
    z = _data(M, N, 1, M + 3 * N)[0]
    z[_holes(M, N, kind, N)] = np.nan
    if not np.isfinite(z).any():
        pytest.skip("nothing known")
    ref = oracle.inpaint_springs(M, N, z.copy())
    got = aldic.inpaint_nans(z.reshape(N, M)).reshape(-1)
    # |r| <= 1e-11 |b|, the Laplacian's smallest eigenvalue on a region of
    # diameter d at least (pi / (2 d))^2
    d = {"blob": max(M, N), "snake": M + N, "dense": 60}.get(kind, 8)
    tol = 1e-11 * 4 * np.linalg.norm(np.nan_to_num(z)) * (2 * d / np.pi) ** 2 + 1e-12
    np.testing.assert_allclose(got, ref, rtol=0, atol=tol)
    np.testing.assert_array_equal(got[np.isfinite(z)], z[np.isfinite(z)])


@pytest.mark.parametrize("M,N", [(2, 2), (33, 31), (97, 70)])
@pytest.mark.parametrize("nf", [1, 2, 4])
def test_smooth_matches_oracle(aldic, oracle, M, N, nf):
    v = _data(M, N, nf, 5).T.copy()
    v[_holes(M, N, "blocks", 1)[:, None] & (np.arange(nf) == 0)] = np.nan
    from importlib import import_module
    lib = import_module("2d_aldic_b200._lib")
    got = v.reshape(-1).copy()
    lib.call("aldic_smooth", aldic.default_context().h, M, N, nf, got.ctypes.data)
    ref = oracle.smooth_fields(M, N, v.reshape(-1).copy(), nf)
    np.testing.assert_allclose(got, ref, rtol=0, atol=1e-11 * np.linalg.norm(np.nan_to_num(v)) / (0.0214 * (np.pi / 24) ** 2))


def _smooth(aldic, M, N, v):
    from importlib import import_module
    out = np.ascontiguousarray(v.T).reshape(-1)    # fields interleaved
    import_module("2d_aldic_b200._lib").call("aldic_smooth", aldic.default_context().h, M, N, len(v), out.ctypes.data)
    return out.reshape(-1, len(v)).T


@pytest.mark.parametrize("M,N", [(40, 33), (97, 70)])
def test_smooth_goes_on_where_the_tiles_cannot_finish(aldic, oracle, M, N):
    """A region without data that the tiles' fixed steps do not cross: the grid-wide
    solver goes on from their result, and convolves."""
    v = _data(M, N, 2, 7)
    hole = np.zeros((N, M), bool)
    hole[6:N - 6, 5:M - 7] = True
    v[0, hole.reshape(-1)] = np.nan
    ref = oracle.smooth_fields(M, N, np.ascontiguousarray(v.T).reshape(-1), 2).reshape(-1, 2).T
    # lam2 (pi / (2 gap))^2 bounds the springs' smallest eigenvalue over the gap
    tol = 1e-11 * np.linalg.norm(np.nan_to_num(v)) / (0.0214 * (np.pi / (2 * max(M, N))) ** 2)
    np.testing.assert_allclose(_smooth(aldic, M, N, v), ref, rtol=0, atol=tol)


@pytest.mark.parametrize("M,N", [(40, 33), (97, 70)])
def test_smooth_of_infinite_data(aldic, oracle, M, N):
    """An infinite value has no finite residual: its field stays as it was and is only
    convolved, in both passes; the other field is smoothed as ever, and the next call
    finds the gate and the tickets as they should be."""
    v = _data(M, N, 2, 9)
    want = oracle.smooth_fields(M, N, np.ascontiguousarray(v.T).reshape(-1), 2).reshape(-1, 2).T
    clean = _smooth(aldic, M, N, v)
    tol = 1e-11 * np.linalg.norm(v) / 0.886
    np.testing.assert_allclose(clean, want, rtol=0, atol=tol)
    w = v.copy()
    w[0, M * (N // 2) + M // 3] = np.inf
    e = np.exp([-4.0, -2.0, -4.0, -2.0, 0.0, -2.0, -4.0, -2.0, -4.0])

    def conv(a):
        pad = np.pad(a.reshape(N, M), 1)
        one = np.pad(np.ones((N, M)), 1)
        near = lambda q: [q[1 + dj:1 + dj + N, 1 + di:1 + di + M] for dj in (-1, 0, 1) for di in (-1, 0, 1)]
        return (sum(c * b for c, b in zip(e, near(pad))) / sum(c * b for c, b in zip(e, near(one)))).reshape(-1)
    got = _smooth(aldic, M, N, w)
    # nine terms of at most max |v|, whose sum and division round ten times, in two passes
    np.testing.assert_allclose(got[0], conv(conv(w[0])), rtol=0, atol=20 * 2.0 ** -53 * np.abs(v).max())
    np.testing.assert_allclose(got[1], want[1], rtol=0, atol=tol)
    np.testing.assert_array_equal(_smooth(aldic, M, N, v), clean)


def test_frame_counts_the_iterations_of_its_solves(aldic, synth):
    """Also where the tiles finish every solve: the fits take their fixed number of
    steps, the refills' iterations are counted by the tile that takes most."""
    f = synth.speckle(200, 180, 900, 3)
    g = synth.warp(f, synth.uniform_affine(0.002, -0.001, 0.4, -0.3), 0.5, 3)
    al = aldic.ALDIC(20, 10, 6, ctx=aldic.Context(0))
    al.set_images(f, g)
    its = [al.frame()["stats"]["max_pcg_iters"] for _ in range(3)]
    assert its[0] >= 12 and its == its[:1] * 3
