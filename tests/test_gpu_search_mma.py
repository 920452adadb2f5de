"""The tensor-core integer search at the edges of its plan, bit for bit
against the oracle's per-point funIntegerSearch restatement (its sums are
exact integers, its estimates only choose what ncc_combine evaluates):
search zones that end just inside and just beyond one pass of lanes (64 shifts
of 16-bit pixels, 128 of 8-bit ones) and of columns (128, 256), one and two
region blocks, window tables beyond shared memory, the smallest subsets, the
largest template taken and the first that is not, odd subsets, points at the
image's border, constant templates and flat regions whose ties overflow the
queue."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _images(oracle, synth, dtype, W, H, seed):
    f = synth.speckle(W, H, W * H // 50, seed)
    g = synth.warp(f, lambda X, Y: (1.3 + 1.5 * np.sin(2 * np.pi * Y / 150),
                                    -1.1 + 1.0 * np.cos(2 * np.pi * X / 170)), 2.0, seed)
    if dtype == np.uint16:
        rng = np.random.default_rng(seed)
        f, g = ((a.astype(np.uint32) * 256 + rng.integers(0, 256, a.shape)).astype(np.uint16) for a in (f, g))
    return f, g


def _check(aldic, oracle, f, g, w, step, s):
    H, W = f.shape
    _, mu_g, _ = oracle.normalize(g)
    x, y, u, v, cc = aldic.funIntegerSearch(f, g, s, [1, W], [1, H], w, step, 0, step, qfactors=False)
    sx, sy = (s, s) if np.isscalar(s) else s
    xo, yo, uo, vo, cco, _ = oracle.int_search(f, g, mu_g, (1, W), (1, H), w, step, (sx, sy))
    assert u.size > 0
    for a, b in ((x, xo), (y, yo), (u, uo), (v, vo), (cc["max"], cco)):
        np.testing.assert_array_equal(a, b)
    return u


@pytest.mark.parametrize("w,step,s", [
    (20, 9, 30), (20, 9, 31), (17, 14, 45),       # 63, 65 and 93 shifts: one pass of 16-bit lanes, two
    (18, 24, 62), (18, 24, 63),                   # 127 and 129: 8-bit lanes, 16-bit columns
    (6, 11, (2, 127)), (6, 11, (2, 128)),         # 257 and 259 rows of shifts: 8-bit columns
    (40, 30, 43), (41, 30, 44),                   # K of 97 .. 128 + 32: the second region block
    (2, 5, 0), (2, 5, 1), (3, 5, 2), (9, 7, 4),   # the smallest
    (127, 40, 6), (128, 40, 6), (96, 40, 20)])    # tw = 128 is the largest template
@pytest.mark.parametrize("dtype", [np.uint8, np.uint16])
def test_plan_edges_bit_exact(aldic, oracle, synth, dtype, w, step, s):
    sx, sy = (s, s) if np.isscalar(s) else s
    W, H = 2 * w + 2 * sx + 5 * step + 7, 2 * w + 2 * sy + 4 * step + 9
    _check(aldic, oracle, *_images(oracle, synth, dtype, W, H, 51), w, step, s)


@pytest.mark.parametrize("w,step,s", [(32, 16, 9), (32, 16, 10), (32, 8, 28), (32, 8, 29), (24, 8, 29), (16, 8, 33),
                                      (16, 8, 34)])
def test_tiles_or_points_bit_exact(aldic, oracle, synth, w, step, s):
    """8-bit geometries with a tile on either side of the line up to which the tiles pay."""
    W, H = 2 * w + 2 * s + 9 * step + 3, 2 * w + 2 * s + 8 * step + 5
    _check(aldic, oracle, *_images(oracle, synth, np.uint8, W, H, 57), w, step, s)


@pytest.mark.parametrize("level", [0, 77, 255])
@pytest.mark.parametrize("dtype", [np.uint8, np.uint16])
def test_flat_and_tied_regions_bit_exact(aldic, oracle, synth, dtype, level):
    W, H = 233, 201
    f, g = _images(oracle, synth, dtype, W, H, 53)
    level = level * (257 if dtype == np.uint16 else 1)
    f[120:170, 20:75] = level                      # constant templates: NaN
    g[60:160, 90:200] = level                      # flat regions: the maximum on the ring
    g[130:, 100:] = np.where(np.add.outer(np.arange(H - 130), np.arange(W - 100)) % 2, level, 3)
    f[130:, 100:] = g[130:, 100:]                  # half of a map's entries tie
    u = _check(aldic, oracle, f, g, 14, 7, 13)
    assert np.isnan(u).any()


def test_full_scale_sums_bit_exact(aldic, oracle):
    """Pixels at the top of the 16-bit range, one count apart: the largest sums
    and the windows of the least variance."""
    rng = np.random.default_rng(7)
    f = (65535 - (rng.random((150, 170)) < 0.02)).astype(np.uint16)
    g = np.roll(f, (2, -1), (0, 1))
    _check(aldic, oracle, f, g, 20, 8, 9)
    _check(aldic, oracle, f >> 8, g >> 8, 20, 8, 9)
    b = (255 - (rng.random((150, 170)) < 0.02)).astype(np.uint8)
    _check(aldic, oracle, b, np.roll(b, (2, -1), (0, 1)), 20, 8, 9)


@pytest.mark.parametrize("dtype", [np.uint8, np.uint16])
def test_waits_that_give_up_are_an_error(aldic, oracle, synth, dtype):
    """Every wait of the kernel gives up at once (no product is issued then): the call
    fails, a frame whose start it was fails, device arrays carry NaN and the next
    status tells; with the usual limit the context works on."""
    import torch
    f, g = _images(oracle, synth, dtype, 200, 180, 59)
    ctx = aldic.Context(0)
    search = lambda a, b: aldic.funIntegerSearch(a, b, 6, [1, 200], [1, 180], 21, 10, 0, 10, qfactors=False, ctx=ctx)
    al = aldic.ALDIC(20, 10, 6, precision=aldic.FP32, ctx=ctx)
    want = search(f, g)
    al.set_images(f, g)
    whole = al.frame()
    aldic._lib.call("aldic_ctx_set_wait_tries", ctx.h, 0)
    with pytest.raises(aldic.AldicError, match="timed out"):
        search(f, g)
    with pytest.raises(aldic.AldicError, match="timed out"):
        al.frame()
    out = search(torch.from_numpy(f).cuda(), torch.from_numpy(g).cuda())
    torch.cuda.synchronize()
    assert bool(torch.isnan(torch.as_tensor(out[2])).all())
    aldic._lib.call("aldic_ctx_set_wait_tries", ctx.h, 1 << 22)
    with pytest.raises(aldic.AldicError, match="timed out"):
        search(f, g)                               # the word of the call before
    for a, b in zip(search(f, g)[:4], want[:4]):
        np.testing.assert_array_equal(a, b)
    al.set_images(f, g)
    np.testing.assert_array_equal(al.frame()["U"], whole["U"])


@pytest.mark.parametrize("dtype,step", [(np.uint16, 2), (np.uint8, 2), (np.uint8, 8)])
def test_work_memory_is_what_the_path_reads(aldic, oracle, synth, dtype, step):
    """Points on the tensor cores need a table of the image, not the tiles' map of every
    point (2.7 GB here at step 2; the tiles of step 8 do not pay at this zone), in the
    search by itself and in a frame, whose other arrays take 2 kB a node."""
    import torch
    W, H = 700, 690
    f, g = _images(oracle, synth, dtype, W, H, 61)
    ctx = aldic.Context(0)
    ctx.set_ref(f)
    ctx.set_def(g)
    torch.cuda.synchronize()
    before = torch.cuda.mem_get_info()[0]
    x = aldic.funIntegerSearch(f, g, 40, [1, W], [1, H], 16, step, 0, step, qfactors=False, ctx=ctx)[0]
    assert before - torch.cuda.mem_get_info()[0] < 128 << 20
    al = aldic.ALDIC(16, step, 40, precision=aldic.FP32, n_admm=1, ctx=ctx)
    al.set_images(f, g)
    al.frame()
    assert before - torch.cuda.mem_get_info()[0] < (256 << 20) + 2048 * x.size
