"""The fused forward pass of the learned guess (k_net.cu) against the same
network in PyTorch with the bf16 roundings at the same places: batches around
a row tile, around the number of resident CTAs, with and without the split of
the dense layer's K range, and every kind of input the entry point takes."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _reference(torch, p, x):
    """x: B x 64 x 64 x 2 bf16 on the GPU -> B x 8, FP32 sums; ReLU of NaN is 0."""
    relu = lambda t: torch.where(t > 0, t, torch.zeros_like(t))
    sizes = [(128, 64), (128, 128), (256, 4096), (8, 256)]
    o, L = 0, []
    for co, ci in sizes:
        L.append((p[o:o + co * ci].view(co, ci), p[o + co * ci:o + co * ci + co]))
        o += co * ci + co
    r = lambda t: t.to(torch.bfloat16).float()
    W = [r(w) for w, _ in L[:3]] + [L[3][0]]
    B = x.shape[0]

    def enc(c):
        cells = x[..., c].float().view(B, 8, 8, 8, 8).permute(0, 1, 3, 2, 4).reshape(B, 64, 64)
        return r(r(relu(cells @ W[0].T + L[0][1])) @ W[1].T + L[1][1])
    corr = r((enc(0) @ enc(1).transpose(1, 2)) * 0.08838834764831845)
    y = r(relu(corr.reshape(B, 4096) @ W[2].T + L[2][1]))
    return y @ W[3].T + L[3][1]


@pytest.fixture(scope="module")
def net(aldic):
    import torch
    torch.backends.cuda.matmul.allow_tf32 = False
    n = aldic.InitNet(0, seed=4)
    p = n.get_params()
    p += 0.05 * np.random.default_rng(1).standard_normal(p.size).astype(np.float32) * (p == 0)  # biases
    n.set_params(p)
    return n, torch.from_numpy(p).cuda()


# a value that falls on the other side of a bf16 rounding in one layer moves the
# next by 2^-9 of a term: 2e-3 of the outputs' size over 256 terms, times 4
RTOL, ATOL = 2e-2, 8e-3


@pytest.mark.parametrize("B", [1, 2, 127, 128, 129, 296, 297, 593, 9472, 9473, 9600])
def test_forward_matches_reference(net, B):
    import torch
    n, p = net
    g = torch.Generator(device="cuda").manual_seed(B)
    x = torch.randn((B, 64, 64, 2), generator=g, device="cuda").to(torch.bfloat16)
    out = n.predict(x)
    ref = _reference(torch, p, x)
    torch.testing.assert_close(out, ref, rtol=RTOL, atol=ATOL * float(ref.abs().max()))


def test_forward_inputs(net):
    import torch
    n, p = net
    B = 37
    flat = torch.randn(B * 8192 + 1, device="cuda").to(torch.bfloat16)
    x = flat[:-1].view(B, 64, 64, 2)
    out = n.predict(x)
    y = flat.roll(1)[1:].view(B, 64, 64, 2)          # the same pairs, two bytes off alignment
    assert y.data_ptr() % 16 == 2
    torch.testing.assert_close(n.predict(y), out, rtol=0, atol=0)
    torch.testing.assert_close(n.predict(x.float()), out, rtol=0, atol=0)
    host = n.predict(x.float().cpu().numpy())
    np.testing.assert_array_equal(host, out.cpu().numpy())
    torch.testing.assert_close(out, _reference(torch, p, x), rtol=RTOL, atol=ATOL * float(out.abs().max()))


def test_forward_does_not_depend_on_the_batch(net):
    """A pair's output has the same bits in every batch: the dense layer's sums have
    the same order whether its slices share a CTA or each has its own."""
    import torch
    n, _ = net
    x = torch.randn((9601, 64, 64, 2), generator=torch.Generator(device="cuda").manual_seed(3), device="cuda")
    x = x.to(torch.bfloat16)
    whole = n.predict(x)
    for B in (1, 127, 129, 2304, 2305, 9472):
        torch.testing.assert_close(n.predict(x[9601 - B:]), whole[9601 - B:], rtol=0, atol=0)


def test_forward_of_values_that_are_not_finite(net):
    """A NaN pixel takes its cell's embedding to 0, an infinite one the pair's hidden
    layer; the other pairs of the batch keep their bits."""
    import torch
    n, p = net
    x = torch.randn((300, 64, 64, 2), generator=torch.Generator(device="cuda").manual_seed(8), device="cuda")
    x = x.to(torch.bfloat16)
    clean = n.predict(x)
    x[3, 10, 20, 0] = x[140, 63, 63, 1] = x[299, :, :, 0] = float("nan")
    x[5, 0, 0, 1], x[201, 33, 1, 0] = float("inf"), float("-inf")
    out, ref = n.predict(x), _reference(torch, p, x)
    assert bool(torch.isfinite(out).all())
    torch.testing.assert_close(out, ref, rtol=RTOL, atol=ATOL * float(ref.abs().max()))
    same = [b for b in range(300) if b not in (3, 140, 299, 5, 201)]
    torch.testing.assert_close(out[same], clean[same], rtol=0, atol=0)
