"""The 16/32-channel tcgen05 convolution over its issuer arrangements, items of one to many per CTA.

The head's two issuing threads share every slab's rows, the 3x3x1 layer's two take slabs in turn, the
masked layers wait for their accumulators in an order of their own.  The head against float64 (1e-4 of
the largest value: FP32 sums of exact BF16 products), the masked layers too, within the rounding of their
BF16 output (2^-8 of the largest value).
"""

import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def env(built_lib):
    import torch
    import _flf
    _flf.load_library()
    return torch, _flf


def conv(torch, x, w):
    W = w.double().reshape(3, 3, 3, w.shape[1], w.shape[2]).permute(4, 3, 0, 1, 2)
    return torch.nn.functional.conv3d(x.double().permute(0, 4, 1, 2, 3), W, padding=1).permute(0, 2, 3, 4, 1)


@pytest.mark.parametrize("T,Zp,Yp,Xp", [(1, 1, 4, 8), (1, 3, 5, 129), (2, 8, 24, 136), (1, 7, 203, 331), (3, 24, 64, 64)])
def test_head(env, T, Zp, Yp, Xp):
    torch, _flf = env
    g = torch.Generator(device="cuda").manual_seed(Zp * Xp)
    d = torch.randn((T, Zp, Yp, Xp, 16), generator=g, device="cuda").clamp_min(0).bfloat16()
    w = torch.zeros((27, 16, 16), device="cuda")
    w[:, :, 0] = torch.randn((27, 16), generator=g, device="cuda") / 20
    w = w.bfloat16()
    Z, Y, X = max(1, Zp - 1), Yp - 1, Xp - 3
    sums = torch.rand(T, generator=g, device="cuda") + 1
    x0 = torch.full((Z, T, Y, X), float("nan"), device="cuda")
    _flf.ws_head(d, w, 0.1, 1e-3, sums, x0)
    torch.cuda.synchronize()
    _flf.net_status()
    want = (conv(torch, d, w[:, :, :1])[..., 0] + 0.1).clamp_min(1e-3)[:, :Z, :Y, :X].permute(1, 0, 2, 3)
    want = want * (sums.double() / (Z * Y * X))[None, :, None, None]
    assert float((x0.double() - want).abs().max()) <= 1e-4 * float(want.abs().max())


@pytest.mark.parametrize("Ci,Co", [(16, 16), (16, 32), (32, 16), (32, 32)])
@pytest.mark.parametrize("shape", [(1, 1, 3, 7), (2, 2, 4, 128), (1, 9, 41, 130), (1, 23, 120, 257)])
def test_masked_layer(env, shape, Ci, Co):
    """In place as well: the mask may be the output (each thread reads its voxels' mask before it writes them)."""
    torch, _flf = env
    g = torch.Generator(device="cuda").manual_seed(Ci + shape[3])
    x = torch.randn(shape + (Ci,), generator=g, device="cuda").bfloat16()
    w = (torch.randn((27, Ci, Co), generator=g, device="cuda") / 20).bfloat16()
    mask = torch.randn(shape + (Co,), generator=g, device="cuda").bfloat16()
    y = torch.full(shape + (Co,), float("nan"), dtype=torch.bfloat16, device="cuda")
    _flf.conv3d(x, w, None, y, mask=mask)
    inplace = mask.clone()
    _flf.conv3d(x, w, None, inplace, mask=inplace)
    torch.cuda.synchronize()
    _flf.net_status()
    want = conv(torch, x, w) * (mask > 0)
    assert float((y.double() - want).abs().max()) <= 2.0 ** -8 * float(want.abs().max())
    assert torch.equal(inplace, y)
