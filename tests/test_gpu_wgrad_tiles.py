"""Weight and bias gradients at the edges of their tiles, against float64.

Row blocks of 4 along y, segments of 64 or 128 voxels along x in steps of 16,
channel tiles of 16 / 32, chunks cut anywhere in the row blocks (a workspace of
one slice up to more than the kernel uses), and without a workspace the nine
(dz, dy) in CTAs of their own.  FP32 sums of exact BF16 products over at most
about 5000 voxels: 1e-4 of the largest gradient.
"""

import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def env(built_lib):
    import torch
    import _flf
    _flf.load_library()
    return torch, _flf


def reference(torch, x, dy):
    p = torch.nn.functional.pad(x.double(), (0, 0, 1, 1, 1, 1, 1, 1))
    B, Z, Y, X, co = dy.shape
    g = dy.double().reshape(-1, co)
    return torch.stack([p[:, k // 9:k // 9 + Z, k // 3 % 3:k // 3 % 3 + Y, k % 3:k % 3 + X].reshape(-1, x.shape[-1]).T @ g
                        for k in range(27)]), g.sum(0)


@pytest.mark.parametrize("shape,Ci,Co", [
    ((1, 1, 1, 1), 16, 16), ((1, 2, 3, 15), 16, 16), ((2, 1, 4, 17), 16, 16), ((1, 3, 5, 128), 16, 16),
    ((1, 2, 9, 129), 16, 16), ((1, 1, 4, 260), 16, 16), ((1, 2, 6, 64), 16, 32), ((1, 3, 7, 65), 32, 16),
    ((2, 2, 8, 33), 32, 32), ((1, 4, 13, 63), 64, 32), ((1, 2, 5, 16), 48, 16), ((3, 3, 21, 20), 32, 64)])
@pytest.mark.parametrize("slices", [0, 1, 3, 64])
def test_gradients_at_tile_edges(env, shape, Ci, Co, slices):
    torch, _flf = env
    g = torch.Generator().manual_seed(Ci * Co + shape[3])
    x = torch.randn(shape + (Ci,), generator=g).bfloat16()
    dy = torch.randn(shape + (Co,), generator=g).bfloat16()
    want, wantb = reference(torch, x, dy)
    ws = torch.full((max(slices * 27 * Ci * Co, 1),), float("nan"), device="cuda")
    dw = torch.ones((27, Ci, Co), dtype=torch.float32, device="cuda")       # both add to what is there
    db = torch.ones(Co, dtype=torch.float32, device="cuda")
    _flf.conv3d_wgrad(x.cuda(), dy.cuda(), dw, ws=ws if slices else None)
    _flf.bias_grad(dy.cuda(), db, ws=ws if slices else None)
    assert float((dw.cpu().double() - 1 - want).abs().max()) <= 1e-4 * float(want.abs().max().clamp_min(1))
    assert float((db.cpu().double() - 1 - wantb).abs().max()) <= 1e-4 * float(wantb.abs().max().clamp_min(1))


@pytest.mark.parametrize("C,M", [(1, 5), (3, 4099), (24, 2049), (40, 70000), (120, 9000), (128, 30000)])
def test_bias_gradient_channel_counts(env, C, M):
    """Any channel count up to 128: 16-byte loads for multiples of 8, one channel per thread else
    (also at an address that is not a multiple of 16)."""
    torch, _flf = env
    g = torch.Generator().manual_seed(C)
    v = torch.randn(M * C + 1, generator=g).bfloat16()
    ws = torch.full((C * 64,), float("nan"), device="cuda")
    d = v.cuda()
    for off in (0, 1):
        rows = v[off:off + M * C].reshape(M, C)
        db = torch.zeros(C, device="cuda")
        lib = _flf.load_library()
        assert lib.flf_bias_grad(d.data_ptr() + 2 * off, db.data_ptr(), M, C, ws.data_ptr(), ws.numel(), None) == 0
        want = rows.double().sum(0)
        assert float((db.cpu().double() - want).abs().max()) <= 1e-4 * float(rows.double().abs().sum(0).max().sqrt() + 1)
