"""The two weight-gradient kernels on either side of the rule between them, against float64.

Small volumes go tap by tap (64-voxel stages), larger ones by row blocks (4 rows, segments of 64 or 128
voxels, steps of 16).  Shapes just below and above each line of the rule, with and without a workspace,
and row-block shapes at the edges of rows, segments and steps.  FP32 sums of exact BF16 products: 1e-4
of the largest gradient.
"""

import pytest

pytestmark = pytest.mark.gpu


def check(shape, Ci, Co, slices):
    import torch
    import _flf
    _flf.load_library()
    g = torch.Generator(device="cuda").manual_seed(Ci * Co + shape[3])
    x = torch.randn(shape + (Ci,), generator=g, device="cuda").bfloat16()
    dy = torch.randn(shape + (Co,), generator=g, device="cuda").bfloat16()
    p = torch.nn.functional.pad(x.double(), (0, 0, 1, 1, 1, 1, 1, 1))
    _, Z, Y, X = shape
    want = torch.stack([p[:, k // 9:k // 9 + Z, k // 3 % 3:k // 3 % 3 + Y, k % 3:k % 3 + X].reshape(-1, Ci).T
                        @ dy.double().reshape(-1, Co) for k in range(27)])
    ws = torch.full((max(slices * 27 * Ci * Co, 1),), float("nan"), device="cuda")
    dw = torch.ones((27, Ci, Co), device="cuda")          # it adds to what is there
    _flf.conv3d_wgrad(x, dy, dw, ws=ws if slices else None)
    assert float((dw.double() - 1 - want).abs().max()) <= 1e-4 * float(want.abs().max().clamp_min(1))
    again = torch.ones_like(dw)
    _flf.conv3d_wgrad(x, dy, again, ws=ws if slices else None)
    assert torch.equal(again, dw)


@pytest.mark.parametrize("shape,Ci,Co", [
    ((1, 25, 16, 9), 16, 16), ((1, 26, 16, 9), 16, 16), ((1, 5, 20, 25), 16, 32), ((1, 5, 20, 26), 16, 32),
    ((1, 10, 20, 15), 32, 32), ((1, 10, 21, 15), 32, 32), ((1, 4, 16, 16), 32, 64), ((1, 4, 16, 17), 32, 64),
    ((1, 4, 11, 16), 64, 64), ((1, 4, 11, 17), 64, 64), ((1, 2, 8, 8), 128, 128), ((1, 2, 8, 9), 128, 128),
    ((1, 2, 7, 9), 96, 96), ((1, 4, 9, 13), 48, 80), ((2, 1, 1, 3), 16, 128)])
@pytest.mark.parametrize("slices", [0, 2, 64])
def test_either_side_of_the_rule(built_lib, shape, Ci, Co, slices):
    check(shape, Ci, Co, slices)


@pytest.mark.parametrize("X", [63, 64, 65, 127, 128, 129, 260])
@pytest.mark.parametrize("Ci,Co", [(16, 16), (16, 32), (32, 16), (32, 32), (64, 32)])
@pytest.mark.parametrize("slices", [0, 1, 3, 64])
def test_row_blocks_at_their_edges(built_lib, X, Ci, Co, slices):
    check((2, 5, 13, X), Ci, Co, slices)


@pytest.mark.parametrize("C", [8, 16, 24, 64, 128])
@pytest.mark.parametrize("M", [1, 7, 63, 64, 65, 128])
def test_bias_gradient_of_few_rows(built_lib, C, M):
    """Up to 64 rows one channel per thread, then 16-byte loads."""
    import torch
    import _flf
    lib = _flf.load_library()
    g = torch.randn((M, C), generator=torch.Generator().manual_seed(C + M)).bfloat16()
    db = torch.ones(C, device="cuda")
    ws = torch.full((256,), float("nan"), device="cuda")
    d = g.cuda()
    assert lib.flf_bias_grad(d.data_ptr(), db.data_ptr(), M, C, ws.data_ptr(), ws.numel(), None) == 0
    want = g.double().sum(0)
    assert float((db.cpu().double() - 1 - want).abs().max()) <= 1e-5 * float(g.double().abs().sum(0).max() + 1)
