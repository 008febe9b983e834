"""Weight gradient: an infinity or NaN of the activations reaches only the taps that multiply it.

A row's last 16-voxel step may run past the image, where dy counts as zero; 0 times infinity must not
enter there.  Every element that is finite in float64 has to be finite and right (1e-4 of the largest, as
for finite activations), every other one not finite.
"""

import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("X", [1, 15, 16, 17, 31, 63, 64, 65, 72, 127, 129, 260])
@pytest.mark.parametrize("planes", [(1, 3, 6), (2, 12, 13)])     # small volumes go tap by tap
@pytest.mark.parametrize("Ci,Co", [(16, 16), (16, 32), (32, 16), (32, 32), (64, 64)])
@pytest.mark.parametrize("slices", [0, 64])
def test_nonfinite_activation_stays_in_its_taps(built_lib, planes, X, Ci, Co, slices):
    import torch
    import _flf
    _flf.load_library()
    g = torch.Generator().manual_seed(X)
    shape = planes + (X,)
    x = torch.randn(shape + (Ci,), generator=g).bfloat16()
    dy = torch.randn(shape + (Co,), generator=g).bfloat16()
    x[0, 1, 2, X - 1, 3] = float("inf")
    x[0, 0, 5, X - 1, 7] = float("nan")
    x[0, 2, 0, 0, 12] = float("-inf")
    ws = torch.full((max(1, slices * 27 * Ci * Co),), float("nan"), device="cuda")
    dw = torch.zeros((27, Ci, Co), device="cuda")
    _flf.conv3d_wgrad(x.cuda(), dy.cuda(), dw, ws=ws if slices else None)
    # float64, tap by tap over the voxels inside the volume only
    want = torch.zeros((27, Ci, Co), dtype=torch.float64)
    B, Z, Y, _ = shape
    for t in range(27):
        lo = [max(0, -d) for d in (t // 9 - 1, t // 3 % 3 - 1, t % 3 - 1)]
        hi = [n - max(0, d) for n, d in zip((Z, Y, X), (t // 9 - 1, t // 3 % 3 - 1, t % 3 - 1))]
        if any(h <= l for l, h in zip(lo, hi)):
            continue
        a = dy[:, lo[0]:hi[0], lo[1]:hi[1], lo[2]:hi[2]].double()
        d = (t // 9 - 1, t // 3 % 3 - 1, t % 3 - 1)
        b = x[:, lo[0] + d[0]:hi[0] + d[0], lo[1] + d[1]:hi[1] + d[1], lo[2] + d[2]:hi[2] + d[2]].double()
        want[t] = b.reshape(-1, Ci).T @ a.reshape(-1, Co)
    got = dw.cpu().double()
    ok = torch.isfinite(want)
    assert torch.equal(torch.isfinite(got), ok)
    assert float((got - want)[ok].abs().max()) <= 1e-4 * float(want[ok].abs().max().clamp_min(1))
