"""The byte counts of the profile follow the layouts: spectra that the multiply-accumulate reads, and those the
back projection writes, in quad order (four values per frequency quad), the forward output in row order.

One transform group of six planes, one, two and five frames (a pass of four and one): counts by formula.
"""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("T", [1, 2, 5])
def test_bytes_of_one_group(built_lib, T):
    import _flf
    import projector
    import psfmatrix
    import synthetic
    _flf.load_library()
    N, Y, X, nz = 5, 165, 160, 6
    H, Ht = synthetic.random_psf(N, [21] * nz, seed=2)
    hm = psfmatrix.HMatrixArrays(H, Ht)
    p = projector.Projector_gb300()
    ctx = p.context(hm)
    ctx.set_option("mac_ctas_per_sm", 1)              # one CTA takes all planes: one set of output spectra
    img = np.ones((T, Y, X), np.float32)
    vol = np.ones((nz, T, Y, X), np.float32)

    def counts(run):
        run()
        ctx.profile(True)
        run()
        return {k: v["bytes"] for k, v in ctx.profile_read().items()}
    fw = counts(lambda: p.ForwardProjectACC(hm, vol, None))
    bk = counts(lambda: p.BackwardProjectACC(hm, img, None))
    g = p.geometry()
    assert g["groups"] == 1
    f, NN, c = g["f"], N * N, N // 2
    fh, passes = f // 2 + 1, 1 if T <= 4 else 2
    Ly, Lx = Y // N, X // N
    chan = 4 * NN * Ly * (-(-Lx // 4) * 4)            # one frame of channel-major images
    quad, row = 8 * NN * 2 * fh * (fh + 1), 8 * NN * f * fh
    matrices = nz * fh * fh * (c + 1) * (c + 2) * 2 * ((NN + 1) // 2) * 8 * passes
    assert fw["k_rfft2"] == T * nz * (chan + quad)
    assert fw["k_mac_fwd"] == matrices + T * (nz * quad + row)
    assert bk["k_rfft2"] == T * (chan + quad)
    assert bk["k_mac_bwd"] == matrices + T * quad * (1 + nz)
    assert bk["k_irfft2"] == T * nz * (chan + quad)
