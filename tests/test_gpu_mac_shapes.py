"""The multiply-accumulate over its thread shapes and plane groups, against the FP64 oracle.

Channel pairs per lane and column warps change with Nnum (5: 13 pairs, one per
lane; 9: 41; 13: 85; 17: 145; 23: 265 pairs in five column warps), the row
shares with mac_split, the operand tables with the frames, and with few CTAs
per SM asked for (mac_ctas_per_sm) a forward CTA walks all planes, the helper
warp filling its two tables in turn.  FP32 against FP64: 2e-5 of the maximum.
"""

import numpy as np
import pytest

from oracle import lf_oracle as O

pytestmark = pytest.mark.gpu
TOL = 2e-5


def rel(a, b):
    return float(np.max(np.abs(np.asarray(a, np.float64) - b)) / np.max(np.abs(b)))


@pytest.fixture(scope="module")
def mods(built_lib):
    import _flf
    import projector
    import psfmatrix
    import synthetic
    _flf.load_library()
    return projector, psfmatrix, synthetic


@pytest.mark.parametrize("N,hs,Y,X,T,split", [
    (3, [7, 13], 14, 9, 1, 1), (3, [7], 11, 12, 5, 4), (9, [19, 37], 40, 31, 2, 1), (9, [37], 36, 45, 3, 2),
    (13, [27, 53], 52, 40, 1, 1), (13, [53], 33, 52, 4, 2), (17, [35], 51, 60, 3, 1), (17, [35, 69], 34, 51, 1, 1),
    (23, [47], 46, 69, 1, 1), (23, [47], 50, 46, 2, 1)])
def test_thread_shapes(mods, N, hs, Y, X, T, split):
    projector, psfmatrix, synthetic = mods
    H, Ht = synthetic.random_psf(N, hs, seed=N + T)
    hm = psfmatrix.HMatrixArrays(H, Ht)
    p = projector.Projector_gb300()
    if split > 1:      # the default otherwise (from Nnum 23 on no split can be asked for)
        p.context(hm).set_option("mac_split", split)
    rng = np.random.default_rng(T)
    img = rng.random((T, Y, X)).astype(np.float32)
    vol = rng.random((len(hs), T, Y, X)).astype(np.float32)
    assert rel(p.BackwardProjectACC(hm, img, None),
               O.backward_project(Ht, img, N, method="direct", dtype=np.float64)) < TOL
    assert rel(p.ForwardProjectACC(hm, vol, None),
               O.forward_project(H, vol, N, method="direct", dtype=np.float64)) < TOL


@pytest.mark.parametrize("planes", [1, 2, 3, 6, 7])
@pytest.mark.parametrize("T", [1, 2])
def test_planes_in_one_cta(mods, planes, T):
    """f = 36: 190 quads, so with one CTA per SM asked for every CTA takes all planes."""
    projector, psfmatrix, synthetic = mods
    N, Y, X = 5, 165, 160
    hs = [21] * planes
    H, Ht = synthetic.random_psf(N, hs, seed=planes)
    hm = psfmatrix.HMatrixArrays(H, Ht)
    p = projector.Projector_gb300()
    p.context(hm).set_option("mac_ctas_per_sm", 1)
    rng = np.random.default_rng(planes)
    vol = rng.random((planes, T, Y, X)).astype(np.float32)
    img = rng.random((T, Y, X)).astype(np.float32)
    assert rel(p.ForwardProjectACC(hm, vol, None),
               O.forward_project(H, vol, N, method="direct", dtype=np.float64)) < TOL
    assert rel(p.BackwardProjectACC(hm, img, None),
               O.backward_project(Ht, img, N, method="direct", dtype=np.float64)) < TOL


def test_dropped_chunk_with_helper_warp(mods):
    """A chunk that never arrives ends the streaming warps' waits and the helper's; the context stays usable."""
    projector, psfmatrix, synthetic = mods
    import _flf
    import torch
    N, Y, X, planes = 5, 165, 160, 5
    H, Ht = synthetic.random_psf(N, [21] * planes, seed=3)
    hm = psfmatrix.HMatrixArrays(H, Ht)
    p = projector.Projector_gb300()
    ctx = p.context(hm)
    ctx.set_option("mac_ctas_per_sm", 1)
    vol = torch.rand((planes, 1, Y, X), device="cuda")
    want = p.ForwardProjectACC(hm, vol, None)
    ctx.set_option("mac_wait_limit_us", 2000)
    ctx.set_option("test_drop_chunk", 2)
    img = torch.zeros((1, Y, X), device="cuda")
    s = torch.cuda.current_stream().cuda_stream
    ctx.forward(vol, img, 1, Y, X, None, stream=s)
    with pytest.raises(_flf.FlfError) as e:
        ctx.synchronize(s)
    assert e.value.code == -5
    ctx.set_option("test_drop_chunk", -1)
    ctx.set_option("mac_wait_limit_us", 1000000)
    assert np.array_equal(p.ForwardProjectACC(hm, vol, None), want)
