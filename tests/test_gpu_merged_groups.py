"""One frame of three or more transform groups: all groups in one multiply-accumulate launch,
their transforms on several streams, the forward output a set per group that the consumer adds.

Against the FP64 oracle (2e-5 of the maximum; Richardson-Lucy 1e-4), and against the same frames
taken two at a time, which go group by group.  Plane subsets reach two, three and all groups; five
frames end in a pass of one.
"""

import numpy as np
import pytest

from oracle import lf_oracle as O

pytestmark = pytest.mark.gpu

HS = [61, 41, 21, 11, 21, 31, 61, 51]     # Nnum 5, 30 x 35 px: transforms of 10, 12, 14 lenslets


def rel(a, b):
    return float(np.max(np.abs(np.asarray(a, np.float64) - b)) / np.max(np.abs(b)))


@pytest.fixture(scope="module")
def env(built_lib):
    import _flf
    import lfdeconv
    import projector
    import psfmatrix
    import synthetic
    _flf.load_library()
    H, Ht = synthetic.random_psf(5, HS, seed=9)
    return projector, lfdeconv, psfmatrix.HMatrixArrays(H, Ht), H, Ht


@pytest.mark.parametrize("streams", [1, 2])
@pytest.mark.parametrize("planes", [None, [0, 2, 3, 6], [7, 1, 5], [4, 2], [6]])
def test_projections(env, streams, planes):
    projector, _, hm, H, Ht = env
    p = projector.Projector_gb300()
    p.context(hm).set_option("streams", streams)
    rng = np.random.default_rng(1)
    img = rng.random((1, 30, 33)).astype(np.float32)
    vol = rng.random((len(HS), 1, 30, 33)).astype(np.float32)
    idx = list(range(len(HS))) if planes is None else planes
    bk = p.BackwardProjectACC(hm, img, planes)
    assert p.geometry()["groups"] >= 3
    want = O.backward_project([Ht[i] for i in idx], img, 5, method="direct", dtype=np.float64)
    assert rel(bk[idx], want) < 2e-5
    assert not np.any(np.delete(bk, idx, axis=0))
    fw = p.ForwardProjectACC(hm, vol, planes)
    assert rel(fw, O.forward_project([H[i] for i in idx], vol[idx], 5, method="direct", dtype=np.float64)) < 2e-5


@pytest.mark.parametrize("frames", [1, 5])
@pytest.mark.parametrize("trust", [False, True])
@pytest.mark.parametrize("graphs", [False, True])
def test_richardson_lucy(env, frames, trust, graphs):
    projector, lfdeconv, hm, H, Ht = env
    p = projector.Projector_gb300()
    p.useGraphs = graphs
    rng = np.random.default_rng(2)
    img = rng.random((frames, 30, 33)).astype(np.float32) + 0.5
    mask = None
    if trust:
        mask = np.ones((30, 33), np.float32)
        mask[10:15, 10:15] = 0
        img *= mask
    got = lfdeconv.DeconvRL(hm, None, 3, None, logPrint=False, projector=p, im=img, prevedel=not trust, trustMask=mask)
    for t in range(frames):       # frames are independent: each against the oracle
        want = O.deconv_rl(H, Ht, 5, 3, im=img[t:t + 1], method="direct", dtype=np.float64, prevedel=not trust,
                           trust_mask=mask) if trust else O.deconv_rl(H, Ht, 5, 3, im=img[t:t + 1], method="direct",
                                                                      dtype=np.float64)
        assert rel(got[:, t:t + 1], want) < 1e-4
