"""flf_autotune where the two directions need different shared memory.

From two frames on, back projection needs more than forward (its output exchange, against one operand
table each): at Nnum 19 with four frames and Nnum 21 with two some shapes fit forward only.  Projections
afterwards against the FP64 oracle: 2e-5 of the maximum.
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


@pytest.mark.parametrize("N,T,Y,X", [(15, 1, 45, 31), (19, 3, 38, 57), (19, 4, 57, 40), (21, 2, 42, 63), (21, 4, 63, 42)])
def test_every_frame_count_can_be_tuned(mods, N, T, Y, X):
    projector, psfmatrix, synthetic = mods
    H, Ht = synthetic.random_psf(N, [2 * N + 1, 4 * N + 1], seed=N + T)
    hm = psfmatrix.HMatrixArrays(H, Ht)
    p = projector.Projector_gb300()
    tuned = p.autotune(hm, T, Y, X)
    assert tuned["stages"] in (2, 3) and tuned["split"] in (1, 2)
    rng = np.random.default_rng(T)
    img = rng.random((T, Y, X)).astype(np.float32)
    vol = rng.random((2, T, Y, X)).astype(np.float32)
    assert rel(p.BackwardProjectACC(hm, img, None),
               O.backward_project(Ht, img, N, method="direct", dtype=np.float64)) < TOL
    assert rel(p.ForwardProjectACC(hm, vol, None),
               O.forward_project(H, vol, N, method="direct", dtype=np.float64)) < TOL
