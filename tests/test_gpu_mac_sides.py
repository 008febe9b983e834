"""Warps per side of a frequency quad in the multiply-accumulate, against the FP64 oracle.

Column warps 1 (Nnum 5: one channel pair per lane; 11: two), 2 (15), 3 (19), 4 (21),
5 (23), 6 (25) and 7 (29: sides together) with the frame counts at which a thread
takes one side; 5 frames: a launch of four or three and the rest.  FP32 against
FP64: 2e-5 of the maximum.
"""

import numpy as np
import pytest

from oracle import lf_oracle as O

pytestmark = pytest.mark.gpu
TOL = 2e-5


def rel(a, b):
    return float(np.max(np.abs(np.asarray(a, np.float64) - b)) / np.max(np.abs(b)))


@pytest.mark.parametrize("N,hs,Y,X,T", [
    (5, [11, 21], 25, 18, 2), (11, [23, 45], 33, 47, 1), (11, [23], 44, 33, 5), (15, [31, 61], 45, 31, 3),
    (19, [39], 57, 40, 1), (19, [39, 77], 38, 57, 2), (21, [43], 42, 63, 2), (23, [47], 46, 70, 4),
    (25, [51], 50, 51, 3), (29, [59], 58, 58, 2)])
def test_side_warps(built_lib, N, hs, Y, X, T):
    import _flf
    import projector
    import psfmatrix
    import synthetic
    _flf.load_library()
    H, Ht = synthetic.random_psf(N, hs, seed=N + T)
    hm = psfmatrix.HMatrixArrays(H, Ht)
    p = projector.Projector_gb300()
    rng = np.random.default_rng(T)
    img = rng.random((T, Y, X)).astype(np.float32)
    vol = rng.random((len(hs), T, Y, X)).astype(np.float32)
    assert rel(p.BackwardProjectACC(hm, img, None),
               O.backward_project(Ht, img, N, method="direct", dtype=np.float64)) < TOL
    assert rel(p.ForwardProjectACC(hm, vol, None),
               O.forward_project(H, vol, N, method="direct", dtype=np.float64)) < TOL
