"""flf_autotune, the shapes it may choose and those it keeps.

The two directions need different shared memory: from two frames on, back projection needs more than
forward (its output exchange, against one operand table each), and at Nnum 19 with four frames and Nnum 21
with two some shapes fit forward only.  Projections afterwards against the FP64 oracle: 2e-5 of the maximum.
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


def test_shapes_of_another_kernel_are_not_taken_over(mods, tmp_path):
    """A cache entry without the kernel's form (its rows per chunk are none that tuning gives) stays unused."""
    import json
    import torch
    projector, psfmatrix, synthetic = mods
    N, Y, X, hs = 7, 56, 63, [43, 15, 29]
    H, Ht = synthetic.random_psf(N, hs, seed=5)
    hm = psfmatrix.HMatrixArrays(H, Ht)
    p = projector.Projector_gb300()
    p._prepare(p.context(hm), Y, X, hm)
    old = "|".join(str(v) for v in (torch.cuda.get_device_name(0), N, len(hs),
                                    tuple(tuple(hm.PSFShape(c)) for c in range(len(hs))), Y, X, 2, p.fft_size,
                                    p._shape_key[3]))
    stale = {"stages": 2, "chunk_rows_forward": 4, "chunk_rows_backward": 4, "split": 1}
    path = tmp_path / "tune.json"
    path.write_text(json.dumps({old: stale}))
    tuned = p.autotune(hm, 2, Y, X, cache_path=str(path))
    assert tuned != stale
    kept = json.loads(path.read_text())
    assert kept.pop(old) == stale and list(kept.values()) == [tuned]


@pytest.mark.parametrize("rows", [3, 7, 15])
def test_any_number_of_rows(mods, rows):
    """The rule takes odd numbers of rows (15 at Nnum 15), so they can be asked for and kept as a tuned shape."""
    projector, psfmatrix, synthetic = mods
    N, T, Y, X = 15, 1, 45, 31
    H, Ht = synthetic.random_psf(N, [31, 61], seed=rows)
    hm = psfmatrix.HMatrixArrays(H, Ht)
    rng = np.random.default_rng(rows)
    img = rng.random((T, Y, X)).astype(np.float32)
    vol = rng.random((2, T, Y, X)).astype(np.float32)
    for tuned in (False, True):
        p = projector.Projector_gb300()
        ctx = p.context(hm)
        if tuned:
            p._prepare(ctx, Y, X, hm)
            ctx.set_tuned(Y, X, {"stages": 2, "chunk_rows_forward": rows, "chunk_rows_backward": rows + 2, "split": 1})
        else:
            ctx.set_option("mac_chunk_rows", rows)
        assert rel(p.BackwardProjectACC(hm, img, None),
                   O.backward_project(Ht, img, N, method="direct", dtype=np.float64)) < TOL
        assert rel(p.ForwardProjectACC(hm, vol, None),
                   O.forward_project(H, vol, N, method="direct", dtype=np.float64)) < TOL


@pytest.mark.parametrize("T", [1, 2])
@pytest.mark.parametrize("N,split", [(13, 2), (15, 2)])
def test_row_shares_of_two_column_warps(mods, N, split, T):
    """mac_split with two column warps, which counts at one and two frames: up to four row shares, forward at one
    frame beside the helper and copy warps."""
    projector, psfmatrix, synthetic = mods
    H, Ht = synthetic.random_psf(N, [2 * N + 1, 4 * N + 1], seed=N)
    hm = psfmatrix.HMatrixArrays(H, Ht)
    p = projector.Projector_gb300()
    p.context(hm).set_option("mac_split", split)
    rng = np.random.default_rng(T)
    img = rng.random((T, 3 * N, 2 * N + 5)).astype(np.float32)
    vol = rng.random((2, T, 3 * N, 2 * N + 5)).astype(np.float32)
    assert rel(p.BackwardProjectACC(hm, img, None),
               O.backward_project(Ht, img, N, method="direct", dtype=np.float64)) < TOL
    assert rel(p.ForwardProjectACC(hm, vol, None),
               O.forward_project(H, vol, N, method="direct", dtype=np.float64)) < TOL
