"""Launch-shape options whose default is a rule can be set back to it.

The plane grouping shows in the byte count of the forward multiply-accumulate (one set of output spectra
per group of planes); the rows per stage change no result beyond rounding.
"""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def env(built_lib):
    import _flf
    import projector
    import psfmatrix
    import synthetic
    _flf.load_library()
    H, Ht = synthetic.random_psf(5, [21] * 6, seed=2)
    return projector, psfmatrix.HMatrixArrays(H, Ht), _flf


def mac_bytes(ctx, run):
    ctx.profile(True)
    run()
    return ctx.profile_read()["k_mac_fwd"]["bytes"]


def test_back_to_the_rule(env):
    projector, hm, _flf = env
    p = projector.Projector_gb300()
    ctx = p.context(hm)
    vol = np.random.default_rng(0).random((6, 1, 165, 160)).astype(np.float32)
    run = lambda: p.ForwardProjectACC(hm, vol, None)  # noqa: E731
    want = run()
    by_rule = mac_bytes(ctx, run)
    ctx.set_option("mac_ctas_per_sm", 1)
    assert mac_bytes(ctx, run) < by_rule
    ctx.set_option("mac_ctas_per_sm", 0)
    assert mac_bytes(ctx, run) == by_rule
    for name in ("mac_chunk_rows", "mac_chunk_rows_forward", "mac_chunk_rows_backward"):
        ctx.set_option(name, 4)
        ctx.set_option(name, 0)
        assert np.array_equal(run(), want)
        for bad in (-2, 66):
            with pytest.raises(_flf.FlfError):
                ctx.set_option(name, bad)
    for bad in (-1, 65):
        with pytest.raises(_flf.FlfError):
            ctx.set_option("mac_ctas_per_sm", bad)
    shape = {"stages": 3, "chunk_rows_forward": 6, "chunk_rows_backward": 8, "split": 1}
    ctx.set_tuned(165, 160, shape)
    got = run()
    assert np.allclose(got, want, rtol=1e-4)
    ctx.set_tuned(165, 160, dict.fromkeys(shape, 0))
    assert np.array_equal(run(), want)
    with pytest.raises(_flf.FlfError):
        ctx.set_tuned(165, 160, dict(shape, stages=0))
