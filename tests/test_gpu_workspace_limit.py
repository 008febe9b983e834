"""A merged single-frame launch whose workspaces do not fit goes group by group instead.

Twelve planes in eight transform groups.  test_workspace_limit stands for a device without more memory:
projections that need more fail as when cudaMalloc does.  Against the FP64 oracle: 2e-5 of the maximum
(Richardson-Lucy 1e-4).
"""

import numpy as np
import pytest

from oracle import lf_oracle as O

pytestmark = pytest.mark.gpu

HS = [21, 31, 41, 51, 61, 71, 81, 91, 101, 111, 121, 131]     # Nnum 5, 30 x 33 px: eight transform groups


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
    return projector, lfdeconv, psfmatrix.HMatrixArrays(H, Ht), H, Ht, _flf


@pytest.mark.parametrize("frames", [1, 5])
@pytest.mark.parametrize("kind", ["forward", "backward", "rl", "rl_graph"])
def test_falls_back_to_one_group_at_a_time(env, kind, frames):
    projector, lfdeconv, hm, H, Ht, _flf = env
    rng = np.random.default_rng(4)
    img = rng.random((frames, 30, 33)).astype(np.float32) + 0.5
    vol = rng.random((len(HS), frames, 30, 33)).astype(np.float32)

    def run(p):
        p.useGraphs = kind == "rl_graph"
        if kind == "forward":
            return p.ForwardProjectACC(hm, vol, None)
        if kind == "backward":
            return p.BackwardProjectACC(hm, img, None)
        return lfdeconv.DeconvRL(hm, None, 2, None, logPrint=False, projector=p, im=img)

    def attempt(limit):
        """(result, bytes held after two calls) in a fresh context, or None where the call is refused."""
        p = projector.Projector_gb300()
        p.context(hm).set_option("test_workspace_limit", limit)
        try:
            out = run(p)
        except _flf.FlfError as e:
            assert e.code == -3               # out of memory, reported as such
            p.context(hm).set_option("test_workspace_limit", 0)
            run(p)                            # and the context stays usable
            return None
        assert np.array_equal(run(p), out)
        return out, p.context(hm).memory_usage()

    free, most = attempt(0)
    limit, got = 1 << 14, None
    while got is None:                        # up to the first limit that the call fits
        limit = limit * 5 // 4
        got = attempt(limit)
    out, held = got
    if frames == 1:
        assert held < most                    # a merged launch holds more: it did not fit, the call went on
    if kind == "forward":
        want = O.forward_project(H, vol, 5, method="direct", dtype=np.float64)
        assert rel(out, want) < 2e-5 and rel(free, want) < 2e-5
    elif kind == "backward":
        want = O.backward_project(Ht, img, 5, method="direct", dtype=np.float64)
        assert rel(out, want) < 2e-5 and rel(free, want) < 2e-5
    else:
        for t in range(frames):
            want = O.deconv_rl(H, Ht, 5, 2, im=img[t:t + 1], method="direct", dtype=np.float64)
            assert rel(out[:, t:t + 1], want) < 1e-4 and rel(free[:, t:t + 1], want) < 1e-4
