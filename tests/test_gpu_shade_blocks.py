"""Shading blocks that work in step (warp_feed.cuh, block_share): queues of one
path, of part of a warp, of part of a block, around one block and around one
block per SM, against the oracle, for lean, full and volume shading."""
import numpy as np
import pytest

from tests.parity import MIN_PATH_FRACTION, close_fraction

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kind", ["glass", "textures", "volume", "alpha"])
@pytest.mark.parametrize("size", [(1, 1), (31, 1), (33, 1), (73, 7), (512, 1), (171, 3), (304, 257)])
def test_frames_match_oracle(photon, oracle_lib, kind, size):
    from photon_gb300 import workloads
    sc, cam, st = workloads.feature_scene(kind)
    st.width, st.height = size
    st.pixel_samples = 1
    st.adaptive_sampling = 0
    r, ref = photon.Renderer(), oracle_lib.CpuRenderer("oracle")
    for x in (r, ref):
        x.set_scene(sc)
        x.render(cam, st, True)
    n = size[0] * size[1]
    for channel in ("color", "albedo"):
        got, want = r.read(channel), ref.read(channel)
        assert np.array_equal(np.isfinite(got), np.isfinite(want))
        # of a short frame at most one path may differ (a transcendental
        # function's last place, 2e-5 of the paths of the workloads)
        assert close_fraction(got, want) >= (MIN_PATH_FRACTION if n > 1000 else 1.0 - 1.0 / n), channel
    r.close()
    ref.close()
