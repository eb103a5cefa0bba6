"""Queues shorter than the grid: the traversal and tracking warps then work on
fewer than 32 rays each (wave_common.cuh, spread_lanes).  Frames whose queues
hold one ray, less than a warp, around a power of two and around the switch to
full warps, against the oracle's per-sample radiance."""
import numpy as np
import pytest

from tests.parity import MIN_PATH_FRACTION, close_fraction

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kind", ["glass", "volume"])
@pytest.mark.parametrize("size", [(1, 1), (5, 1), (64, 38), (65, 75), (300, 260), (320, 245)])
def test_short_queue_frames_match_oracle(photon, oracle_lib, kind, size):
    from photon_gb300 import workloads
    sc, cam, st = workloads.feature_scene(kind)
    st.width, st.height = size
    st.pixel_samples = 1
    st.adaptive_sampling = 0
    r, ref = photon.Renderer(), oracle_lib.CpuRenderer("oracle")
    for x in (r, ref):
        x.set_scene(sc)
        x.render(cam, st, True)
    for channel in ("color", "depth", "normal", "albedo"):
        got, want = r.read(channel), ref.read(channel)
        assert np.array_equal(np.isfinite(got), np.isfinite(want))
        # of a few paths every one has to agree
        assert close_fraction(got, want) >= (MIN_PATH_FRACTION if size[0] * size[1] > 1000 else 1.0), channel
    assert r.stats()["pixel_samples"] == size[0] * size[1]
    r.close()
    ref.close()
