"""Adaptive sampling with several samples of a pixel in flight (AdaptState)
against one sample per wave: the same images bit for bit and the same number
of samples, around the 16 samples every pixel takes, over frames that hold
whole and broken waves, progressive calls and a wave after a failed one."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

CHANNELS = ("color", "depth", "normal", "albedo")


def _frames(photon, sc, cam, st, wave_paths, calls):
    from photon_gb300 import tuning_get, tuning_set
    default = tuning_get("wave_paths")
    tuning_set("wave_paths", wave_paths or default)
    try:
        r = photon.Renderer()
        r.set_scene(sc)
        out = []
        for k in range(calls):
            r.render(cam, st, reset=k == 0)
            out.append([r.read(c) for c in CHANNELS] + [np.array(r.stats()["pixel_samples"])])
        r.close()
        return out
    finally:
        tuning_set("wave_paths", default)


@pytest.mark.parametrize("kind", ["volume", "env", "alpha"])
@pytest.mark.parametrize("size,spp", [((1, 1), 40), ((33, 7), 2), ((64, 64), 16), ((127, 93), 17), ((301, 200), 35)])
def test_samples_side_by_side_equal_one_at_a_time(photon, kind, size, spp):
    from photon_gb300 import workloads
    sc, cam, st = workloads.feature_scene(kind)
    st.width, st.height = size
    st.pixel_samples, st.adaptive_sampling = spp, 1
    one = _frames(photon, sc, cam, st, 1024, 2)
    many = _frames(photon, sc, cam, st, None, 2)
    for a, b in zip(one, many):
        for x, y in zip(a, b):
            assert np.array_equal(x, y, equal_nan=True)


def test_planes_are_cleared_after_an_error(photon):
    from photon_gb300 import PhotonError, tuning_get, tuning_set, workloads
    sc, cam, st = workloads.feature_scene("volume")
    st.width, st.height, st.pixel_samples, st.adaptive_sampling = 64, 48, 20, 1
    want = _frames(photon, sc, cam, st, None, 1)[0]
    r = photon.Renderer()
    r.set_scene(sc)
    cap = tuning_get("wave_trip_cap")
    tuning_set("wave_trip_cap", 12)
    try:
        with pytest.raises(PhotonError):
            r.render(cam, st, True)
    finally:
        tuning_set("wave_trip_cap", cap)
    r.render(cam, st, True)
    for c, x in zip(CHANNELS, want):
        assert np.array_equal(r.read(c), x, equal_nan=True)
    r.close()
