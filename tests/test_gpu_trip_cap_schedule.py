"""The loop-trip cap running out anywhere in a wave whose kernels run beside one
another: shadow rays beside the next bounce's sort, the adjoint's gradients
beside its rays.  Whatever the cap, a call either ends with the error or gives
the image of an uncapped one, and the renderer goes on as before."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

CAPS = [1, 2, 4, 7, 11, 16, 23, 32, 45, 64, 91, 128]


def _capped(cap, call):
    """call() under a trip cap; None when it reported the cap."""
    from photon_gb300 import PhotonError, tuning_get, tuning_set
    default = tuning_get("wave_trip_cap")
    tuning_set("wave_trip_cap", cap)
    try:
        return call()
    except PhotonError as e:
        assert "loop-trip cap" in str(e)
        return None
    finally:
        tuning_set("wave_trip_cap", default)


@pytest.mark.parametrize("kind", ["glass", "volume", "procedural"])
@pytest.mark.parametrize("use_graph", [0, 1])
def test_sorted_waves(photon, kind, use_graph):
    from photon_gb300 import tuning_get, tuning_set, workloads
    sc, cam, st = workloads.procedural_500k() if kind == "procedural" else workloads.feature_scene(kind)
    st.width, st.height, st.pixel_samples, st.adaptive_sampling = 160, 120, 3, 0
    keys = {k: tuning_get(k) for k in ("sort_threshold", "class_threshold", "use_graph", "wave_paths")}
    r, ref = photon.Renderer(), photon.Renderer()

    def image(x):  # the next samples of every pixel; a failed call takes none
        x.render(cam, st, True)
        return x.read_color()

    try:
        for x in (r, ref):
            x.set_scene(sc)
        tuning_set("sort_threshold", 1)
        tuning_set("class_threshold", 0)
        tuning_set("use_graph", use_graph)
        tuning_set("wave_paths", 160 * 120)  # three waves
        for cap in CAPS:
            got = _capped(cap, lambda: image(r))
            assert got is None or np.array_equal(got, image(ref)), cap
            assert np.array_equal(image(r), image(ref)), cap
    finally:
        r.close()
        ref.close()
        for k, v in keys.items():
            tuning_set(k, v)


@pytest.mark.parametrize("kind", ["glass", "volume"])
def test_adjoint(photon, kind):
    from photon_gb300 import tuning_get, tuning_set, workloads
    sc, cam, st = workloads.feature_scene(kind)
    st.width, st.height, st.pixel_samples, st.adaptive_sampling = 64, 48, 4, 0
    d = np.full((48, 64, 3), 1e-3, np.float32)
    default = tuning_get("sort_threshold")
    r = photon.Renderer()
    try:
        r.set_scene(sc)
        tuning_set("sort_threshold", 1)
        want = r.adjoint(cam, st, d, color=True)["color"]
        for cap in CAPS:
            _capped(cap, lambda: r.adjoint(cam, st, d))
            g = r.adjoint(cam, st, d, color=True)
            assert g["replay_mismatches"] == 0
            # sums of four samples per pixel, added in any order
            assert np.allclose(g["color"], want, rtol=4 * 2 ** -23, atol=0), cap
    finally:
        r.close()
        tuning_set("sort_threshold", default)
