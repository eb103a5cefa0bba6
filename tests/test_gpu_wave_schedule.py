"""The branched schedule of a wave (shadow rays beside the next bounce, the parts
of a bounce's shading beside one another), captured into a graph or launched
as it is, against every kernel on one stream in turn (time_kernels): the same
frames bit for bit and the same rays, over several waves, for every kind of
scene that takes another set of launches."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SIZE = (96, 64)
CHANNELS = ("color", "depth", "normal", "albedo")
COUNTS = ("pixel_samples", "closest_rays", "shadow_rays")


def _scene(kind):
    from photon_gb300 import workloads
    if kind == "procedural":
        return workloads.procedural_500k(n_objects=24, n_spheres=8, sphere_subdiv=2, torus_res=(20, 12), env_res=(16, 8))
    return workloads.instanced_objects() if kind == "instanced" else workloads.feature_scene(kind)


def _frames(photon, scene, keys):
    from photon_gb300 import tuning_get, tuning_set
    old = {k: tuning_get(k) for k in keys}
    sc, cam, st = scene
    r = photon.Renderer()
    try:
        for k, v in keys.items():
            tuning_set(k, v)
        r.set_scene(sc)
        out = []
        for reset in (True, False):
            r.render(cam, st, reset)
            out += [r.read(c) for c in CHANNELS] + [np.array([r.stats()[c] for c in COUNTS])]
        return out
    finally:
        r.close()
        for k, v in old.items():
            tuning_set(k, v)


@pytest.mark.parametrize("adaptive,spp,lanes", [(0, 3, 1), (0, 9, 4), (1, 20, 1), (1, 40, 16)])
@pytest.mark.parametrize("sort", [False, True])
@pytest.mark.parametrize("kind", ["procedural", "glass", "lights", "alpha", "volume", "instanced"])
def test_branched_equals_serial(photon, kind, sort, adaptive, spp, lanes):
    sc, cam, st = _scene(kind)
    st.width, st.height = SIZE
    st.pixel_samples, st.adaptive_sampling = spp, adaptive
    keys = dict(wave_paths=lanes * SIZE[0] * SIZE[1], class_threshold=0)
    if sort:
        keys["sort_threshold"] = 1
    want = _frames(photon, (sc, cam, st), dict(keys, time_kernels=1))
    for graph in (0, 1):
        got = _frames(photon, (sc, cam, st), dict(keys, time_kernels=0, use_graph=graph))
        for a, b in zip(want, got):
            assert np.array_equal(a, b, equal_nan=True), graph


@pytest.mark.parametrize("waves", [1, 3])
@pytest.mark.parametrize("kind", ["procedural", "lights", "volume"])
def test_batch_equals_single_renders(photon, kind, waves):
    """One wave of a batch is launched as it is, several are captured."""
    from photon_gb300 import tuning_get, tuning_set
    from photon_gb300.renderer import render_batch
    sc, cam, st = _scene(kind)
    st.width, st.height = SIZE
    st.pixel_samples, st.adaptive_sampling = 6, 0
    want = _frames(photon, (sc, cam, st), dict(time_kernels=1))[0]
    old = tuning_get("batch_wave_paths")
    rs = [photon.Renderer() for _ in range(3)]
    try:
        tuning_set("batch_wave_paths", 18 * SIZE[0] * SIZE[1] // waves)
        for r in rs:
            r.set_scene(sc)
        render_batch([(r, cam, st, True) for r in rs])
        for r in rs:
            assert np.array_equal(r.read("color"), want)
    finally:
        tuning_set("batch_wave_paths", old)
        for r in rs:
            r.close()
