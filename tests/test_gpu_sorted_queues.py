"""Hit queues sorted by material or by shading class where the wave is large
enough and the bounce's queue passes the threshold: frames whose first bounces
are sorted and whose later ones are not, the class kernels on the plain and on the
batched path, class 0's kernel over the unsorted queues between, against the
frame without any sorting, bit for bit."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

WAVE = 256 * 256 * 8
DEPTH = 8


def _scene(kind):
    from photon_gb300 import workloads
    sc, cam, st = workloads.procedural_500k() if kind == "procedural" else workloads.feature_scene(kind)
    st.width = st.height = 256
    st.pixel_samples, st.max_depth, st.adaptive_sampling = 8, DEPTH, 0
    return sc, cam, st


def _render(photon, scene, keys, batch):
    from photon_gb300 import tuning_get, tuning_set
    from photon_gb300.renderer import render_batch
    old = {k: tuning_get(k) for k in keys}
    sc, cam, st = scene
    rs = [photon.Renderer() for _ in range(2 if batch else 1)]
    try:
        for k, v in keys.items():
            tuning_set(k, v)
        for r in rs:
            r.set_scene(sc)
        if batch:
            render_batch([(r, cam, st, True) for r in rs])
        else:
            rs[0].render(cam, st, True)
        return np.stack([r.read("color") for r in rs]), rs[0].stats()
    finally:
        for r in rs:
            r.close()
        for k, v in old.items():
            tuning_set(k, v)


@pytest.mark.parametrize("batch", [False, True])
@pytest.mark.parametrize("threshold", [1, 1 << 14, 1 << 16])
@pytest.mark.parametrize("kind", ["procedural", "glass", "lights"])
def test_sorted_and_unsorted_bounces(photon, kind, threshold, batch):
    sc, cam, st = _scene(kind)
    want, _ = _render(photon, (sc, cam, st), dict(sort_threshold=0, shade_classes=0), batch)
    assert 8 * threshold <= WAVE  # the wave sorts at all
    for classes, class_threshold in ((0, 0), (1, 0), (1, 1 << 30)):
        keys = dict(sort_threshold=threshold, shade_classes=classes, class_threshold=class_threshold)
        got, _ = _render(photon, (sc, cam, st), keys, batch)
        assert np.array_equal(got.view(np.uint32), want.view(np.uint32)), (classes, class_threshold)


def test_the_threshold_lies_between_the_bounces(photon):
    """The procedural frame above at 2^16: camera hits pass it (every path of
    the second bounce comes from one), a later bounce has paths but fewer."""
    sc, cam, st = _scene("procedural")
    total = []
    for depth in range(1, DEPTH + 1):
        st.max_depth = depth
        total.append(_render(photon, (sc, cam, st), {}, False)[1]["closest_rays"])
    paths = np.diff([WAVE] + [t for t in total])  # paths of bounce 1, 2, ...
    assert paths[0] >= 1 << 16
    assert 0 < paths[-1] < 1 << 16
