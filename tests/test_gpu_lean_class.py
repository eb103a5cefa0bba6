"""Unsorted lean scenes are shaded by the kernel of the smallest shading class
that has the lobes their materials have between them (lean_class_of): the same
images as the kernel with every lobe (tuning key shade_classes 0), bit for
bit, for material sets that end in each class, alone and in a batch."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

#            metallic, specTrans, specular, clearcoat, sheen
SETS = {
    "diffuse": [(0, 0, 0, 0, 0)],
    "diffuse_spec": [(0.4, 0, 0.5, 0, 0), (0, 0, 0, 0, 0)],
    "metal": [(1, 0, 0.5, 0, 0)],
    "metal_coat": [(1, 0, 0.5, 0.8, 0)],
    "plastic_coat": [(0.2, 0, 0.5, 0.7, 0)],
    "glass": [(0, 1, 0, 0, 0)],
    "glass_spec_coat": [(0, 1, 0.5, 0.6, 0)],
    "sheen": [(0, 0, 0.5, 0, 0.7), (0, 1, 0.5, 0.5, 0)],
}


def _scene(name):
    from photon_gb300 import workloads
    sc, cam, st = workloads.box_room()
    for k, m in enumerate(sc.materials[:3]):
        p = SETS[name][k % len(SETS[name])]
        m.metallic, m.transmission, m.specular, m.clearcoat, m.sheen = (float(x) for x in p)
        m.roughness = 0.3 + 0.2 * k
    st.width, st.height, st.pixel_samples, st.max_depth = 96, 80, 3, 6
    return sc, cam, st


def _image(photon, scene, classes, batch):
    from photon_gb300 import tuning_get, tuning_set
    from photon_gb300.renderer import render_batch
    old = tuning_get("shade_classes")
    tuning_set("shade_classes", classes)
    try:
        sc, cam, st = scene
        rs = [photon.Renderer() for _ in range(2 if batch else 1)]
        for r in rs:
            r.set_scene(sc)
        if batch:
            render_batch([(r, cam, st, True) for r in rs])
        else:
            rs[0].render(cam, st, True)
        out = [r.read_color() for r in rs]
        for r in rs:
            r.close()
        return np.stack(out)
    finally:
        tuning_set("shade_classes", old)


@pytest.mark.parametrize("batch", [False, True])
@pytest.mark.parametrize("name", sorted(SETS))
def test_smallest_class_keeps_the_image(photon, name, batch):
    scene = _scene(name)
    a, b = _image(photon, scene, 1, batch), _image(photon, scene, 0, batch)
    assert np.isfinite(a).all() and a.max() > 0
    assert np.array_equal(a, b)
