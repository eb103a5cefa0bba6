"""The adjoint on frames whose queues are no multiple of the 256 bytes its
per-path fields are aligned to (the fields come from one allocation, padded
field by field)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("size,spp", [((1, 1), 1), ((17, 13), 3), ((31, 33), 5), ((40, 23), 7)])
def test_adjoint_of_odd_sizes(photon, size, spp):
    from photon_gb300 import workloads
    sc, cam, st = workloads.differentiable(res=16, spp=spp, depth=6, texture=16)
    st.width, st.height = size
    r = photon.Renderer()
    r.set_scene(sc)
    r.render(cam, st, True)
    image = r.read_color()
    w = np.random.default_rng(3).uniform(0.5, 1.5, (size[1], size[0], 3)).astype(np.float32)
    g = r.adjoint(cam, st, w, sample_offset=0, color=True)
    assert g["replay_mismatches"] == 0
    # the pass's own samples are the rendered ones; its image adds them per
    # channel with atomics, in any order: 2^-24 per addition of the spp
    assert np.allclose(g["color"][..., :3], image[..., :3], rtol=(spp + 2) * 2.0 ** -23, atol=1e-7)
    for k in ("materials", "volumes", "texels"):
        assert np.isfinite(g[k]).all()
    h = r.adjoint(cam, st, 2.0 * w, sample_offset=0)
    # linear in the loss gradient: the products double exactly, their atomic
    # sums round in another order (about 1e4 addends, 2^-24 each, as a random walk)
    scale = np.abs(g["materials"]).max()
    assert np.allclose(h["materials"], 2.0 * g["materials"], rtol=1e-4, atol=1e-4 * scale)
    r.close()
