"""Which surfaces let a path pass without a bounce: only scenes that have some
run the bounce iterations past the depth limit (scene_build.cpp,
material_may_pass).  Six layers in front of a lit wall at depth limits 1 and 2,
each material form that may pass and each that may not, against the oracle."""
import numpy as np
import pytest

from tests.parity import MIN_PATH_FRACTION, close_fraction

pytestmark = pytest.mark.gpu


def _hidden(m):
    m.hidden_to_camera = 1


def _blend(m):
    m.alpha_mode, m.opacity = 0, 0.4


def _blend_full(m):
    m.alpha_mode, m.opacity = 0, 1.0


def _mask_out(m):
    m.alpha_mode, m.opacity, m.alpha_cutoff = 2, 0.4, 0.5


def _mask_in(m):
    m.alpha_mode, m.opacity, m.alpha_cutoff = 2, 0.6, 0.5


def _opaque_mode(m):
    m.alpha_mode, m.opacity = 1, 0.3


def _attribute(m):
    m.alpha_mode = 0
    m.opacity_src.kind, m.opacity_src.index = 1, 0


def _colour_alpha(m):
    m.alpha_mode, m.base_color_alpha = 0, 1
    m.base_color_src.kind, m.base_color_src.index = 1, 0


@pytest.mark.parametrize("depth", [1, 2])
@pytest.mark.parametrize("form", [_hidden, _blend, _blend_full, _mask_out, _mask_in, _opaque_mode, _attribute,
                                  _colour_alpha])
def test_layers_match_oracle(photon, oracle_lib, form, depth):
    from photon_gb300 import _abi
    from photon_gb300.scene import SceneData, camera, settings
    pos, idx, mat = [], [], []
    for k in range(7):  # six layers, then the wall
        z, s = -0.3 * k, (1.0 if k < 6 else 3.0)
        pos += [(-s, -s, z), (s, -s, z), (s, s, z), (-s, s, z)]
        idx += [(4 * k, 4 * k + 1, 4 * k + 2), (4 * k, 4 * k + 2, 4 * k + 3)]
        mat += [0 if k < 6 else 1] * 2
    layer, wall = _abi.material_default(), _abi.material_default()
    layer.base_color[:] = (0.2, 0.5, 0.8)
    form(layer)
    wall.emission[:] = (1.0, 2.0, 3.0)
    attr = np.tile(np.float32([0.3, 0.6, 0.9, 0.35]), (28, 1))
    sc = SceneData(positions=np.float32(pos), indices=np.uint32(idx), material_ids=np.uint32(mat),
                   attributes=[attr, None, None, None, None], materials=[layer, wall])
    st = settings(48, 40, 1, depth, adaptive_sampling=0, background=(0.1, 0.2, 0.3, 1.0))
    cam = camera((0.0, 0.0, 3.0), (0.0, 0.0, 0.0), fovy_deg=50.0)
    r, ref = photon.Renderer(), oracle_lib.CpuRenderer("oracle")
    for x in (r, ref):
        x.set_scene(sc)
        x.render(cam, st, True)
    for channel in ("color", "depth", "albedo"):
        assert close_fraction(r.read(channel), ref.read(channel)) >= MIN_PATH_FRACTION, channel
    r.close()
    ref.close()
