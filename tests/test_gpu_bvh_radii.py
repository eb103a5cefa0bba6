"""The GPU build at every search radius on meshes whose clustering fills the
grid: one cluster tile per block of the whole grid, and several (bvh_gpu.cu,
k_ploc); hits as the host-built tree's."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", params=[100_003, 200_000])
def mesh(request, photon):
    import torch
    from photon_gb300 import tuning_get, tuning_set
    tris, n = request.param, 50_000
    rng = np.random.default_rng(tris)
    corner = rng.uniform(-5, 5, (tris, 1, 3))
    pos = np.float32(corner + rng.uniform(-0.1, 0.1, (tris, 3, 3))).reshape(-1, 3)
    idx = np.arange(3 * tris, dtype=np.uint32).reshape(-1, 3)
    o = np.float32(rng.uniform(-7, 7, (n, 3)))
    d = rng.normal(size=(n, 3))
    d = np.float32(d / np.linalg.norm(d, axis=1, keepdims=True))
    rays = [torch.from_numpy(a).cuda() for a in (o, d, np.zeros(n, np.float32), np.full(n, 1e3, np.float32))]
    old = tuning_get("gpu_bvh")
    tuning_set("gpu_bvh", 0)
    try:
        acc = photon.Accel(pos, idx)
        want = acc.trace_closest_compact(*rays).cpu().numpy()
        acc.close()
    finally:
        tuning_set("gpu_bvh", old)
    return pos, idx, rays, want


@pytest.mark.parametrize("radius", [2, 4, 8, 16, 32])
def test_hits_equal_host_tree(photon, mesh, radius):
    from photon_gb300 import tuning_get, tuning_set
    pos, idx, rays, want = mesh
    old = tuning_get("ploc_radius")
    tuning_set("ploc_radius", radius)
    try:
        acc = photon.Accel(pos, idx)
        got = acc.trace_closest_compact(*rays).cpu().numpy()
        acc.close()
    finally:
        tuning_set("ploc_radius", old)
    assert (got[:, 1].view(np.uint32) != 0xFFFFFFFF).mean() > 0.2
    assert np.array_equal(got[:, 0].view(np.uint32), want[:, 0].view(np.uint32))  # distances, bit for bit
