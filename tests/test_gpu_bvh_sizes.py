"""The GPU build around the sizes where its clustering changes from the whole
grid to one block (512 clusters) and where blocks fill (bvh_gpu.cu, k_ploc),
with duplicate and degenerate triangles: the leaves cover the triangles and
every ray's hit equals the host-built tree's (same triangle tests, other
tree)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("radius", [2, 8, 32])
@pytest.mark.parametrize("tris", [1, 2, 3, 511, 512, 513, 1023, 1025, 4097, 40_000])
def test_gpu_tree_hits_equal_host_tree(photon, tris, radius):
    import torch
    from photon_gb300 import tuning_get, tuning_set
    rng = np.random.default_rng(tris)
    corner = rng.uniform(-5, 5, (tris, 1, 3))
    pos = np.float32(corner + rng.uniform(-0.4, 0.4, (tris, 3, 3)))
    if tris > 500:
        pos[5] = pos[6]            # a duplicate
        pos[7] = pos[7, :1]        # a point
        pos[9:40, :, 1] = 0.25     # a flat patch
    pos = pos.reshape(-1, 3)
    idx = np.arange(3 * tris, dtype=np.uint32).reshape(-1, 3)
    n = 20_000
    o = np.float32(rng.uniform(-7, 7, (n, 3)))
    d = rng.normal(size=(n, 3))
    d = np.float32(d / np.linalg.norm(d, axis=1, keepdims=True))
    rays = [torch.from_numpy(a).cuda() for a in (o, d, np.zeros(n, np.float32), np.full(n, 1e3, np.float32))]
    keys = {k: tuning_get(k) for k in ("gpu_bvh", "ploc_radius")}
    try:
        tuning_set("ploc_radius", radius)
        hits = []
        for gpu in (1, 0):
            tuning_set("gpu_bvh", gpu)
            acc = photon.Accel(pos, idx)
            assert acc.info()["tri_bytes"] == 48 * tris
            hits.append(acc.trace_closest_compact(*rays).cpu().numpy())
            acc.close()
    finally:
        for k, v in keys.items():
            tuning_set(k, v)
    a, b = hits
    assert np.array_equal(a[:, 0].view(np.uint32), b[:, 0].view(np.uint32))  # distances, bit for bit
    other = a[:, 1].view(np.uint32) != b[:, 1].view(np.uint32)  # another triangle at the same distance: ties
    prim = np.stack([a[:, 1].view(np.uint32), b[:, 1].view(np.uint32)], 1)[other]
    assert set(prim.ravel().tolist()) <= {5, 6, *range(9, 40)}  # the duplicates, and the patch's overlaps
