"""Ray batches of every length class of the back-end's kernels (accel.cu): one
ray per warp, fewer than 32, one full batch per warp without the work counter,
and batches drawn from it; each entry point against one long call."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_batch_lengths_agree(photon):
    import torch
    from photon_gb300 import workloads
    sc, cam, _ = workloads.procedural_500k(seed=3, n_objects=24, n_spheres=8, sphere_subdiv=2, torus_res=(20, 12),
                                           env_res=(16, 8))
    acc = photon.Accel(sc.positions, sc.indices, sc.normals, sc.material_ids)
    n = 400_003
    rng = np.random.default_rng(1)
    o = np.float32(rng.uniform(-15, 15, (n, 3)) + (0, 8, 0))
    d = rng.normal(size=(n, 3))
    d = np.float32(d / np.linalg.norm(d, axis=1, keepdims=True))
    t1 = np.full(n, 100.0, np.float32)
    t1[::97] = 0.0  # empty rays
    rays = [torch.from_numpy(a).cuda() for a in (o, d, np.zeros(n, np.float32), t1)]
    whole = [f(*rays) for f in (acc.trace_closest, acc.trace_closest_compact, acc.trace_occluded)]
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    warps = sms * 16 * 4
    for m in (1, 31, 33, warps // 2, warps // 2 + 1, 3 * warps, 32 * warps, 32 * warps + 1):
        m = min(m, n)
        for first in (0, n - m):
            part = [r[first:first + m].contiguous() for r in rays]
            for f, w in zip((acc.trace_closest, acc.trace_closest_compact, acc.trace_occluded), whole):
                out = f(*part)
                assert torch.equal(out.view(torch.uint8), w[first:first + m].contiguous().view(torch.uint8)), (m, first)
    acc.close()
