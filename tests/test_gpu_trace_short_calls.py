"""Ray back-end calls at the edges of brief_lanes (warp_rules.h): 8 rays a warp
and whole warps, the last call whose rays are all in flight at once and the
first one that takes batches from the counter; single-level and two-level
scenes, with and without traversal counters, and the entry point without scratch
memory.  Every part equals the same rays of one long call."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("two_level", [False, True])
def test_edges_agree_with_a_long_call(photon, two_level):
    import torch
    from photon_gb300 import tuning_get, tuning_set, workloads
    sc = workloads.instanced_objects(n_instances=40, sphere_subdiv=2, flatten=not two_level)[0]
    more = dict(objects=sc.pt.objects, instances=sc.pt.instances) if two_level else {}
    acc = photon.Accel(sc.positions, sc.indices, sc.normals, sc.material_ids, **more)
    n = 200_001
    rng = np.random.default_rng(2)
    o = np.float32(rng.uniform(-3, 3, (n, 3)) + (0, 2, 0))
    d = rng.normal(size=(n, 3))
    d = np.float32(d / np.linalg.norm(d, axis=1, keepdims=True))
    rays = [torch.from_numpy(a).cuda() for a in (o, d, np.zeros(n, np.float32), np.full(n, 50.0, np.float32))]
    lib = photon.load()

    def static(*r):
        m = r[2].numel()
        out = torch.empty((m, 4), dtype=torch.float32, device="cuda")
        torch.cuda.synchronize()
        rc = lib.phc_trace_closest_compact_static(acc.h, *(x.data_ptr() for x in r), m, out.data_ptr(), None)
        assert rc == 0, lib.phc_accel_error().decode()
        return out

    calls = [acc.trace_closest, acc.trace_closest_compact, acc.trace_occluded, static]
    half = torch.cuda.get_device_properties(0).multi_processor_count * 16 * 4 // 2
    whole = [f(*rays) for f in calls]
    assert whole[2].any()
    count = tuning_get("count_traversal")
    try:
        for m in (4 * half + 1, 8 * half, 8 * half + 1, 16 * half + 1, 32 * half, 32 * half + 1):
            part = [r[n - m:].contiguous() for r in rays]
            for counting in (0, 1):
                tuning_set("count_traversal", counting)
                for f, w in zip(calls, whole):
                    assert torch.equal(f(*part).view(torch.uint8), w[n - m:].contiguous().view(torch.uint8)), m
    finally:
        tuning_set("count_traversal", count)
        acc.close()
