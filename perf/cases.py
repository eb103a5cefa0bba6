"""The renderer's timed workloads: what a program that uses this library has it
do, through the public entry points, over the sizes it is used at.

  trace   the ray back-end on device arrays (photon_gb300.Accel): closest hits
          as full or compact records, and occlusion
  accel   a mesh that changes from frame to frame: acceleration structure built
          again, then traced
  render  one frame of a scene (photon_gb300.Renderer) and its channels read back
  batch   several independent renders in one call (photon_gb300.render_batch)
  diff    one optimisation step: image, loss, gradients (photon_gb300.diff)

listed() are the cases that are always measured, draw() gives more of the same
ranges.
"""
from __future__ import annotations

import math

import numpy as np
import torch

import photon_gb300
from photon_gb300 import diff, workloads
from photon_gb300.renderer import Accel, Renderer, render_batch

T_FAR = 200.0  # ray length limit, in units of a scene about 80 across


def listed():
    return [
        # picking, probes, a few sensor rays against a small scene: latency
        dict(name="trace_probe", kind="trace", op="compact", rays="camera", n=1000, tris=6000),
        # first hits of a full frame, with the whole hit record, as an
        # application that shades by itself asks for
        dict(name="trace_camera", kind="trace", op="closest", rays="camera", n=1024 * 1024, tris=500000),
        # texture-space bounces (light baking): origins in mesh order,
        # directions that share nothing
        dict(name="trace_bounce", kind="trace", op="compact", rays="bounce", n=723067, tris=500000),
        # visibility of light samples from surface points
        dict(name="trace_shadow", kind="trace", op="occluded", rays="shadow", n=1000003, tris=500000),
        # deforming geometry: build, then trace a quarter-size frame
        dict(name="accel_rebuild", kind="accel", op="closest", rays="camera", n=480 * 270, tris=50000),
        # interactive view of a large scene: one more sample per pixel and the
        # colour back on the host, every frame
        dict(name="viewer", kind="render", scene="procedural", tris=500000, width=640, height=360, spp=1, depth=6,
             progressive=True),
        # the small box room, final quality
        dict(name="box_room", kind="render", scene="box_room", tris=36, width=512, height=512, spp=64, depth=8,
             progressive=False),
        # the 500K-triangle scene under an environment map, final quality, with
        # the channels a denoiser wants: the largest case
        dict(name="procedural", kind="render", scene="procedural", tris=500000, width=1024, height=1024, spp=128,
             depth=8, progressive=False),
        # textures with normal maps and a heterogeneous volume, adaptive
        # sampling, an odd frame size
        dict(name="volume", kind="render", scene="volume", tris=500000, width=811, height=613, spp=20, depth=12,
             progressive=False),
        # two-level scene: 2000 placements of four objects
        dict(name="instanced", kind="render", scene="instanced", tris=2000, width=960, height=540, spp=16, depth=6,
             progressive=False),
        # many small independent renders (thumbnails, data generation)
        dict(name="batch", kind="batch", jobs=16, max_tris=100000, max_res=512, max_spp=32),
        # inverse rendering: one step's image, loss and gradients
        dict(name="diff_step", kind="diff", width=256, spp=64, adjoint_spp=16, depth=6, texture=512),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(("trace", "trace", "trace", "accel", "render", "render", "render", "batch", "diff"))
    if kind == "trace":
        return dict(kind=kind, op=rng.choice(("closest", "compact", "occluded")),
                    rays=rng.choice(("camera", "bounce", "shadow")), n=_log(rng, 1000, 1 << 20),
                    tris=_log(rng, 2000, 500000))
    if kind == "accel":
        return dict(kind=kind, op=rng.choice(("closest", "compact", "occluded")), rays="camera",
                    n=_log(rng, 1000, 1 << 18), tris=_log(rng, 2000, 500000))
    if kind == "batch":
        return dict(kind=kind, jobs=rng.randint(3, 16), max_tris=_log(rng, 4000, 100000), max_res=_log(rng, 150, 512),
                    max_spp=rng.randint(5, 32))
    if kind == "diff":
        return dict(kind=kind, width=_log(rng, 40, 256), spp=_log(rng, 4, 64), adjoint_spp=_log(rng, 2, 16),
                    depth=rng.randint(3, 6), texture=rng.choice((64, 128, 256, 512)))
    scene = rng.choice(("box_room", "procedural", "volume", "instanced"))
    c = dict(kind=kind, scene=scene, width=_log(rng, 100, 1024), height=_log(rng, 100, 1024))
    c["progressive"] = rng.random() < 0.3
    c["spp"] = 1 if c["progressive"] else _log(rng, 2, {"volume": 20, "instanced": 16}.get(scene, 64))
    c["depth"] = rng.randint(3, 12 if scene == "volume" else 8)
    c["tris"] = {"box_room": 36, "instanced": _log(rng, 50, 2000)}.get(scene) or _log(rng, 5000, 500000)
    return c


# ------------------------------------------------------------------- inputs


def _procedural(seed, tris, env=True):
    """The procedural scene of about `tris` triangles: displaced spheres and
    tori on a ground plane, Disney materials, sun and sky, 4 emitters."""
    env_res = (1024, 512) if env else (16, 8)
    if tris >= 500000:
        return workloads.procedural_500k(seed=seed, env_res=env_res)
    objects = 200 if tris >= 150000 else 24
    per = tris / objects
    subdiv = int(np.clip(round(math.log(max(per, 20) / 20.0) / math.log(4.0)), 0, 5))
    nu = int(np.clip(math.sqrt(per), 3, 80))
    return workloads.procedural_500k(seed=seed, n_objects=objects, n_spheres=objects // 3, sphere_subdiv=subdiv,
                                     torus_res=(nu, int(np.clip(per / (2 * nu), 3, 80))), env_res=env_res)


def _camera_rays(rng, cam, n):
    w = max(1, int(round(math.sqrt(n * 16 / 9)))) if n != 1024 * 1024 else 1024
    i = np.arange(n)
    x, y, h = i % w, i // w, -(-n // w)
    fwd, up = np.array(cam.direction[:], np.float64), np.array(cam.up[:], np.float64)
    right = np.cross(fwd, up)
    right /= np.linalg.norm(right)
    up = np.cross(right, fwd)
    th = math.tan(0.5 * cam.fovy)
    sx = (2 * (x + rng.random(n)) / w - 1) * th * (w / h)
    sy = (2 * (y + rng.random(n)) / h - 1) * th
    d = fwd + sx[:, None] * right + sy[:, None] * up
    d /= np.linalg.norm(d, axis=1, keepdims=True)
    pos = np.array(cam.position[:], np.float64) + rng.uniform(-0.5, 0.5, 3)
    return np.broadcast_to(pos, d.shape), d, np.full(n, T_FAR)


def _surface_rays(rng, sc, n, shadow):
    """Rays from points on the objects' triangles, in mesh order: cosine
    directions about the normal, or toward points of the emitters."""
    tri = np.sort(rng.integers(2, sc.triangle_count - 4, n))  # neither the ground nor the emitters
    v = sc.positions[sc.indices[tri]].astype(np.float64)
    e1, e2 = v[:, 1] - v[:, 0], v[:, 2] - v[:, 0]
    ng = np.cross(e1, e2)
    ng /= np.maximum(np.linalg.norm(ng, axis=1, keepdims=True), 1e-20)
    a, b = np.sqrt(rng.random(n))[:, None], rng.random(n)[:, None]
    p = v[:, 0] + a * (1 - b) * e1 + a * b * e2
    if shadow:
        light = sc.positions[sc.indices[sc.triangle_count - 4 + rng.integers(0, 4, n)]].astype(np.float64)
        w = rng.dirichlet((1.0, 1.0, 1.0), n)
        d = (light * w[:, :, None]).sum(1) - p
        dist = np.linalg.norm(d, axis=1)
        side = np.where((d * ng).sum(1) < 0, -1.0, 1.0)[:, None]
        return p + 1e-3 * side * ng, d / dist[:, None], dist * (1 - 1e-3)
    r, phi = np.sqrt(rng.random(n)), 2 * np.pi * rng.random(n)
    t1 = np.cross(ng, np.where(np.abs(ng[:, :1]) > 0.9, [[0.0, 1.0, 0.0]], [[1.0, 0.0, 0.0]]))
    t1 /= np.maximum(np.linalg.norm(t1, axis=1, keepdims=True), 1e-20)
    t2 = np.cross(ng, t1)
    d = (r * np.cos(phi))[:, None] * t1 + (r * np.sin(phi))[:, None] * t2 + np.sqrt(1 - r * r)[:, None] * ng
    return p + 1e-3 * ng, d / np.linalg.norm(d, axis=1, keepdims=True), np.full(n, T_FAR)


def _trace_inputs(case, seed):
    """The scene and the rays of a trace or accel case, on the host."""
    sc, cam, _ = _procedural(seed, case["tris"], env=False)
    rng = np.random.default_rng(seed + 1)
    if case["rays"] == "camera":
        rays = _camera_rays(rng, cam, case["n"])
    else:
        rays = _surface_rays(rng, sc, case["n"], case["rays"] == "shadow")
    o, d, far = (np.ascontiguousarray(a, np.float32) for a in rays)
    return sc, (o, d, np.zeros(case["n"], np.float32), far)


def _render_inputs(case, seed):
    scene = case["scene"]
    if scene == "box_room":
        sc, cam, st = workloads.box_room()
        rng = np.random.default_rng(seed)
        for m in sc.materials[:3]:
            m.base_color[:] = np.clip(np.array(m.base_color[:]) + rng.uniform(-0.05, 0.05, 3), 0, 1).tolist()
        cam.position[:] = (np.array(cam.position[:]) + rng.uniform(-0.1, 0.1, 3)).tolist()
    elif scene == "procedural":
        sc, cam, st = _procedural(seed, case["tris"])
    elif scene == "volume":
        sc, cam, st = workloads.instanced_2m(seed=seed, tex_res=512, grid=128,
                                             n_instances=max(8, case["tris"] // 5150))
    else:
        sc, cam, st = workloads.instanced_objects(seed=seed, n_instances=case["tris"])
    st.width, st.height, st.pixel_samples, st.max_depth = case["width"], case["height"], case["spp"], case["depth"]
    cam.aspect = 0.0
    return sc, cam, st


def _params(ds):
    return [p.requires_grad_(True) for p in ds.params()]


def prepare(case, seed):
    kind = case["kind"]
    s = {"case": case}
    if kind in ("trace", "accel"):
        sc, rays = _trace_inputs(case, seed)
        s["mesh"] = (sc.positions, sc.indices, sc.normals, sc.material_ids)
        s["rays"] = [torch.from_numpy(a).cuda() for a in rays]
        if kind == "trace":
            s["accel"] = Accel(*s["mesh"])
    elif kind == "render":
        sc, s["cam"], s["settings"] = _render_inputs(case, seed)
        s["renderer"] = Renderer()
        s["renderer"].set_scene(sc)
    elif kind == "batch":
        s["jobs"] = []
        rng = np.random.default_rng(seed)
        for sc, cam, st in _batch_inputs(case, rng):
            r = Renderer()
            r.set_scene(sc)
            s["jobs"].append((r, cam, st, True))
    else:
        w = case["width"]
        sc, cam, st = workloads.differentiable(seed=seed, res=w, spp=case["spp"], depth=case["depth"],
                                               texture=case["texture"])
        s["diff"] = diff.DiffScene(sc, cam, st, adjoint_spp=case["adjoint_spp"])
        s["params"] = _params(s["diff"])
        x = np.linspace(0.0, 1.0, w, dtype=np.float32)  # the target: a smooth picture
        g = np.random.default_rng(seed + 5).uniform(0.2, 0.8, (3, 3)).astype(np.float32)
        s["target"] = torch.from_numpy(g[0] + g[1] * x[:, None, None] * 0.3 + g[2] * x[None, :, None] * 0.3)
    return s


def _batch_inputs(case, rng):
    for k in range(case["jobs"]):
        # sizes spread over their ranges, the same for every seed
        a, b, c, d = ((k + 0.5) * g % 1.0 for g in (0.6180340, 0.4142136, 0.7320508, 0.2360680))
        tris = 1500.0 * (case["max_tris"] / 1500.0) ** a
        sc, cam, st = _procedural(int(rng.integers(1 << 30)), tris, env=False)
        st.width = st.height = int(100.0 * (case["max_res"] / 100.0) ** b)
        st.pixel_samples = 4 + int(c * (case["max_spp"] - 3))
        st.max_depth = 4 + int(d * 9)
        yield sc, cam, st


# ---------------------------------------------------------------------- run


def _trace(accel, op, rays):
    if op == "occluded":
        return accel.trace_occluded(*rays)
    if op == "compact":
        hit = accel.trace_closest_compact(*rays)  # t, primitive id bits, u, v
        return {"t": hit[:, 0], "prim": hit[:, 1].view(torch.int32), "uv": hit[:, 2:]}
    rec = accel.trace_closest(*rays)  # HitResult records: 17 floats, 4 ids, the hit bytes
    return {"values": rec.view(torch.float32)[:, :17], "ids": rec.view(torch.int32)[:, 17:]}


def run(s):
    case = s["case"]
    kind = case["kind"]
    if kind == "trace":
        return _trace(s["accel"], case["op"], s["rays"])
    if kind == "accel":
        accel = Accel(*s["mesh"])
        out = _trace(accel, case["op"], s["rays"])
        accel.close()
        return out
    if kind == "render":
        r = s["renderer"]
        r.render(s["cam"], s["settings"], reset=not case["progressive"])
        if case["progressive"]:
            return r.read_color()
        return {c: r.read(c) for c in ("color", "depth", "normal", "albedo")}
    if kind == "batch":
        render_batch(s["jobs"])
        return [j[0].read_color() for j in s["jobs"]]
    p = s["params"]
    for x in p:
        x.grad = None
    image = diff.render(s["diff"], *p)
    loss = ((image - s["target"]) ** 2).mean()
    loss.backward()
    return {"image": image.detach(), "loss": loss.detach(), "materials": p[0].grad, "texels": p[1].grad,
            "volumes": p[2].grad}


# --------------------------------------------------------------------- work

NODE_FLOPS, TRI_FLOPS, SHADE_FLOPS = 8 * 14, 45, 400  # an eight-wide node's boxes, a triangle test, a shaded vertex


def _ray_flops(tris):
    return (1.0 + math.log(max(tris, 8), 8)) * NODE_FLOPS + 2 * TRI_FLOPS


def work(case):
    """Scene and inputs read once, outputs written once; per ray one descent of
    an eight-wide tree, per path vertex one shading."""
    kind = case["kind"]
    if kind in ("trace", "accel"):
        n, tris = case["n"], case["tris"]
        out = {"closest": 88, "compact": 16, "occluded": 4}[case["op"]]
        mesh = tris * (12 + 6 * 2)  # indices; half a vertex a triangle
        build = tris * 100.0 if kind == "accel" else 0.0
        return {"bytes": n * (32 + out) + mesh, "flops": n * _ray_flops(tris) + build}
    if kind == "batch":
        px = 100.0 * case["max_res"]  # the square of the middle size
        samples = case["jobs"] * px * (4 + case["max_spp"]) / 2
        return {"bytes": case["jobs"] * (px * 16 + 20000 * 36), "flops": samples * 2 * (_ray_flops(20000) + SHADE_FLOPS)}
    if kind == "diff":
        px, texels = case["width"] ** 2, 8 * case["texture"] ** 2
        samples = px * (case["spp"] + 2 * case["adjoint_spp"])
        return {"bytes": px * 24 + texels * 32 + 50000 * 36, "flops": samples * 2.5 * (_ray_flops(50000) + 2 * SHADE_FLOPS)}
    px = case["width"] * case["height"]
    tris = case["tris"] * (900 if case["scene"] == "instanced" else 1)
    channels = 16 if case["progressive"] else 44
    vertices = {"box_room": 3.0, "procedural": 2.0, "volume": 2.5, "instanced": 2.5}[case["scene"]]
    return {"bytes": px * channels + case["tris"] * 36,
            "flops": px * case["spp"] * vertices * (_ray_flops(tris) + SHADE_FLOPS)}


# -------------------------------------------------------------------- exact

CHUNK = 1024       # consecutive triangles that share a bounding sphere
PAIRS = 1 << 24    # ray-triangle pairs tested at once


def _closest(sc, rays):
    """Closest hits in 64 bits: distance, triangle (-1: none), barycentrics.
    Every ray against every triangle of the chunks whose sphere it meets."""
    o, d, t0, t1 = (torch.from_numpy(a).cuda().double() for a in rays)
    n = o.shape[0]
    v = torch.from_numpy(sc.positions).cuda().double()[torch.from_numpy(sc.indices.astype(np.int64)).cuda()]
    best, prim = t1.clone(), torch.full((n,), -1, dtype=torch.int64, device="cuda")
    bu, bv = torch.zeros_like(best), torch.zeros_like(best)
    for c in range(0, v.shape[0], CHUNK):
        tri = v[c:c + CHUNK]
        lo, hi = tri.reshape(-1, 3).amin(0), tri.reshape(-1, 3).amax(0)
        mid, r2 = (lo + hi) / 2, ((hi - lo) / 2).square().sum() * 1.001
        m = mid - o
        along = (m * d).sum(1)
        meets = ((m.square().sum(1) - along.square()) <= r2) & ((along > 0) | (m.square().sum(1) <= r2))
        which = meets.nonzero()[:, 0]
        e1, e2, v0 = tri[:, 1] - tri[:, 0], tri[:, 2] - tri[:, 0], tri[:, 0]
        step = max(1, PAIRS // tri.shape[0])
        for k in range(0, which.shape[0], step):
            i = which[k:k + step]
            oi, di = o[i][:, None], d[i][:, None]
            p = torch.linalg.cross(di, e2[None], dim=2)
            det = (e1[None] * p).sum(2)
            tv = oi - v0[None]
            u = (tv * p).sum(2) / det
            q = torch.linalg.cross(tv, e1[None].expand_as(tv), dim=2)
            w = (di * q).sum(2) / det
            t = (e2[None] * q).sum(2) / det
            ok = (u >= 0) & (w >= 0) & (u + w <= 1) & (t >= t0[i][:, None])
            t, at = torch.where(ok, t, torch.inf).min(1)
            g = (t < best[i]).nonzero()[:, 0]
            j, a = i[g], at[g]
            best[j], prim[j], bu[j], bv[j] = t[g], a + c, u[g, a], w[g, a]
    return o, d, best, prim, bu, bv, v


def exact(case, seed):
    """Trace and accel cases; a path-traced image has no closed form, and an
    occlusion answer is a whole number."""
    if case["kind"] not in ("trace", "accel") or case["op"] == "occluded":
        return None
    if case["n"] * float(case["tris"]) > 6e11:
        return None
    sc, rays = _trace_inputs(case, seed)
    o, d, t, prim, u, w, v = _closest(sc, rays)
    if case["op"] == "compact":
        return {"t": t, "prim": None, "uv": torch.stack([u, w], 1)}
    hit = prim >= 0
    k = prim.clamp(min=0)
    ng = torch.linalg.cross(v[k, 1] - v[k, 0], v[k, 2] - v[k, 0], dim=1)
    ng = ng / ng.norm(dim=1, keepdim=True)
    vn = torch.from_numpy(sc.normals).cuda().double()[torch.from_numpy(sc.indices.astype(np.int64)).cuda()][k]
    sn = vn[:, 0] * (1 - u - w)[:, None] + vn[:, 1] * u[:, None] + vn[:, 2] * w[:, None]
    sn = sn / sn.norm(dim=1, keepdim=True)
    sn = torch.where((sn * ng).sum(1, keepdim=True) < 0, -sn, sn)
    out = torch.cat([t[:, None], o + d * t[:, None], ng, sn, torch.zeros_like(t)[:, None].expand(-1, 2),
                     u[:, None], w[:, None], torch.zeros_like(t)[:, None].expand(-1, 3)], 1)
    return {"values": torch.where(hit[:, None], out, 0.0), "ids": None}
