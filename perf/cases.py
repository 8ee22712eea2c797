"""Performance cases of the wavefront path tracer, through its public Python entry points.

A case is a dict of plain values.  `listed()` gives the fixed ones, `draw(rng)` one more of the
same ranges, `prepare(case, seed)` what a program has in hand before the call (scenes, plans,
buffers and inputs made from the seed), `run(state)` one pass, `work(case)` the bytes and
operations that a pass cannot do without, and `exact(case, seed)` the outputs in 64 bits where a
plain evaluation gives them.

Families:
  keys     Morton keys -> radix sort -> reorder of a wavefront of rays (all three key kinds)
  gather   reorder gather of fixed-width ray records by a sorted permutation
  bounce   traceSort of one bounce: keys, sort, reorder, closest-hit traversal
  shadow   shadow rays of a wavefront: generation, any-hit traversal, reconstruction
  shade    the shading stages of one bounce without the traversals
  frame    one frame of the renderer
  batch    one replay of batched render requests
  rebuild  acceleration structures rebuilt on the GPU for a moved mesh, then camera rays traced
"""
import math

import numpy as np
import torch

import vulkanwavefrontpathtracer_gb300 as wf

api = wf.api
DEV = "cuda"

# Scenes of the benchmark: the triangle soup in the unit cube, the courtyard, the city block and
# a smaller city of about the asked number of triangles.  kind, triangles (0: fixed), light,
# light radius, background, camera.
SKY = (0.529, 0.808, 0.98)
SCENES = {
    "soup": dict(kind=0, ntris=65536, light=(0.5, 1.6, 0.5), radius=0.1,
                 camera=dict(position=(0.5, 0.5, 2.2), rotation_deg=(0.0, 0.0, 0.0), fov_deg=45.0, znear=0.001, zfar=10.0)),
    "courtyard": dict(kind=1, ntris=0, light=(15.0, 11.0, 10.0), radius=1.0,
                      camera=dict(position=(15.0, 5.0, 19.4), rotation_deg=(-8.0, 12.0, 0.0), fov_deg=60.0, znear=0.1, zfar=512.0)),
    "city": dict(kind=2, ntris=0, light=(320.0, 300.0, 320.0), radius=4.0,
                 camera=dict(position=(320.0, 90.0, 700.0), rotation_deg=(-25.0, 0.0, 0.0), fov_deg=60.0, znear=0.1, zfar=2048.0)),
    "town": dict(kind=3, ntris=1000000, light=(185.0, 300.0, 185.0), radius=4.0,
                 camera=dict(position=(185.0, 60.0, 420.0), rotation_deg=(-12.0, 0.0, 0.0), fov_deg=60.0, znear=0.1, zfar=2000.0)),
}
TRIANGLES = {"soup": 65536, "courtyard": 268304, "city": 3000320, "town": 1000000}
# The two forms of the benchmark: 8-wide BVH, sort + reorder at every bounce, one captured graph;
# and the renderer's defaults (binary BVH, unsorted, every stage launched directly).
FORMS = {
    "chosen": dict(bvh_kind=1, sort_path_rays=1, reorder_path_rays=1, use_graph=1),
    "plain": dict(bvh_kind=0, use_graph=0),
}
KEY_BITS = (32, 48, 63)


def listed():
    return [
        # The small configuration's wavefront: 256x256 rays, 32-bit keys; launches and latency count.
        {"name": "keys_64k", "family": "keys", "n": 65536, "kind": 0, "clusters": 0},
        # One bounce of a 1080p frame: 63-bit six-dimensional keys of clustered rays.
        {"name": "keys_1080p", "family": "keys", "n": 2073600, "kind": 2, "clusters": 256},
        # A wavefront far beyond L2, odd size: the sort and the reorder are bound by memory.
        {"name": "keys_32m", "family": "keys", "n": 33554467, "kind": 2, "clusters": 4096},
        # 48-byte ray + payload records gathered by a sorted permutation of randomly ordered rays.
        {"name": "gather_16m", "family": "gather", "n": 16777216, "bytes": 48, "maps": True},
        # The incoherent bounce of the benchmark frame, sorted and traced with the 8-wide BVH.
        {"name": "bounce_1080p", "family": "bounce", "scene": "courtyard", "w": 1920, "h": 1080, "bvh": 1, "kind": 2, "reorder": True},
        # Shadow rays (any hit) in the 3M-triangle city, whose BVH exceeds L2.
        {"name": "shadow_city", "family": "shadow", "scene": "city", "w": 1920, "h": 1080, "bvh": 1, "samples": 2},
        # The shading stages of one bounce at a ragged resolution.
        {"name": "shade_ragged", "family": "shade", "scene": "courtyard", "w": 1013, "h": 767, "samples": 2},
        # The smallest frame in use: the soup at 256x256, 4 bounces, 32-bit keys.
        {"name": "frame_256", "family": "frame", "scene": "soup", "w": 256, "h": 256, "spp": 1, "depth": 4, "samples": 2, "form": "chosen", "kind": 0},
        # The benchmark frame: the courtyard at 1080p, 8 bounces.
        {"name": "frame_1080p", "family": "frame", "scene": "courtyard", "w": 1920, "h": 1080, "spp": 1, "depth": 8, "samples": 2, "form": "chosen", "kind": 2},
        # The city at 4K with the renderer's default form (binary BVH, no sorting, direct launches).
        {"name": "frame_4k_plain", "family": "frame", "scene": "city", "w": 3840, "h": 2160, "spp": 1, "depth": 8, "samples": 2, "form": "plain", "kind": 0},
        # Serving: twelve requests of mixed scenes, resolutions, samples and depths in one graph.
        {"name": "batch_12", "family": "batch", "requests": 12, "mix": 7},
        # A moved 3M-triangle mesh: both BVHs rebuilt on the GPU, then 960x540 camera rays.
        {"name": "rebuild_city", "family": "rebuild", "scene": "city", "ntris": 0, "w": 960, "h": 540, "bvh": 1},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    family = rng.choice(["keys", "gather", "bounce", "shadow", "shade", "frame", "batch", "rebuild"])
    small = rng.choice(["soup", "courtyard"])
    if family == "keys":
        return {"family": family, "n": _log(rng, 4000, 33554432), "kind": rng.choice([0, 1, 2]), "clusters": rng.choice([0, 64, 1024])}
    if family == "gather":
        return {"family": family, "n": _log(rng, 50000, 16777216), "bytes": rng.choice([16, 32, 48, 64]), "maps": rng.choice([True, True, False])}
    w = _log(rng, 120, 1920)
    h = max(90, int(w * rng.uniform(0.5, 0.57)))
    if family == "bounce":
        return {"family": family, "scene": small, "w": w, "h": h, "bvh": rng.choice([0, 1]), "kind": rng.choice([0, 1, 2]), "reorder": rng.choice([True, True, False])}
    if family == "shadow":
        return {"family": family, "scene": rng.choice(["courtyard", "city"]), "w": w, "h": h, "bvh": rng.choice([0, 1]), "samples": rng.choice([1, 2, 3])}
    if family == "shade":
        return {"family": family, "scene": small, "w": w, "h": h, "samples": rng.choice([1, 2, 3])}
    if family == "frame":
        return {"family": family, "scene": small, "w": w, "h": h, "spp": 1 if w > 700 else rng.choice([1, 2, 4]), "depth": rng.randint(1, 8),
                "samples": rng.choice([1, 2]), "form": rng.choice(["chosen", "plain"]), "kind": rng.choice([0, 2])}
    if family == "batch":
        return {"family": family, "requests": rng.randint(2, 12), "mix": rng.randint(1, 1000)}
    return {"family": family, "scene": "soup", "ntris": _log(rng, 4000, 1000000), "w": 960, "h": 540, "bvh": rng.choice([0, 1])}


# ------------------------------------------------------------------ inputs
_meshes, _scenes = {}, {}


def _mesh(name, ntris=0):
    """Positions, normals, indices (host arrays) of a named scene."""
    key = (name, ntris)
    if key not in _meshes:
        _meshes[key] = api.generate_scene(SCENES[name]["kind"], 1, ntris or SCENES[name]["ntris"])
    return _meshes[key]


def _scene(name):
    """The scene and its shading geometry, which a program keeps from call to call."""
    if name not in _scenes:
        pos, nrm, idx = _mesh(name)
        _scenes[name] = (api.Scene(pos, idx), api.Geometry(pos, nrm, idx, device=DEV))
    return _scenes[name]


def _camera(name, seed):
    """The scene's camera, moved a little by the seed."""
    c = dict(SCENES[name]["camera"])
    rng = np.random.default_rng(seed)
    step = 0.01 * abs(c["position"][2])
    c["position"] = tuple(float(p + step * d) for p, d in zip(c["position"], rng.uniform(-1, 1, 3)))
    c["rotation_deg"] = tuple(float(r + d) for r, d in zip(c["rotation_deg"], rng.uniform(-2, 2, 3)))
    return c


_tables = {}


def _pixel_table(w, h):
    if (w, h) not in _tables:
        _tables.clear()
        _tables[(w, h)] = torch.from_numpy(api.pixel_table(w, h)[0]).to(DEV)
    return _tables[(w, h)]


def _i32(*shape):
    return torch.zeros(shape, dtype=torch.int32, device=DEV)


def _f32(*shape):
    return torch.zeros(shape, dtype=torch.float32, device=DEV)


def _primary(name, w, h, seed):
    """Camera rays of a frame."""
    cam = _camera(name, seed)
    s2w = api.camera_screen_to_world(cam["position"], cam["rotation_deg"], cam["fov_deg"], w / h, cam["znear"], cam["zfar"])
    rays = _f32(w * h, 8)
    i2p = _pixel_table(w, h).clone()
    api.raygen_primary(s2w, i2p, rays, list(cam["position"]), seed % 1000, w, h, cam["zfar"])
    return rays, i2p


def _wavefront(name, w, h, seed, bounce):
    """Rays, hits and pixel map of the primary pass, or of the first bounce (compacted)."""
    scene, geom = _scene(name)
    rays, i2p = _primary(name, w, h, seed)
    hits = _i32(w * h, 4)
    api.trace(scene, wf.BVH8_Q8, rays, hits)
    if not bounce:
        return rays, hits, i2p
    seeds, dec, count = _i32(w * h), torch.ones((w * h, 4), device=DEV), _i32(1)
    path, p_i2p = torch.empty_like(rays), torch.empty_like(i2p)
    api.init_seeds(seeds, 1 + seed % 1000)
    api.raygen_path(seeds, geom.table, rays, path, i2p, p_i2p, hits, dec, count)
    m = max(1, int(count.item()))
    path, p_i2p, hits = path[:m].clone(), p_i2p[:m].clone(), _i32(m, 4)
    api.trace(scene, wf.BVH8_Q8, path, hits)
    return path, hits, p_i2p


def _hits(h):
    return {"ids": h[:, :2], "t": h.view(torch.float32)[:, 2], "bary": h[:, 3]}


def _random_rays(n, clusters, seed):
    """Rays in the unit box: uniform, or around `clusters` points and directions (six-dimensional Gaussians)."""
    g = torch.Generator(device=DEV).manual_seed(seed)
    rays = torch.empty((n, 8), device=DEV)
    if clusters:
        c = torch.randint(clusters, (n,), generator=g, device=DEV)
        at = torch.rand((clusters, 3), generator=g, device=DEV)
        to = torch.randn((clusters, 3), generator=g, device=DEV)
        rays[:, :3] = at[c] + 0.02 * torch.randn((n, 3), generator=g, device=DEV)
        d = torch.nn.functional.normalize(to, dim=1)[c] + 0.2 * torch.randn((n, 3), generator=g, device=DEV)
    else:
        rays[:, :3] = torch.rand((n, 3), generator=g, device=DEV)
        d = torch.randn((n, 3), generator=g, device=DEV)
    rays[:, 4:7] = torch.nn.functional.normalize(d, dim=1)
    rays[:, 3], rays[:, 7] = 1e-4, 3.4e38
    return rays


def _config(case, q, radius):
    return dict(FORMS[case["form"]], ray_type=2, num_primary_samples=q["spp"], num_shadow_samples=q["samples"], shadow_radius=radius,
                recursion_depth=q["depth"], key_value=0.6, white_point=2.0, albedo=0.8, morton_kind=case["kind"])


def _requests(case):
    """The mixed requests of a batch (scenes, resolutions, samples, depths drawn by case["mix"])."""
    rng = np.random.default_rng(case["mix"])
    return [dict(scene=str(rng.choice(["soup", "courtyard", "town"])), w=int(r), h=int(r), spp=int(rng.integers(1, 5)), depth=int(rng.integers(1, 9)), samples=2)
            for r in rng.choice([128, 256, 512], case["requests"])]


def prepare(case, seed):
    f = case["family"]
    st = {"case": case}
    if f == "keys":
        n, bits = case["n"], KEY_BITS[case["kind"]]
        st.update(rays=_random_rays(n, case["clusters"], seed), keys=torch.empty(n, dtype=torch.int32 if bits == 32 else torch.int64, device=DEV),
                  ids=_i32(n), out=_f32(n, 8), s2i=torch.arange(n, dtype=torch.int32, device=DEV), os2i=_i32(n), oi2s=_i32(n), bits=bits,
                  scratch=torch.empty(api.sort_scratch_bytes(n, bits), dtype=torch.uint8, device=DEV))
    elif f == "gather":
        n, words = case["n"], case["bytes"] // 4
        g = torch.Generator(device=DEV).manual_seed(seed)
        st.update(records=torch.randn((n, words), generator=g, device=DEV), ids=torch.randperm(n, generator=g, device=DEV).to(torch.int32),
                  out=_f32(n, words), s2i=torch.randperm(n, generator=g, device=DEV).to(torch.int32) if case["maps"] else None,
                  os2i=_i32(n) if case["maps"] else None, oi2s=_i32(n) if case["maps"] else None)
    elif f == "bounce":
        rays, _, i2p = _wavefront(case["scene"], case["w"], case["h"], seed, True)
        n = case["w"] * case["h"]  # buffers hold a whole wavefront; the compacted one fills their front
        st.update(scene=_scene(case["scene"])[0], n=rays.shape[0], rays=rays, i2p=i2p, hits=_i32(n, 4), out=_f32(n, 8), os2i=_i32(n), oi2s=_i32(n), ids=_i32(n),
                  keys=torch.zeros(n, dtype=torch.int32 if case["kind"] == 0 else torch.int64, device=DEV),
                  scratch=torch.empty(api.sort_scratch_bytes(n, 64), dtype=torch.uint8, device=DEV))
    elif f == "shadow":
        rays, hits, i2p = _wavefront(case["scene"], case["w"], case["h"], seed, True)
        n, S, px = rays.shape[0], case["samples"], case["w"] * case["h"]
        seeds = _i32(n)
        api.init_seeds(seeds, 2 + seed % 1000)
        g = torch.Generator(device=DEV).manual_seed(seed)
        st.update(scene=_scene(case["scene"])[0], rays=rays, hits=hits, i2p=i2p, seeds=seeds, srays=_f32(px * S, 8), shits=_i32(px * S, 4), s2i=_i32(px * S),
                  i2s=_i32(px * S), color=torch.rand((px, 4), generator=g, device=DEV), frame=_f32(px, 4))
    elif f == "shade":
        scene, geom = _scene(case["scene"])
        rays, hits, i2p = _wavefront(case["scene"], case["w"], case["h"], seed, False)
        n, S, sc = rays.shape[0], case["samples"], SCENES[case["scene"]]
        st.update(geom=geom, rays=rays, hits=hits, i2p=i2p, frame_index=2 + seed % 1000, seeds=_i32(n), dec=_f32(n, 4), color=_f32(n, 4), frame=_f32(n, 4),
                  mean=torch.rand((n, 4), generator=torch.Generator(device=DEV).manual_seed(seed), device=DEV), hit_count=_i32(1), path_count=_i32(1),
                  srays=_f32(n * S, 8), shits=_i32(n * S, 4), s2i=_i32(n * S), i2s=_i32(n * S), path=_f32(n, 8), path_i2p=_i32(n),
                  scratch=torch.empty(api.raygen_path_scratch_bytes(n), dtype=torch.uint8, device=DEV))
        api.init_seeds(st["seeds"], st["frame_index"])
        api.raygen_shadow(st["seeds"], rays, hits, st["srays"], st["s2i"], st["i2s"], sc["light"], sc["radius"], 0, n, S)
        api.trace(scene, wf.BVH8_Q8, st["srays"], st["shits"], closest_hit=False)
    elif f == "frame":
        scene, geom = _scene(case["scene"])
        sc = SCENES[case["scene"]]
        r = api.Renderer(**_config(case, case, sc["radius"]))
        r.set_scene(scene, geom, sc["light"], SKY)
        n = case["w"] * case["h"]
        st.update(renderer=r, camera=api.make_camera(**_camera(case["scene"], seed)), pixels=_f32(n, 4), frame=_f32(n, 4))
    elif f == "batch":
        reqs = []
        for i, q in enumerate(_requests(case)):
            sc, n = SCENES[q["scene"]], q["w"] * q["h"]
            scene, geom = _scene(q["scene"])
            reqs.append(dict(scene=scene, geometry=geom, light=sc["light"], background=SKY, camera=api.make_camera(**_camera(q["scene"], seed + i)),
                             width=q["w"], height=q["h"], config=api.default_config(**_config(dict(form="chosen", kind=2), q, sc["radius"])),
                             pixels=_f32(n, 4), frame_pixels=_f32(n, 4)))
        st.update(requests=reqs, batch=api.Batch(reqs, streams=4))
    else:
        pos, _, idx = _mesh(case["scene"], case["ntris"])
        p = torch.from_numpy(pos).to(DEV)
        size = (p.max(0).values - p.min(0).values).max()
        rng = np.random.default_rng(seed)
        k, phase = rng.uniform(2.0, 4.0), rng.uniform(0.0, 6.28)
        p = p + 0.01 * size * torch.sin(k * p.roll(1, dims=1) / size + phase)
        rays, _ = _primary(case["scene"], case["w"], case["h"], seed)
        st.update(pos=p.contiguous(), idx=torch.from_numpy(idx.view(np.int32)).to(DEV), rays=rays, hits=_i32(rays.shape[0], 4))
    return st


# -------------------------------------------------------------------- pass
def run(st):
    case = st["case"]
    f = case["family"]
    if f == "keys":
        api.morton(st["rays"], (0.0, 0.0, 0.0), (1.0, 1.0, 1.0), case["kind"], st["keys"], st["ids"])
        api.sort_pairs(st["keys"], st["ids"], st["bits"], scratch=st["scratch"])
        api.reorder(st["ids"], st["rays"], st["out"], st["s2i"], st["os2i"], st["oi2s"])
        return {"keys": st["keys"], "ids": st["ids"], "rays": st["out"], "s2i": st["os2i"], "i2s": st["oi2s"]}
    if f == "gather":
        api.reorder_records(st["ids"], st["records"], st["out"], st["s2i"], st["os2i"], st["oi2s"])
        return {"records": st["out"], "s2i": st["os2i"], "i2s": st["oi2s"]}
    if f == "bounce":
        s = st["scene"]
        api.trace_sort(s, case["bvh"], st["rays"], st["hits"], s.bounds_min, s.bounds_max, case["kind"], case["reorder"], st["keys"], st["ids"],
                       rays_out=st["out"], slot_to_index=st["i2p"], slot_to_index_out=st["os2i"], index_to_slot_out=st["oi2s"], scratch=st["scratch"], n=st["n"])
        out = {"keys": st["keys"], "ids": st["ids"], "hits": _hits(st["hits"])}
        return dict(out, rays=st["out"], s2i=st["os2i"]) if case["reorder"] else out
    if f == "shadow":
        sc, n, S = SCENES[case["scene"]], st["rays"].shape[0], case["samples"]
        api.raygen_shadow(st["seeds"], st["rays"], st["hits"], st["srays"], st["s2i"], st["i2s"], sc["light"], sc["radius"], 0, n, S)
        api.trace(st["scene"], case["bvh"], st["srays"], st["shits"], closest_hit=False, n=n * S)
        api.reconstruct_shadow(st["shits"], st["i2p"], st["i2s"], st["color"], st["frame"], 0, n, S, replace=True)
        return {"rays": st["srays"], "pixels": st["frame"]}
    if f == "shade":
        sc, n, S = SCENES[case["scene"]], st["rays"].shape[0], case["samples"]
        api.init_seeds(st["seeds"], st["frame_index"])
        api.fill_u32(st["dec"], 0x3F800000, 4 * n)
        api.fill_u32(st["color"], 0, 4 * n)
        api.fill_u32(st["frame"], 0, 4 * n)
        api.fill_u32(st["hit_count"], 0, 1)
        api.reconstruct_smooth(st["rays"], st["hits"], st["i2p"], st["color"], st["dec"], st["geom"].table, sc["light"], SKY, 1)
        api.count_hits(st["hits"], st["hit_count"])
        api.raygen_shadow(st["seeds"], st["rays"], st["hits"], st["srays"], st["s2i"], st["i2s"], sc["light"], sc["radius"], 0, n, S)
        api.reconstruct_shadow(st["shits"], st["i2p"], st["i2s"], st["color"], st["frame"], 0, n, S)
        api.raygen_path(st["seeds"], st["geom"].table, st["rays"], st["path"], st["i2p"], st["path_i2p"], st["hits"], st["dec"], st["path_count"],
                        albedo=0.8, scratch=st["scratch"])
        api.interpolate_colors(st["frame"], st["mean"], st["frame_index"], 0.6, 2.0)
        return {k: st[k] for k in ("color", "dec", "frame", "hit_count", "mean", "path", "path_count", "path_i2p", "seeds", "srays")}
    if f == "frame":
        st["renderer"].render(st["camera"], case["w"], case["h"], st["pixels"], st["frame"])
        return {"pixels": st["pixels"], "frame": st["frame"]}
    if f == "batch":
        st["batch"].render()
        return [{"pixels": q["pixels"], "frame": q["frame_pixels"]} for q in st["requests"]]
    scene = api.Scene.from_device(st["pos"], st["idx"])
    api.trace(scene, case["bvh"], st["rays"], st["hits"])
    scene.close()
    return _hits(st["hits"])


# -------------------------------------------------------------------- work
def _frame_work(q):
    """Bytes of a frame: every path and shadow ray written, read and answered once (48 bytes a ray, every
    path taken to hit), the pixel state once per pass, the image once; about 30 node and triangle tests a ray."""
    px = q["w"] * q["h"]
    rays = px * q["spp"] * (1 + q["depth"]) * (1 + q["samples"])
    return {"bytes": rays * 80.0 + px * q["spp"] * (1 + q["depth"]) * 32.0 + px * 48.0, "flops": rays * 30 * 40.0}


def work(case):
    f = case["family"]
    if f == "keys":
        # rays read, reordered rays, keys, order and both maps written; the map read
        kb = 4 if case["kind"] == 0 else 8
        return {"bytes": case["n"] * (32.0 + 32 + kb + 4 + 4 + 4 + 4), "flops": 0}
    if f == "gather":
        return {"bytes": case["n"] * (2.0 * case["bytes"] + 4 + (12 if case["maps"] else 0)), "flops": 0}
    if f == "rebuild":
        n = case["ntris"] or TRIANGLES[case["scene"]]
        # vertices and indices read; both node arrays (about 64 and 20 bytes a triangle) and both triangle tables written
        return {"bytes": n * (12.0 + 18 + 64 + 20 + 96) + case["w"] * case["h"] * 48.0, "flops": case["w"] * case["h"] * 30 * 40.0}
    if f == "batch":
        ws = [_frame_work(q) for q in _requests(case)]
        return {k: sum(w[k] for w in ws) for k in ("bytes", "flops")}
    if f == "frame":
        return _frame_work(case)
    px = float(case["w"] * case["h"])
    if f == "bounce":
        # ray and map read; keys, order, reordered rays, maps and hits written
        return {"bytes": px * (36 + (4 if case["kind"] == 0 else 8) + 4 + 16 + (40 if case["reorder"] else 0)), "flops": px * 30 * 40}
    if f == "shadow":
        # ray, hit, seed, map and colour read, image written; the shadow rays and their two maps written
        return {"bytes": px * (32 + 16 + 4 + 4 + 16 + 16 + case["samples"] * 40.0), "flops": px * case["samples"] * 20 * 40}
    # shade: ray, hit, map, mean and three vertices read; colour, throughput, image, mean, seed, path ray, its map, shadow rays and maps written
    return {"bytes": px * (32 + 16 + 4 + 16 + 96 + 16 * 4 + 4 + 32 + 4 + case["samples"] * (40.0 + 16)), "flops": 0}


# ------------------------------------------------------------ 64-bit values
M32 = 0xFFFFFFFF


def _f(x):
    """A single-precision constant as a double."""
    return float(np.float32(x))


def _normalize(v):
    return v / v.norm(dim=1, keepdim=True)


def _tea(i, frame):
    """TEA, 16 rounds, of the index and the frame number (32-bit words in 64-bit integers)."""
    v0, v1, s = i.clone(), torch.full_like(i, frame), 0
    for _ in range(16):
        s = (s + 0x9E3779B9) & M32
        v0 = (v0 + ((((v1 << 4) + 0xA341316C) & M32) ^ ((v1 + s) & M32) ^ (((v1 >> 5) + 0xC8013EA4) & M32))) & M32
        v1 = (v1 + ((((v0 << 4) + 0xAD90777D) & M32) ^ ((v0 + s) & M32) ^ (((v0 >> 5) + 0x7E95761E) & M32))) & M32
    return v0


def _mix(a, b, c):
    """Jenkins' mix of three 32-bit words."""
    for x, y, z in ((13, 8, 13), (12, 16, 5), (3, 10, 15)):
        a = ((a - b - c) & M32) ^ (c >> x)
        b = ((b - c - a) & M32) ^ ((a << y) & M32)
        c = ((c - a - b) & M32) ^ (b >> z)
    return a, b, c


def _sobol(i):
    r1 = r2 = 0
    v1, v2 = 1 << 31, 3 << 30
    while i:
        if i & 1:
            r1 ^= v1
            r2 ^= (v2 << 1) & M32
        v1 |= v1 >> 1
        v2 ^= v2 >> 1
        i >>= 1
    return r1 / 2.0**32, r2 / 2.0**32


def _tonemap(c, key, white):
    rgb = [[_f(x) for x in r] for r in ((0.5141364, 0.265068, 0.0241188), (0.3238786, 0.67023428, 0.1228178), (0.16036376, 0.06409157, 0.84442666))]
    xyz = [[_f(x) for x in r] for r in ((2.5651, -1.0217, 0.0753), (-1.1665, 1.9777, -0.2543), (-0.3986, 0.0439, 1.1892))]
    c = c @ torch.tensor(rgb, dtype=torch.float64, device=c.device).T
    s = c.sum(1)
    x, y = c[:, 0] / s, c[:, 1] / s
    lp = c[:, 1] * _f(key) / 0.5
    ld = lp * (1 + lp / (_f(white) * _f(white))) / (1 + lp)
    return torch.stack([ld * x / y, ld, ld * (1 - x - y) / y], 1) @ torch.tensor(xyz, dtype=torch.float64, device=c.device).T


def _exact_shade(case, seed):
    st = prepare(case, seed)
    sc, S = SCENES[case["scene"]], case["samples"]
    rays, hits, i2p, n = st["rays"].double(), st["hits"], st["i2p"].long(), st["rays"].shape[0]
    o, d = rays[:, :3], rays[:, 4:7]
    hit = hits[:, 0] >= 0
    t = st["hits"].view(torch.float32)[:, 2].double().unsqueeze(1)
    vec = lambda v: torch.tensor([_f(x) for x in v], dtype=torch.float64, device=DEV)  # noqa: E731
    ones = lambda v: torch.cat([v, torch.ones_like(v[:, :1])], 1)  # noqa: E731
    light, sky = vec(sc["light"]), vec(SKY)
    # interpolated normals, turned against the ray
    tri = st["geom"].indices.view(-1, 3)[hits[:, 0].clamp(min=0).long()].long()
    u, v = (hits[:, 3] & 0xFFFF).double() / 65535.0, ((hits[:, 3].long() & M32) >> 16).double() / 65535.0
    vn = st["geom"].vertices[:, 3:6].double()
    nrm = _normalize(vn[tri[:, 0]] * (1 - u - v).unsqueeze(1) + vn[tri[:, 1]] * u.unsqueeze(1) + vn[tri[:, 2]] * v.unsqueeze(1))
    nrm = torch.where((nrm * d).sum(1, keepdim=True) < 0, nrm, -nrm)
    # colours: diffuse light, or the sky
    at = o + d * t
    lit = (nrm * _normalize(light - at)).sum(1, keepdim=True).clamp(min=_f(0.1)).expand(n, 3)
    shade = torch.where(hit.unsqueeze(1), lit, sky.expand(n, 3))
    color = torch.zeros((n, 4), dtype=torch.float64, device=DEV)
    color[i2p] = ones(shade)
    # shadow rays
    seeds = _tea(torch.arange(n, device=DEV), st["frame_index"])
    a, b, c = (seeds + torch.arange(n, device=DEV)) & M32, torch.full_like(seeds, 0x9E3779B9), torch.full_like(seeds, 0x9E3779B9)
    for _ in range(2):
        a, b, c = _mix(a, b, c)
    off = torch.stack([a, b, c], 1).double() / 2.0**32
    org = o + d * (t - _f(1e-5)).clamp(min=0)
    org[~hit] = 0
    srays = torch.zeros((n, S, 8), dtype=torch.float64, device=DEV)
    for i in range(S):
        x, y = _sobol(i)
        p = off + torch.tensor([x, y, (i + 0.5) / S], dtype=torch.float64, device=DEV)
        p = torch.where(p >= 1, p - 1, p)
        to = light + (2 * p - 1) * _f(sc["radius"]) - org
        length = to.norm(dim=1)
        srays[:, i, :3], srays[:, i, 3] = org, _f(1e-5)
        srays[:, i, 4:7] = torch.where(hit.unsqueeze(1), to / length.unsqueeze(1), vec((1, 0, 0)).expand(n, 3))
        srays[:, i, 7] = torch.where(hit, length, torch.full_like(length, -1.0))
    # shadowed image, running mean and tone map
    seen = (st["shits"][:, 0] == -1).view(n, S).double().mean(1, keepdim=True)
    frame = torch.zeros_like(color)
    frame[i2p] = ones(shade * seen)
    fi = st["frame_index"]
    mean = frame[:, :3] / fi + st["mean"].double()[:, :3] * ((fi - 1) / fi)
    # bounce rays of the hits, in order
    r = []
    for _ in range(2):
        seeds = torch.where(hit, (seeds * 1103515245 + 12345) & M32, seeds)
        r.append((seeds & 0xFFFFFF).double() / 2.0**24)
    rad, ang = r[0].sqrt(), 2 * math.pi * r[1]
    s = torch.where(nrm[:, 2] >= 0, 1.0, -1.0).double()
    k = -1 / (s + nrm[:, 2])
    bb = nrm[:, 0] * nrm[:, 1] * k
    uu = torch.stack([1 + s * nrm[:, 0] ** 2 * k, s * bb, -s * nrm[:, 0]], 1)
    vv = torch.stack([bb, s + nrm[:, 1] ** 2 * k, -nrm[:, 1]], 1)
    nd = uu * (rad * ang.sin()).unsqueeze(1) + vv * (rad * ang.cos()).unsqueeze(1) + nrm * (1 - r[0]).sqrt().unsqueeze(1)
    full = torch.full((n, 1), _f(1e-4), dtype=torch.float64, device=DEV)
    path = torch.zeros((n, 8), dtype=torch.float64, device=DEV)
    m = int(hit.sum())
    path[:m] = torch.cat([at + nd * _f(1e-4), full, nd, torch.full_like(full, float(np.finfo(np.float32).max))], 1)[hit]
    dec = torch.ones_like(color)
    dec[i2p[hit], :3] = _f(0.8)
    return {"color": color, "dec": dec, "frame": ones(_tonemap(mean, 0.6, 2.0)), "hit_count": None, "mean": ones(mean), "path": path, "path_count": None,
            "path_i2p": None, "seeds": None, "srays": srays.view(n * S, 8)}


def exact(case, seed):
    if case["family"] == "shade":
        return _exact_shade(case, seed)
    if case["family"] == "gather":
        # a copy: whole records by the permutation
        st = prepare(case, seed)
        return {"records": st["records"].double()[st["ids"].long()], "s2i": None, "i2s": None}
    # Traced and sorted outputs follow from decisions (which triangle is nearest, which key is
    # smaller): no plain 64-bit evaluation of these wavefronts takes under 20 seconds.
    return None
