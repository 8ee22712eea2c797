"""A renderer's captured frame graph is replayed only while everything that it was captured with is
still there: frames of a renderer with a graph equal those of one that launches every stage."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

LIGHT, BG = (0.5, 1.6, 0.5), (0.5, 0.8, 1.0)


def config(wf, **over):
    return wf.api.default_config(**dict(dict(ray_type=wf.PATH_RAYS, recursion_depth=2, num_shadow_samples=2,
                                             shadow_radius=0.2, sort_path_rays=1, reorder_path_rays=1, morton_kind=2,
                                             bvh_kind=1, use_graph=1), **over))


def camera(wf):
    return wf.api.make_camera(position=(0.5, 0.5, 2.2), rotation_deg=(0, 0, 0), fov_deg=45.0, znear=0.001, zfar=10.0)


def render(wf, dev, r, w, h, px=None):
    """One first frame's bits; px: its buffers, for frames that share a graph."""
    import torch
    px = torch.zeros((2, w * h, 4), dtype=torch.float32, device=dev) if px is None else px
    r.reset_frame_index()
    r.render(camera(wf), w, h, px[0], px[1])
    out = px[1].cpu().numpy()
    out[np.isnan(out)] = np.nan
    return out.view(np.uint32)


def direct(wf, dev, scene, w, h, **over):
    r = wf.api.Renderer(config(wf, use_graph=0, **over))
    r.set_scene(*scene, LIGHT, BG)
    out = render(wf, dev, r, w, h)
    r.close()
    return out


def test_scene_rebuilt_between_frames(wf, dev):
    """The mesh moves inside unchanged bounds: same geometry table, light and bounds, and often the
    same address of the new scene."""
    import torch
    api = wf.api
    pos, nrm, idx = api.generate_scene(0, 41, 3000)
    geom = api.Geometry(pos, nrm, idx, device=dev)
    inside = np.all((pos > pos.min(0)) & (pos < pos.max(0)), 1)
    ind = torch.from_numpy(idx.view(np.int32)).to(dev)
    r = api.Renderer(config(wf))
    px = torch.zeros((2, 96 * 64, 4), dtype=torch.float32, device=dev)
    frames = []
    for step in range(6):
        moved = pos.copy()
        moved[inside] = pos.mean(0) + (1.0 - 0.1 * step) * (pos[inside] - pos.mean(0))
        sc = api.Scene.from_device(torch.from_numpy(moved).to(dev), ind)
        r.set_scene(sc, geom, LIGHT, BG)
        got = render(wf, dev, r, 96, 64, px)
        assert np.array_equal(got, direct(wf, dev, (sc, geom), 96, 64)), step
        frames.append(got)
        torch.cuda.synchronize()
        sc.close()
    assert not np.array_equal(frames[0], frames[5])
    assert api.device_status() == 0


@pytest.mark.parametrize("bigger", [dict(num_shadow_samples=5), dict(timing=1), dict(sort_shadow_rays=1)])
def test_buffers_grown_between_frames(wf, dev, bigger):
    """A frame without the graph that needs larger buffers, then the captured frame again."""
    import torch
    api = wf.api
    pos, nrm, idx = api.generate_scene(0, 42, 3000)
    scene = api.Scene(pos, idx), api.Geometry(pos, nrm, idx, device=dev)
    r = api.Renderer(config(wf))
    r.set_scene(*scene, LIGHT, BG)
    px = torch.zeros((2, 64 * 48, 4), dtype=torch.float32, device=dev)
    first = render(wf, dev, r, 64, 48, px)
    r.set_config(config(wf, use_graph=0, **bigger))
    render(wf, dev, r, 640, 480)
    r.set_config(config(wf))
    # Whatever takes the place of the released buffers must not be written.
    hold = [torch.full((1 << k,), 7, dtype=torch.int32, device=dev) for k in range(8, 22)]
    assert np.array_equal(render(wf, dev, r, 64, 48, px), first)
    assert np.array_equal(first, direct(wf, dev, scene, 64, 48))
    assert all(bool((h == 7).all()) for h in hold)
    r.close()
    assert api.device_status() == 0


def test_knobs_changed_between_frames(wf, dev):
    """A knob set after the capture reaches the next frame: counting counts the rays of a frame without
    a graph, and stops."""
    import torch
    api = wf.api
    pos, nrm, idx = api.generate_scene(0, 43, 3000)
    scene = api.Scene(pos, idx), api.Geometry(pos, nrm, idx, device=dev)
    r = api.Renderer(config(wf))
    r.set_scene(*scene, LIGHT, BG)
    px = torch.zeros((2, 80 * 60, 4), dtype=torch.float32, device=dev)

    def counted(frame):
        api.trace_counters(reset=True)
        bits = frame()
        return bits, api.trace_counters(reset=True)["rays"]

    graph, rays = counted(lambda: render(wf, dev, r, 80, 60, px))
    assert rays == 0
    api.tune_set("trace.count", 1)
    try:
        ref, ref_rays = counted(lambda: direct(wf, dev, scene, 80, 60))
        got, rays = counted(lambda: render(wf, dev, r, 80, 60, px))
    finally:
        api.tune_set("trace.count", 0)
    assert ref_rays >= 80 * 60 and rays == ref_rays
    assert np.array_equal(got, ref) and np.array_equal(got, graph)
    assert counted(lambda: render(wf, dev, r, 80, 60, px))[1] == 0
    launches = []
    for tiles in (1, 0):
        api.tune_set("sort.tiles", tiles)
        assert np.array_equal(render(wf, dev, r, 80, 60, px), graph)
        k0 = wf.api.lib().wfpt_kernel_launch_count()
        assert np.array_equal(render(wf, dev, r, 80, 60, px), graph)
        launches.append(wf.api.lib().wfpt_kernel_launch_count() - k0)
    assert launches[0] != launches[1]  # the tiny tiles' scratch is cleared by a kernel, not by a memset
    r.close()
    assert api.device_status() == 0
