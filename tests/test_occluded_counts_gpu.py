"""Traversal counting of a frame's shadow rays: the counting forms of the occlusion kernels, not of
others, around the sizes where the launch shape changes."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def scene(wf, dev):
    pos, nrm, idx = wf.api.generate_scene(0, 51, 4000)
    return wf.api.Scene(pos, idx), wf.api.Geometry(pos, nrm, idx, device=dev)


def counted(wf, dev, scene, w, h, knobs=(), **cfg):
    """(the frame's bits, its counters, the rays of its statistics)"""
    import torch
    api = wf.api
    r = api.Renderer(**dict(dict(ray_type=wf.PATH_RAYS, recursion_depth=1, num_shadow_samples=2, shadow_radius=0.2), **cfg))
    r.set_scene(*scene, (0.5, 1.6, 0.5), (0.5, 0.8, 1.0))
    px = torch.zeros((2, w * h, 4), dtype=torch.float32, device=dev)
    old = [(k, api.tune_get(k)) for k, _ in knobs]
    try:
        for k, v in knobs:
            api.tune_set(k, v)
        api.trace_counters(reset=True)
        r.render(api.make_camera(position=(0.5, 0.5, 1.4), rotation_deg=(0, 0, 0), fov_deg=30.0, znear=0.001, zfar=10.0),
                 w, h, px[0], px[1])
        st = r.stats()
        counts = api.trace_counters(reset=True)
    finally:
        for k, v in old:
            api.tune_set(k, v)
    r.close()
    out = px[1].cpu().numpy()
    out[np.isnan(out)] = np.nan
    return out.view(np.uint32), counts, st.num_primary_rays + st.num_path_rays + st.num_shadow_rays


@pytest.mark.parametrize("w,h", [(1, 1), (37, 23), (240, 200), (320, 310), (640, 487)])
def test_every_ray_is_counted(wf, dev, scene, w, h):
    # The record form: per-lane triangle tests of the BVH8.
    ref, _, rays = counted(wf, dev, scene, w, h, [("trace.bvh8.coop", 0)], bvh_kind=1)
    for kind in (0, 1):
        bits, counts, total = counted(wf, dev, scene, w, h, [("trace.count", 1)], bvh_kind=kind)
        assert np.array_equal(bits, ref)
        assert counts["rays"] == total == rays
        assert counts["nodes"] >= rays and (w * h < 800 or counts["tris"] > 0)
    assert wf.api.device_status() == 0


def test_counts_are_those_of_the_occlusion_kernel(wf, dev, scene):
    """One warp of shadow rays, whose steps are always the same.  The occlusion kernel has no batch;
    the kernel with any-hit records tests later with a larger one and takes more node steps."""
    def run(batch):
        return counted(wf, dev, scene, 8, 4, [("trace.count", 1), ("trace.bvh8.any_batch", batch)], bvh_kind=1,
                       ray_type=wf.SHADOW_RAYS, num_shadow_samples=1)[1]
    one = run(1)
    assert one == run(1) and one["rays"] > 32
    assert one == run(32)
