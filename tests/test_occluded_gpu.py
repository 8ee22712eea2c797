"""Shadow passes of the renderer trace for occlusion alone (one word per ray);
with traversal counting or per-lane triangle tests they trace any-hit records.
The same frames both ways, for both BVHs, sorted, reordered and unsorted shadow
rays, on both sides of the sizes at which the kernels change (97,280 rays of
the BVH2, 622,592 of the BVH8), and two of the frames replayed as graphs."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def scene(wf, dev):
    pos, nrm, idx = wf.api.generate_scene(0, 21, 4000)
    sc = wf.api.Scene(pos, idx)
    return sc, wf.api.Geometry(pos, nrm, idx, device=dev)


def frame(wf, dev, scene, w, h, **cfg):
    import torch
    r = wf.api.Renderer(**dict(dict(ray_type=wf.PATH_RAYS, recursion_depth=2, num_shadow_samples=2, shadow_radius=0.2,
                                    sort_path_rays=1, reorder_path_rays=1, morton_kind=2), **cfg))
    r.set_scene(*scene, (0.5, 1.6, 0.5), (0.5, 0.8, 1.0))
    cam = wf.api.make_camera(position=(0.5, 0.5, 2.2), rotation_deg=(0, 0, 0), fov_deg=45.0, znear=0.001, zfar=10.0)
    px = torch.zeros((w * h, 4), dtype=torch.float32, device=dev)
    fp = torch.zeros_like(px)
    for _ in range(2):
        r.render(cam, w, h, px, fp)
    out = fp.cpu().numpy()
    r.close()
    out[np.isnan(out)] = np.nan
    return out.view(np.uint32)


@pytest.mark.parametrize("w,h", [(1, 1), (37, 23), (240, 200), (250, 200), (640, 486), (640, 487)])
@pytest.mark.parametrize("kind", [0, 1])
def test_same_frames(wf, dev, scene, w, h, kind):
    for cfg in (dict(), dict(sort_shadow_rays=1), dict(sort_shadow_rays=1, reorder_shadow_rays=1), dict(use_graph=1),
                dict(shadow_overlap=0, num_shadow_samples=3)):
        got = frame(wf, dev, scene, w, h, bvh_kind=kind, **cfg)
        for knob, value, back in (("trace.count", 1, 0), ("trace.bvh8.coop", 0, 1)):
            wf.api.tune_set(knob, value)
            try:
                assert np.array_equal(got, frame(wf, dev, scene, w, h, bvh_kind=kind, **cfg)), (cfg, knob)
            finally:
                wf.api.tune_set(knob, back)
    assert wf.api.device_status() == 0
