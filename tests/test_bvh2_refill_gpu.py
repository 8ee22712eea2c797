"""FP32 BVH2 traversal with lanes that take new rays (a renderer's bounce rays
whose capacity is 194,560 or more, shadow rays from that many on): the frames
of the BVH8, bit for bit, on both sides of that size, for one to three shadow
samples, sorted, reordered and unsorted rays, counted traversal, graphs."""
import numpy as np
import pytest

from test_occluded_gpu import frame, scene  # noqa: F401

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("w,h", [(320, 304), (512, 379), (512, 380), (779, 501)])
def test_same_frames(wf, dev, scene, w, h):  # noqa: F811
    for cfg in (dict(), dict(num_shadow_samples=1, sort_path_rays=0), dict(num_shadow_samples=3, sort_shadow_rays=1),
                dict(reorder_path_rays=0, use_graph=1, recursion_depth=4), dict(shadow_overlap=0)):
        ref = frame(wf, dev, scene, w, h, bvh_kind=wf.BVH8_Q8, **cfg)
        assert np.array_equal(ref, frame(wf, dev, scene, w, h, bvh_kind=wf.BVH2_FP32, **cfg)), cfg
    wf.api.tune_set("trace.count", 1)
    try:
        got = frame(wf, dev, scene, w, h, bvh_kind=wf.BVH2_FP32, **cfg)
    finally:
        wf.api.tune_set("trace.count", 0)
    assert np.array_equal(ref, got)
    assert wf.api.device_status() == 0
