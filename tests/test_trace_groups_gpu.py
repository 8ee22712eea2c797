"""BVH8 loop iterations that hand a lane two groups of triangles: hits do not
depend on the knobs, on the wavefront's size (below, at and past the rays
that the grid holds at once, where refills begin) or on a ray's warp-mates,
and the any-hit occluder is the first group's of the traversal order however
many node steps an iteration takes."""
import numpy as np
import pytest

from conftest import random_rays

pytestmark = pytest.mark.gpu

KNOBS = ("trace.bvh8.steps", "trace.bvh8.batch", "trace.bvh8.any_steps", "trace.bvh8.any_batch", "trace.bvh8.refill")


@pytest.fixture(scope="module")
def soup(wf):
    # Triangles packed so that most nodes hand out several triangles at once.
    pos, _, idx = wf.api.generate_scene(0, 31, 20000)
    c = pos.reshape(-1, 3, 3).mean(1, keepdims=True)
    pos = (c + 6.0 * (pos.reshape(-1, 3, 3) - c)).reshape(-1, 3).astype(np.float32)
    return wf.api.Scene(pos, idx)


def rays(dev, n, seed):
    import torch
    r = random_rays(np.random.default_rng(seed), n, tmax=1.5)
    r[::97, 7] = -1.0  # empty intervals
    return torch.from_numpy(r).to(dev)


def trace(wf, scene, kind, r, closest):
    import torch
    out = torch.full((r.shape[0], 4), 7, dtype=torch.int32, device=r.device)
    wf.api.trace(scene, kind, r, out, closest_hit=closest)
    return out


@pytest.mark.parametrize("n", [1, 31, 33, 4097, 152 * 4 * 256 - 1, 152 * 4 * 256, 152 * 4 * 256 + 1, 300001])
def test_sizes(wf, dev, soup, n):
    import torch
    r = rays(dev, n, n)
    assert torch.equal(trace(wf, soup, wf.BVH8_Q8, r, True), trace(wf, soup, wf.BVH2_FP32, r, True))
    a8, a2 = trace(wf, soup, wf.BVH8_Q8, r, False), trace(wf, soup, wf.BVH2_FP32, r, False)
    assert torch.equal(a8[:, 0] >= 0, a2[:, 0] >= 0)
    k = max(1, n // 3)
    assert torch.equal(trace(wf, soup, wf.BVH8_Q8, r[:k].contiguous(), False), a8[:k])
    assert wf.api.device_status() == 0


def test_knobs(wf, dev, soup):
    import torch
    r = rays(dev, 200003, 5)
    ref_c, ref_a = trace(wf, soup, wf.BVH8_Q8, r, True), trace(wf, soup, wf.BVH8_Q8, r, False)
    old = [wf.api.tune_get(k) for k in KNOBS]
    try:
        for steps, batch, refill in ((1, 1, 1), (1, 32, 32), (2, 2, 8), (3, 24, 4), (8, 32, 16), (8, 1, 6)):
            for k, v in zip(KNOBS, (steps, batch, steps, 1, refill)):
                wf.api.tune_set(k, v)
            assert torch.equal(trace(wf, soup, wf.BVH8_Q8, r, True), ref_c)
            assert torch.equal(trace(wf, soup, wf.BVH8_Q8, r, False), ref_a)
            wf.api.tune_set("trace.bvh8.any_batch", 32)
            assert torch.equal(trace(wf, soup, wf.BVH8_Q8, r, False)[:, 0] >= 0, ref_a[:, 0] >= 0)
    finally:
        for k, v in zip(KNOBS, old):
            wf.api.tune_set(k, v)
    assert wf.api.device_status() == 0
