"""FP32 BVH2 traversal on both sides of the wavefront size from which it runs
as blocks of two warps (half of the 152 x 20 x 64 rays resident in that
shape): the same records, closest and any hit, as a smaller wavefront of the
same rays and (closest) as the BVH8, with device counts and indirect rays."""
import numpy as np
import pytest

from conftest import random_rays

pytestmark = pytest.mark.gpu

EDGE = 152 * 20 * 64 // 2


@pytest.mark.parametrize("n", [EDGE - 1, EDGE, EDGE + 1, EDGE + 63, 2 * EDGE + 65])
def test_both_block_shapes(wf, dev, n):
    import torch
    pos, _, idx = wf.api.generate_scene(0, 41, 30000)
    sc = wf.api.Scene(pos, idx)
    r = random_rays(np.random.default_rng(n), n, tmax=1.0)
    r[::89, 7] = -1.0
    r = torch.from_numpy(r).to(dev)
    small = EDGE - 1
    for closest in (True, False):
        out = torch.full((n, 4), 7, dtype=torch.int32, device=dev)
        wf.api.trace(sc, wf.BVH2_FP32, r, out, closest_hit=closest)
        for a in range(0, n, small):  # the other shape, piece by piece
            part = torch.empty((min(small, n - a), 4), dtype=torch.int32, device=dev)
            wf.api.trace(sc, wf.BVH2_FP32, r[a:a + small].contiguous(), part, closest_hit=closest)
            assert torch.equal(out[a:a + small], part)
        if closest:
            ref = torch.empty_like(out)
            wf.api.trace(sc, wf.BVH8_Q8, r, ref)
            assert torch.equal(out, ref)
        # indirect, and only the first rays of the order
        order = torch.randperm(n, device=dev).to(torch.int32)
        got = torch.full((n, 4), 7, dtype=torch.int32, device=dev)
        cnt = torch.tensor([n - 100], dtype=torch.int32, device=dev)
        wf.api.trace(sc, wf.BVH2_FP32, r, got, ray_index=order, closest_hit=closest, n=n, n_dev=cnt)
        done = order[:n - 100].long()
        assert torch.equal(got[done], out[done]) and bool((got[order[n - 100:].long()] == 7).all())
    assert wf.api.device_status() == 0
