"""BVH8 traversal on both sides of the wavefront size (four times the 152 x 4
x 256 rays resident at once) from which it runs with four blocks per SM: the
same records, closest and any hit, as the same rays in smaller wavefronts,
and with a device count far below the capacity."""
import numpy as np
import pytest

from conftest import random_rays

pytestmark = pytest.mark.gpu

EDGE = 4 * 152 * 4 * 256


@pytest.mark.parametrize("n", [EDGE - 1, EDGE, EDGE + 1])
@pytest.mark.parametrize("closest", [True, False])
def test_both_register_shapes(wf, dev, n, closest):
    import torch
    pos, _, idx = wf.api.generate_scene(0, 61, 8000)
    sc = wf.api.Scene(pos, idx)
    r = torch.from_numpy(random_rays(np.random.default_rng(3), n, tmax=1.2)).to(dev)
    out = torch.full((n, 4), 7, dtype=torch.int32, device=dev)
    for _ in range(2):
        wf.api.trace(sc, wf.BVH8_Q8, r, out, closest_hit=closest)
    for a in range(0, n, 150001):
        part = torch.empty_like(out[a:a + 150001])
        wf.api.trace(sc, wf.BVH8_Q8, r[a:a + 150001].contiguous(), part, closest_hit=closest)
        assert torch.equal(out[a:a + 150001], part)
    cnt = torch.tensor([12345], dtype=torch.int32, device=dev)
    got = torch.full((n, 4), 7, dtype=torch.int32, device=dev)
    wf.api.trace(sc, wf.BVH8_Q8, r, got, closest_hit=closest, n=n, n_dev=cnt)
    assert torch.equal(got[:12345], out[:12345]) and bool((got[12345:] == 7).all())
    assert wf.api.device_status() == 0
