"""Any-hit records: the kernel without a ring (tests after every iteration, the
default) against the one with a ring, which traversal counting brings back, at
the same batch -- the same records, below, at and above the sizes at which the
launch shape changes, with duplicate distances, empty intervals, an index and
a device count."""
import numpy as np
import pytest

from conftest import random_rays

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def scene(wf):
    pos, _, idx = wf.api.generate_scene(0, 31, 6000)
    pos, idx = np.asarray(pos), np.asarray(idx)
    # every triangle of a part of the scene twice: equal distances
    return wf.api.Scene(pos, np.concatenate([idx.reshape(-1, 3), idx.reshape(-1, 3)[:1000]]))


def both(wf, run):
    a = run()
    wf.api.tune_set("trace.count", 1)
    try:
        b = run()
    finally:
        wf.api.tune_set("trace.count", 0)
    return a, b


@pytest.mark.parametrize("n", [1, 31, 33, 255, 257, 5000, 116735, 116737, 155649, 622591, 622592, 700001])
def test_same_records(wf, dev, scene, n):
    import torch
    rays = torch.from_numpy(random_rays(np.random.default_rng(n), n, tmax=3.0)).to(dev)
    if n > 40:
        rays[7::40, 7] = -1.0
        rays[9::40, 7] = float("nan")
    order = torch.randperm(n, device=dev).to(torch.int32)
    for index, count in ((None, None), (order, None), (order, n // 2)):
        cnt = None if count is None else torch.tensor([count], dtype=torch.int32, device=dev)

        def run():
            out = torch.full((n, 4), 7, dtype=torch.int32, device=dev)
            wf.api.trace(scene, wf.BVH8_Q8, rays, out, ray_index=index, closest_hit=False, n=n, n_dev=cnt)
            return out
        a, b = both(wf, run)
        assert torch.equal(a, b), (index is None, count)
    assert wf.api.device_status() == 0
