"""Device builds of meshes that are wrong or degenerate."""
import time

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def build(wf, dev, pos, idx):
    import torch
    return wf.api.Scene.from_device(torch.from_numpy(np.ascontiguousarray(pos, np.float32)).to(dev),
                                    torch.from_numpy(np.ascontiguousarray(idx).astype(np.int32)).to(dev))


def test_bad_indices_are_refused_at_once(wf, dev):
    """An index buffer that is wrong throughout: every triangle is read as one point, whose clustering
    would take a pass per triangle."""
    pos = np.random.default_rng(1).random((1000, 3))
    idx = np.arange(1000, 6001000).reshape(-1, 3)
    build(wf, dev, pos, idx[:4] % 1000).close()
    t = time.perf_counter()
    with pytest.raises(wf.WfptError):
        build(wf, dev, pos, idx)
    assert time.perf_counter() - t < 2.0  # 2M triangles: the sort's milliseconds, not 2M passes
    assert wf.api.device_status() == 0
