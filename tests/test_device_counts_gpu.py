"""Stage kernels whose count is on the device and whose capacity is beyond
152 x 64 blocks run 152 x 16 blocks that go on until the count is done: the
same outputs as a launch of exactly that many rays, at counts around one
grid's rays (622,592), empty and full, and nothing touched past the count.  A
BVH2 traversal of more than 2^22 rays gives the hits of its halves."""
import numpy as np
import pytest

from conftest import random_rays

pytestmark = pytest.mark.gpu

GRID = 152 * 16 * 256
CAP = 4 * GRID + 77


@pytest.fixture(scope="module")
def wave(wf, dev):
    """Camera-like rays of a small scene and their hits, at capacity."""
    import torch
    pos, nrm, idx = wf.api.generate_scene(0, 51, 3000)
    sc = wf.api.Scene(pos, idx)
    geom = wf.api.Geometry(pos, nrm, idx, device=dev)
    rays = torch.from_numpy(random_rays(np.random.default_rng(1), CAP, tmax=10.0)).to(dev)
    hits = torch.empty((CAP, 4), dtype=torch.int32, device=dev)
    wf.api.trace(sc, wf.BVH8_Q8, rays, hits)
    i2p = torch.randperm(CAP, device=dev).to(torch.int32)
    return geom, rays, hits, i2p


def run(wf, dev, wave, n, count):
    """Every stage over n rays, of which the device count names `count` (None: all)."""
    import torch
    api, S = wf.api, 2
    geom, rays, hits, i2p = wave
    f = lambda *s: torch.full(s, 3.0, dtype=torch.float32, device=dev)
    z = lambda *s: torch.full(s, -9, dtype=torch.int32, device=dev)
    cd = None if count is None else torch.tensor([count], dtype=torch.int32, device=dev)
    o = dict(seeds=z(CAP), srays=f(CAP * S, 8), s2i=z(CAP * S), i2s=z(CAP * S), px=f(CAP, 4), frame=f(CAP, 4), dec=f(CAP, 4), path=f(CAP, 8),
             pi2p=z(CAP), cnt=z(1))
    api.init_seeds(o["seeds"], 5)
    light = (0.5, 1.5, 0.5)
    api.raygen_shadow(o["seeds"], rays, hits, o["srays"], o["s2i"], o["i2s"], light, 0.1, 0, n, S, n_in_dev=cd)
    api.reconstruct_smooth(rays, hits, i2p, o["px"], o["dec"], geom.table, light, (0.1, 0.2, 0.3), 1, n=n, n_dev=cd)
    ident = torch.arange(CAP * S, dtype=torch.int32, device=dev)
    shits = torch.where((ident % 3 == 0)[:, None], torch.full((CAP * S, 4), -1, dtype=torch.int32, device=dev), ident[:, None].expand(-1, 4)).contiguous()
    api.reconstruct_shadow(shits, i2p, ident, o["px"], o["frame"], 0, n, S, n_in_dev=cd)
    scratch = torch.empty(api.raygen_path_scratch_bytes(n), dtype=torch.uint8, device=dev)
    api.raygen_path(o["seeds"], geom.table, rays, o["path"], i2p, o["pi2p"], hits, o["dec"], o["cnt"], n=n, n_dev=cd, scratch=scratch)
    return o


@pytest.mark.parametrize("count", [0, 1, 255, 257, GRID - 1, GRID, GRID + 1, CAP - 1, CAP, CAP + 9])
def test_stages(wf, dev, wave, count):
    import torch
    a, b = run(wf, dev, wave, CAP, count), run(wf, dev, wave, min(count, CAP), None)
    for k in a:
        assert torch.equal(a[k], b[k]), k
    assert wf.api.device_status() == 0


def test_large_bvh2_wavefront(wf, dev):
    import torch
    pos, _, idx = wf.api.generate_scene(0, 52, 500)
    sc = wf.api.Scene(pos, idx)
    n = (1 << 22) + 33
    g = torch.Generator(device=dev).manual_seed(3)
    r = torch.zeros((n, 8), device=dev)
    r[:, :3] = torch.rand((n, 3), generator=g, device=dev)
    r[:, 4:7] = torch.nn.functional.normalize(torch.randn((n, 3), generator=g, device=dev), dim=1)
    r[:, 7] = 2.0
    for closest in (True, False):
        out, part = torch.empty((n, 4), dtype=torch.int32, device=dev), torch.empty((n // 2, 4), dtype=torch.int32, device=dev)
        wf.api.trace(sc, wf.BVH2_FP32, r, out, closest_hit=closest)
        wf.api.trace(sc, wf.BVH2_FP32, r[: n // 2].contiguous(), part, closest_hit=closest)
        assert torch.equal(out[: n // 2], part)
        wf.api.trace(sc, wf.BVH2_FP32, r[n - n // 2:].contiguous(), part, closest_hit=closest)
        assert torch.equal(out[n - n // 2:], part)
    assert wf.api.device_status() == 0
