"""Ray records are written by 256-bit stores where the buffer starts on a
multiple of 32 bytes and by 128-bit ones otherwise: the same records either
way, from every kernel that writes rays; and the 6-D Morton keys against a
bit-by-bit interleaving."""
import numpy as np
import pytest

from conftest import random_rays

pytestmark = pytest.mark.gpu


def buffers(dev, n):
    """A 32-byte aligned ray buffer and one 16 bytes past that."""
    import torch
    out = []
    for skip in (0, 4):
        t = torch.full((n * 8 + 8,), 5.0, dtype=torch.float32, device=dev)
        assert t.data_ptr() % 32 == 0
        out.append(t[skip:skip + 8 * n].view(n, 8))
    return out


@pytest.mark.parametrize("n", [1, 257, 4000])
def test_every_ray_writer(wf, dev, n):
    import torch
    api = wf.api
    pos, nrm, idx = api.generate_scene(0, 71, 2000)
    sc, geom = api.Scene(pos, idx), api.Geometry(pos, nrm, idx, device=dev)
    src = torch.from_numpy(random_rays(np.random.default_rng(n), n, tmax=10.0)).to(dev)
    hits = torch.empty((n, 4), dtype=torch.int32, device=dev)
    api.trace(sc, wf.BVH8_Q8, src, hits)
    z = lambda m: torch.zeros(m, dtype=torch.int32, device=dev)
    ident = torch.arange(n, dtype=torch.int32, device=dev)
    perm = torch.randperm(n, device=dev).to(torch.int32)
    s2w = api.camera_screen_to_world((0.5, 0.5, 2.2), (0, 0, 0), 45.0, n / 1, 0.1, 10.0)

    def primary(o):
        api.raygen_primary(s2w, ident, o, (0.5, 0.5, 2.2), 3, n, 1, 10.0)

    def shadow(o):
        api.raygen_shadow(ident, src, hits, o, z(n), z(n), (0.5, 1.5, 0.5), 0.1, 0, n, 1)

    def path(o):
        seeds = ident.clone()
        api.raygen_path(seeds, geom.table, src, o, ident, z(n), hits, torch.ones((n, 4), device=dev), z(1))

    def reorder(o):
        api.reorder(perm, src, o, ident, z(n), z(n))

    for write in (primary, shadow, path, reorder):
        a, b = buffers(dev, n)
        write(a)
        write(b)
        assert torch.equal(a, b), write.__name__
    # rays and vertices read from buffers 16 bytes past a multiple of 32
    odd = buffers(dev, n)[1]
    odd.copy_(src)
    seeds, o, ref = [ident.clone(), ident.clone()], torch.empty_like(src), torch.empty_like(src)
    verts = torch.zeros(geom.vertices.numel() + 4, dtype=torch.float32, device=dev)[4:]
    verts.copy_(geom.vertices.view(-1))
    table = torch.tensor([[verts.data_ptr(), geom.indices.data_ptr()]], dtype=torch.int64, device=dev)
    for sd, tab, r, out in ((seeds[0], geom.table, src, ref), (seeds[1], table, odd, o)):
        out.fill_(0)
        api.raygen_path(sd, tab, r, out, ident, z(n), hits, torch.ones((n, 4), device=dev), z(1))
    assert torch.equal(o, ref) and torch.equal(seeds[0], seeds[1])
    misread = buffers(dev, n)[1]
    misread.copy_(src)
    o = torch.empty_like(src)
    api.reorder(perm, misread, o, ident, z(n), z(n))
    assert torch.equal(o, src[perm.long()])


@pytest.mark.parametrize("kind,ob,db", [(1, 8, 8), (2, 11, 10)])
def test_morton_interleaving(wf, dev, kind, ob, db):
    import torch
    n = 20000
    rays = random_rays(np.random.default_rng(kind), n, lo=-0.2, hi=1.2)
    rays[:64, :3] = np.array([[(i >> k) & 1 for k in range(3)] for i in range(64)], np.float32)
    for i in range(6):
        rays[64 + i, 4:7] = np.eye(3)[i % 3] * (1 if i < 3 else -1)
    keys = torch.zeros(n, dtype=torch.int64, device=dev)
    ids = torch.zeros(n, dtype=torch.int32, device=dev)
    wf.api.morton(torch.from_numpy(rays).to(dev), (0, 0, 0), (1, 1, 1), kind, keys, ids)
    f = np.float32
    o = np.clip(rays[:, :3], f(0), f(1))
    d = rays[:, 4:7]
    ln = np.sqrt(f(d[:, 0] * d[:, 0]) + d[:, 1] * d[:, 1] + d[:, 2] * d[:, 2], dtype=f)
    b = ((d / ln[:, None] + f(1)) * f(0.5)).astype(f)
    q = np.concatenate([(o * f(2**ob - 1)).astype(np.uint64), (b * f(2**db - 1)).astype(np.uint64)], 1)
    ref = np.zeros(n, np.uint64)
    for axis in range(6):
        for bit in range(10):
            ref |= ((q[:, axis] >> np.uint64(bit)) & np.uint64(1)) << np.uint64(6 * bit + 5 - axis)
    for axis in range(3):
        ref |= ((q[:, axis] >> np.uint64(10)) & np.uint64(1)) << np.uint64(62 - axis)
    assert np.array_equal(keys.cpu().numpy().view(np.uint64), ref)
