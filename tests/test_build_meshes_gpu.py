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


def area(lo, hi):
    d = (hi - lo).astype(np.float32)
    return np.float32(2) * (d[:, 0] * d[:, 1] + d[:, 1] * d[:, 2] + d[:, 2] * d[:, 0])


def ploc(lo, hi, radius):
    """The clustering on the host: (children of the inner nodes in creation order, clusters before
    each pass, depth).  Ties of the merged area go to the run of equal boxes, the least i xor j first, then
    to the smaller position (after a pass that merged less than 1 in 32 of its clusters the least i xor j)."""
    n = lo.shape[0]
    ids = np.arange(n)
    depth = np.zeros(n, int)
    kids, sizes, pair_ties = [], [], False
    while ids.size > 1:
        m = ids.size
        sizes.append(m)
        run = np.concatenate([[0], np.cumsum(np.any((lo[1:] != lo[:-1]) | (hi[1:] != hi[:-1]), 1))])
        best, tie, nn = np.full(m, np.inf, np.float32), np.full(m, 2**40), np.full(m, -1)
        for d in [x for x in range(-radius, radius + 1) if x and abs(x) < m]:
            i = np.arange(max(0, -d), min(m, m - d))
            a = area(np.minimum(lo[i], lo[i + d]), np.maximum(hi[i], hi[i + d]))
            same = run[i] == run[i + d]
            x = np.where(same, i ^ (i + d), 2**30 + (i ^ (i + d) if pair_ties else i + d))
            better = (a < best[i]) | ((a == best[i]) & (x < tie[i]))
            j = i[better]
            best[j], tie[j], nn[j] = a[better], x[better], j + d
        pos = np.arange(m)
        mutual = nn[nn] == pos
        first, second = mutual & (pos < nn), mutual & (pos > nn)
        a, b = pos[first], nn[first]
        kids += list(zip(ids[a].tolist(), ids[b].tolist()))
        ids, depth = ids.copy(), depth.copy()
        ids[a] = n + len(kids) - a.size + np.arange(a.size)
        depth[a] = np.maximum(depth[a], depth[b]) + 1
        lo, hi = lo.copy(), hi.copy()
        lo[a], hi[a] = np.minimum(lo[a], lo[b]), np.maximum(hi[a], hi[b])
        ids, depth, lo, hi = ids[~second], depth[~second], lo[~second], hi[~second]
        pair_ties = pair_ties or m - ids.size < m // 32
    return kids, sizes, int(depth[0])


def strip(x):
    """Triangles of a strip along x with vertices at the given places."""
    pos = np.stack([x, 0 * x, np.arange(x.size) % 2], 1).astype(np.float32)
    i = np.arange(x.size - 2)
    return pos, np.stack([i, i + 1, i + 2], 1)


def coincident(n):
    return np.array([[0, 0, 0], [1, 0, 0], [0, 1, 0]], np.float32), np.tile(np.arange(3), (n, 1))


def graded(n):
    return strip(np.cumsum(np.arange(n + 2, 0, -1, dtype=np.float64)) / n)


# mesh, radius, passes at most, depth at most; the graded strip's passes go past the 128 that the
# clustering's look-back states tell apart, with several tiles of clusters at the time, and past the
# 256 of one launch
MESHES = [("coincident", 40, 8, 6, 6), ("coincident", 241, 8, 8, 8), ("coincident", 400, 8, 9, 9),
          ("coincident", 600, 64, 10, 10), ("coincident", 100000, 8, 17, 17), ("coincident", 100000, 1, 17, 17),
          ("padded", 80, 8, 40, 30), ("padded", 5000, 8, 40, 30), ("equal", 63, 8, 40, 20),
          ("equal", 5000, 8, 32, 20), ("graded", 40000, 64, 300, 40), ("graded", 40000, 8, 300, 40)]


def padded(n):
    """A soup of triangles, and an index buffer filled up with 0, 0, 0."""
    g = np.random.default_rng(7).random((3000, 1, 3)) * 50
    pos = (g + np.random.default_rng(8).random((3000, 3, 3))).reshape(-1, 3).astype(np.float32)
    return pos, np.concatenate([np.arange(9000).reshape(-1, 3), np.zeros((n, 3), int)])


def mesh(name, n):
    return dict(coincident=coincident, padded=padded, equal=lambda k: strip(np.arange(k + 2.0)), graded=graded)[name](n)


@pytest.mark.parametrize("name,n,radius,passes,depth", MESHES)
def test_ties_do_not_make_chains(wf, dev, name, n, radius, passes, depth):
    import torch
    pos, idx = mesh(name, n)
    n = idx.shape[0]
    old = wf.api.tune_get("build.ploc.radius")
    try:
        wf.api.tune_set("build.ploc.radius", radius)
        launches = wf.api.lib().wfpt_kernel_launch_count()
        sc = build(wf, dev, pos, idx)
    finally:
        wf.api.tune_set("build.ploc.radius", old)
    launches = wf.api.lib().wfpt_kernel_launch_count() - launches
    nodes, tris = sc.export_bvh2()
    v = tris.view(np.float32).reshape(-1, 12)[:, [0, 1, 2, 4, 5, 6, 8, 9, 10]].reshape(-1, 3, 3)
    kids, sizes, deep = ploc(v.min(1), v.max(1), radius)
    assert len(sizes) <= passes and deep <= depth
    # Three kernels, the sort's ten (clear, histograms, eight passes), clustering and emission.
    assert launches == 13 + 2 * -(-len(sizes) // 256)
    if (name, radius) == ("graded", 64):
        assert len(sizes) > 256 and sizes[128] > 256 - 2 * radius
    links = nodes.view(np.int32).reshape(-1, 16)[::-1, 12:14].astype(np.int64)
    assert np.array_equal(np.where(links < 0, (~links & 0xFFFFFFFF) >> 3, 2 * n - 2 - links), np.array(kids))
    ids = sc.export_bvh8()[1].view(np.uint32).reshape(-1, 12)[:, 11]
    assert np.array_equal(np.sort(ids), np.arange(n))
    # Rays through the middles of triangles, the same hits as in a scene built on the host.
    v = pos[idx[:: max(1, n // 500)]]
    normal = np.cross(v[:, 1] - v[:, 0], v[:, 2] - v[:, 0])
    rays = np.zeros((v.shape[0], 8), np.float32)
    rays[:, :3], rays[:, 4:7], rays[:, 7] = v.mean(1) + normal, -normal, 10
    rays = torch.from_numpy(rays).to(dev)
    ref = torch.empty((v.shape[0], 4), dtype=torch.int32, device=dev)
    wf.api.trace(wf.api.Scene(pos, idx.astype(np.uint32)), 0, rays, ref)
    assert int(ref[0, 0]) >= 0
    for kind in (0, 1):
        hits = torch.empty_like(ref)
        wf.api.trace(sc, kind, rays, hits)
        assert torch.equal(hits, ref)
    assert wf.api.device_status() == 0


def test_nested_triangles_are_refused_by_name(wf, dev):
    """A thousand triangles nested in one another cluster into a chain, deeper than the BVH8's limit."""
    scale = 100 * 1.05 ** -np.arange(1000.0)
    pos = np.array([[-1, -1, 0], [1, -1, 0.1], [0, 1, 0.2]]) * scale[:, None, None]
    pos, idx = pos.reshape(-1, 3).astype(np.float32), np.arange(3000).reshape(-1, 3)
    with pytest.raises(wf.WfptError) as err:
        build(wf, dev, pos, idx)
    assert "nested too deep" in str(err.value) and "UNSUPPORTED" in str(err.value)
    assert wf.api.Scene(pos, idx.astype(np.uint32)).info.num_triangles == 1000
    assert wf.api.device_status() == 0
