"""The device build's two cooperative launches (clustering with the collapse
tables, BVH8 emission) against a plain evaluation on the host of the same
rules, from the exported BVHs: the tree is the one that pass-by-pass PLOC
gives, at sizes around one tile of clusters (256 - 2 R), one warp's
look-back window of tiles and one tile of 32 emitted nodes."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def area(lo, hi):
    d = (hi - lo).astype(np.float32)
    return np.float32(2) * (d[..., 0] * d[..., 1] + d[..., 1] * d[..., 2] + d[..., 2] * d[..., 0])


def ploc(lo, hi, radius):
    """Children (pairs of ids) of the inner nodes in creation order."""
    n = lo.shape[0]
    lo, hi = list(lo), list(hi)
    cl = list(range(n))
    kids = []
    while len(cl) > 1:
        m = len(cl)
        L, H = np.array([lo[c] for c in cl]), np.array([hi[c] for c in cl])
        best = np.full(m, np.inf, np.float32)
        nn = np.full(m, -1)
        for d in [x for x in range(-radius, radius + 1) if x]:
            i = np.arange(max(0, -d), min(m, m - d))
            if i.size == 0:
                continue
            a = area(np.minimum(L[i], L[i + d]), np.maximum(H[i], H[i + d]))
            better = a < best[i]
            best[i[better]] = a[better]
            nn[i[better]] = i[better] + d
        out = []
        for i in range(m):
            j = nn[i]
            mutual = j >= 0 and nn[j] == i
            if mutual and i > j:
                continue
            if mutual:
                kids.append((cl[i], cl[j]))
                lo.append(np.minimum(L[i], L[j]))
                hi.append(np.maximum(H[i], H[j]))
                out.append(len(lo) - 1)
            else:
                out.append(cl[i])
        cl = out
    return kids


@pytest.mark.parametrize("n,radius", [(2, 8), (31, 8), (239, 8), (240, 8), (241, 8), (481, 8), (8000, 8), (129, 64),
                                      (1000, 64), (255, 1), (7700, 1)])
def test_clusters_follow_the_passes(wf, dev, n, radius):
    import torch
    pos, _, idx = wf.api.generate_scene(0, 21, n)
    old = wf.api.tune_get("build.ploc.radius")
    try:
        wf.api.tune_set("build.ploc.radius", radius)
        sc = wf.api.Scene.from_device(torch.from_numpy(pos).to(dev), torch.from_numpy(idx.view(np.int32)).to(dev))
    finally:
        wf.api.tune_set("build.ploc.radius", old)
    nodes, tris = sc.export_bvh2()
    v = tris.view(np.float32).reshape(-1, 12)[:, [0, 1, 2, 4, 5, 6, 8, 9, 10]].reshape(-1, 3, 3)
    kids = ploc(v.min(1), v.max(1), radius)
    links = nodes.view(np.int32).reshape(-1, 16)[:, 12:14]
    assert links.shape[0] == n - 1 == len(kids)
    last = 2 * n - 2
    for k, pair in enumerate(kids):
        got = [(~int(x) & 0xFFFFFFFF) >> 3 if x < 0 else last - int(x) for x in links[last - (n + k)]]
        assert got == list(pair)
    assert wf.api.device_status() == 0


def test_degenerate_meshes(wf, dev):
    """Coincident triangles (every area ties; a pass merges few pairs) and a flat strip."""
    import torch
    pos = np.array([[0, 0, 0], [1, 0, 0], [0, 1, 0]], np.float32)
    idx = np.tile(np.arange(3, dtype=np.int32), (40, 1))
    sc = wf.api.Scene.from_device(torch.from_numpy(pos).to(dev), torch.from_numpy(idx).to(dev))
    assert sc.info.bvh2_nodes == 39
    rays = torch.tensor([[0.2, 0.2, 1, 0, 0, 0, -1, 10]], dtype=torch.float32, device=dev)
    hits = torch.empty((1, 4), dtype=torch.int32, device=dev)
    for kind in (0, 1):
        wf.api.trace(sc, kind, rays, hits)
        assert int(hits[0, 0]) == 0  # ties go to the smallest triangle index
    x = np.arange(1002, dtype=np.float32)
    strip = np.stack([x, np.zeros_like(x), (x % 2)], 1)
    tri = np.stack([np.arange(1000), np.arange(1, 1001), np.arange(2, 1002)], 1).astype(np.int32)
    sc = wf.api.Scene.from_device(torch.from_numpy(strip).to(dev), torch.from_numpy(tri).to(dev))
    assert sc.info.bvh2_nodes == 999
    ids = sc.export_bvh8()[1].view(np.uint32).reshape(-1, 12)[:, 11]
    assert np.array_equal(np.sort(ids), np.arange(1000))
    assert wf.api.device_status() == 0
