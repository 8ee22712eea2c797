"""Reorder gathers beyond 10 * 2^20 records, where the records and the two
slot maps go in launches of their own and maps beyond 2^24 entries in
ranges: around the threshold, past a range, odd counts, device counts,
pixel-numbered maps (values past the ray count), index arrays that are not
16-byte aligned, and records without maps at small sizes."""
import pytest

pytestmark = pytest.mark.gpu

SPLIT = 10 << 20
RANGE = 1 << 24


def check(wf, dev, n, words, maps, count=None, offset=0, spread=0):
    import torch
    g = torch.Generator(device=dev).manual_seed(n + words)
    rec = torch.randint(-2**31, 2**31 - 1, (n, words), generator=g, device=dev, dtype=torch.int64).to(torch.int32)
    m = n if count is None else count
    # A permutation of the rays that are gathered, in an array that starts
    # `offset` entries past a 16-byte boundary.
    idx = torch.zeros(n + offset, dtype=torch.int32, device=dev)[offset:]
    idx[:m] = torch.randperm(m, generator=g, device=dev).to(torch.int32)
    s2i = torch.randperm(n + spread, generator=g, device=dev).to(torch.int32)[:n].contiguous() if maps else None
    out = torch.full_like(rec, 7)
    os2i = torch.full((n + offset,), -5, dtype=torch.int32, device=dev)[offset:] if maps else None
    oi2s = torch.full((n + spread,), -6, dtype=torch.int32, device=dev) if maps else None
    n_dev = None if count is None else torch.tensor([count], dtype=torch.int32, device=dev)
    wf.api.reorder_records(idx, rec, out, s2i, os2i, oi2s, n=n, n_dev=n_dev)
    at = idx[:m].long()
    assert torch.equal(out[:m], rec[at])
    assert bool((out[m:] == 7).all())
    if maps:
        assert torch.equal(os2i[:m], s2i[at])
        assert bool((os2i[m:] == -5).all())
        ref = torch.full_like(oi2s, -6)
        ref[s2i[at].long()] = torch.arange(m, dtype=torch.int32, device=dev)
        assert torch.equal(oi2s, ref)


@pytest.mark.parametrize("n,words,count,offset,spread", [
    (SPLIT - 1, 8, None, 0, 0), (SPLIT, 8, None, 0, 0), (SPLIT + 5, 8, None, 1, 1000), (SPLIT + 3, 4, SPLIT - 77, 0, 0),
    (SPLIT + 2, 12, 3, 2, 0), (SPLIT + 1, 16, None, 3, 5 << 20), (SPLIT + 64, 8, 0, 0, 0), (RANGE, 8, None, 0, 1),
    (RANGE + 1, 8, None, 0, 0), (RANGE + 3, 12, None, 1, 1 << 20), (2 * RANGE + 7, 4, 2 * RANGE - 9, 0, 123)])
def test_split_reorder(wf, dev, n, words, count, offset, spread):
    check(wf, dev, n, words, True, count, offset, spread)


@pytest.mark.parametrize("words", [4, 8, 12, 16])
@pytest.mark.parametrize("n,count", [(1, None), (255, None), (341, None), (342, 341), (1024, None), (65537, 60000), (SPLIT + 1, None)])
def test_records_without_maps(wf, dev, words, n, count):
    check(wf, dev, n, words, False, count)


def test_reorder_rays_split(wf, dev):
    """wfpt_reorder (32-byte rays) takes the same launches."""
    import torch
    n = SPLIT + 11
    g = torch.Generator(device=dev).manual_seed(1)
    rays = torch.rand((n, 8), generator=g, device=dev)
    idx = torch.randperm(n, generator=g, device=dev).to(torch.int32)
    s2i = torch.randperm(n, generator=g, device=dev).to(torch.int32)
    out, os2i, oi2s = torch.empty_like(rays), torch.empty_like(s2i), torch.empty_like(s2i)
    wf.api.reorder(idx, rays, out, s2i, os2i, oi2s)
    assert torch.equal(out, rays[idx.long()])
    assert torch.equal(os2i, s2i[idx.long()])
    assert torch.equal(oi2s[os2i.long()], torch.arange(n, dtype=torch.int32, device=dev))
    assert wf.api.device_status() == 0
