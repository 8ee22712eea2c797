"""Reorder with the new slot map written over the index array, at the sizes where the gather's route
changes: fused, split, and split with the maps in ranges."""
import pytest

pytestmark = pytest.mark.gpu

SPLIT = 10 << 20
RANGE = 1 << 24


@pytest.mark.parametrize("n,count,offset", [(1000, None, 0), (SPLIT - 1, None, 0), (SPLIT + 5, SPLIT - 3, 1), (RANGE, None, 0),
                                            (RANGE + 1, None, 0), (RANGE + 6, RANGE - 11, 1), (2 * RANGE + 3, None, 0)])
@pytest.mark.parametrize("words", [4, 8])
def test_map_over_the_index(wf, dev, n, count, offset, words):
    import torch
    g = torch.Generator(device=dev).manual_seed(n)
    m = n if count is None else count
    idx = torch.zeros(n + offset, dtype=torch.int32, device=dev)[offset:]
    idx[:m] = torch.randperm(m, generator=g, device=dev).to(torch.int32)
    at = idx[:m].long()
    rec = torch.randint(0, 2**31 - 1, (n, words), generator=g, device=dev, dtype=torch.int32)
    s2i = torch.randperm(n, generator=g, device=dev).to(torch.int32)
    out, i2s = torch.empty_like(rec), torch.full_like(s2i, -1)
    n_dev = None if count is None else torch.tensor([count], dtype=torch.int32, device=dev)
    if words == 8:
        wf.api.reorder(idx, rec.view(torch.float32), out.view(torch.float32), s2i, idx, i2s, n=n, n_dev=n_dev)
    else:
        wf.api.reorder_records(idx, rec, out, s2i, idx, i2s, n=n, n_dev=n_dev)
    assert torch.equal(out[:m], rec[at])
    assert torch.equal(idx[:m], s2i[at])
    assert torch.equal(i2s[idx[:m].long()], torch.arange(m, dtype=torch.int32, device=dev))
    assert int((i2s == -1).sum()) == n - m
