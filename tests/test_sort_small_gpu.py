"""Small sorts (tiles of 1,024 pairs up to 131,072 of them, of 2,048 up to
393,216, the larger tiles also where three passes or fewer leave too little
look-back space): sizes at the edges of tiles and of both ranges, every number
of passes, device counts, scratch that starts with arbitrary bytes, and few
distinct keys (stability)."""
import pytest

pytestmark = pytest.mark.gpu

SIZES = [1, 2, 1023, 1024, 1025, 3000, 66001, 131071, 131072, 131073, 133121, 393215, 393216, 393217]


@pytest.mark.parametrize("bits", [5, 8, 16, 20, 24, 30, 32, 33, 47, 63, 64])
def test_small_sorts(wf, dev, bits):
    import torch
    g = torch.Generator(device=dev).manual_seed(bits)
    wide = bits > 32
    mask = -1 if bits in (32, 64) else (1 << bits) - 1
    for n in SIZES:
        for distinct in (0, 3):
            lo, hi, dt = (-(2**63), 2**63 - 1, torch.int64) if wide else (-(2**31), 2**31 - 1, torch.int32)
            keys = torch.randint(lo, hi, (n,), generator=g, device=dev, dtype=dt)
            if distinct:
                keys = keys[torch.randint(0, min(n, distinct), (n,), generator=g, device=dev)]
            keys = keys & mask
            for count in (None, 0, n // 2 + 1, n):
                k, v = keys.clone(), torch.arange(n, device=dev, dtype=torch.int32)
                scratch = torch.full((wf.api.sort_scratch_bytes(n, bits),), 0xA5, dtype=torch.uint8, device=dev)
                cnt = None if count is None else torch.tensor([count], dtype=torch.int32, device=dev)
                wf.api.sort_pairs(k, v, bits, n_dev=cnt, scratch=scratch)
                c = n if count is None else count
                order = torch.arange(n, device=dev)
                # unsigned order: flip the sign bit
                flip = (keys ^ lo)[:c]
                order[:c] = torch.sort(flip, stable=True).indices
                assert torch.equal(v.long(), order), (n, distinct, count)
                assert torch.equal(k, keys[order]), (n, distinct, count)
    assert wf.api.device_status() == 0
