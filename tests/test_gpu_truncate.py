"""Cutting a row does not wait for the GPU: it takes its place in its stream, and calls on the cache from other streams come after it."""
import pytest
import torch

from helpers import pkg

pytestmark = pytest.mark.gpu


def filled(rows, n):
    gen = torch.Generator(device="cuda").manual_seed(n)
    cache = pkg().KVCache(n + 8, 2, 128, 4, batch=rows, dtype="bf16")
    k, v = (torch.randn((rows, n, 2, 128), generator=gen, device="cuda").bfloat16() for _ in range(2))
    cache.append(0, k, v)
    cache.commit(n, row0=0, nrows=rows)
    return cache, k, v


def test_a_cut_takes_its_place_in_the_stream():
    cache, k, _ = filled(3, 40)
    side = torch.cuda.Stream()
    torch.cuda.synchronize()
    with torch.cuda.stream(side):
        torch.cuda._sleep(200_000_000)       # the cut below is still to come when the call returns
        cache.truncate(7, 1)
    assert cache.seq_len(1) == 7 and not side.query()
    new = torch.ones((1, 1, 2, 128), device="cuda", dtype=torch.bfloat16)
    cache.append(0, new, new, row0=1)        # another stream: after the cut
    cache.commit(1, row0=1, nrows=1)
    got = cache.read(1)[0]
    assert got.shape[0] == 8 and torch.equal(got[:7].bfloat16(), k[1, :7]) and (got[7] == 1).all()
    q = torch.randn((3, 4, 128), device="cuda", dtype=torch.bfloat16)
    assert torch.isfinite(pkg().dispatch.attention_decode(cache, q, 0.1).float()).all()
    assert [cache.seq_len(r) for r in range(3)] == [40, 8, 40]


def test_many_cuts_in_a_row():
    cache, k, _ = filled(33, 50)
    for n in (49, 20, 3):
        for r in range(33):
            cache.truncate(n if r % 2 else 50 if n == 49 else n + 1, r)
    for r in (0, 1, 32):
        n = 3 if r % 2 else 4
        assert torch.equal(cache.read(r)[0].bfloat16(), k[r, :n])
