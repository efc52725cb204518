"""Decode attention over INT8 and bf16 caches on tensor cores where the kernel's work changes: contexts at the edges of its blocks of
16 keys and of a row's splits, ragged batches of more rows than a warp has lanes, 1 to 8 query heads a KV head, and whatever a
cache holds past a row's end.  Against 64 bits over what the cache holds."""
import math

import pytest
import torch

from helpers import pkg

pytestmark = pytest.mark.gpu


def attend(q, k, v):
    """q [H, hd], k, v [n, G, hd] in 64 bits."""
    k, v = (t.double().repeat_interleave(q.shape[0] // k.shape[1], 1) for t in (k, v))
    s = torch.einsum("hd,nhd->hn", q.double(), k) / math.sqrt(q.shape[1])
    return torch.einsum("hn,nhd->hd", torch.softmax(s, -1), v)


@pytest.mark.parametrize("kv", ["int8", "bf16"])
@pytest.mark.parametrize("h,kvh,lens", [
    (8, 8, [1, 2, 15, 16, 17]),
    (4, 2, [127, 128, 129, 511, 512, 513]),
    (8, 2, [1, 3000, 40, 1025, 700]),
    (32, 8, [5000]),
    (16, 2, [(37 * r) % 900 + 1 for r in range(70)]),
])
def test_decode_attention(kv, h, kvh, lens):
    p = pkg()
    gen = torch.Generator(device="cuda").manual_seed(len(lens) + h)
    cache = p.KVCache(max(lens) + 21, kvh, 128, h, batch=len(lens), dtype=kv)
    for row, n in enumerate(lens):
        k, v = (torch.randn((1, n + 21, kvh, 128), generator=gen, device="cuda").bfloat16() for _ in range(2))
        k[:, n:] = v[:, n:] = math.nan if kv == "bf16" else 1e4  # past the end of the row: never attended
        cache.append(0, k, v, row0=row)
        cache.commit(n, row0=row, nrows=1)
    q = torch.randn((len(lens), h, 128), generator=gen, device="cuda").bfloat16()
    got = p.dispatch.attention_decode(cache, q, 128 ** -0.5).double().view(len(lens), h, 128)
    for row, n in enumerate(lens):
        k, v = (t.view(n, kvh, 128) if t.shape[-2] == kvh else t.transpose(-3, -2).reshape(n, kvh, 128) for t in cache.read(row))
        want = attend(q[row], k, v)
        # the output's rounding (2^-9 of each value), and over INT8 rows weights of 11 bits
        assert float((got[row] - want).norm()) <= 2.0 ** -8 * float(want.norm())
    again = p.dispatch.attention_decode(cache, q, 128 ** -0.5).double().view(len(lens), h, 128)
    assert torch.equal(got, again)  # the arrival counters are back at rest, and the merge does not depend on the order
