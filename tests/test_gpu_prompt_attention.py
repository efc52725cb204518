"""Prompt attention over bf16 and INT8 caches (the tcgen05 kernel from 16 queries on): edges of its tiles of 128 queries and
128 keys, a cached prefix, head sizes that fill one and two boxes of 64, heads per KV head; against 64 bits over exactly what
the cache holds.  The weights enter as two bf16 parts (2^-16), the output is rounded once (2^-9 of each value): the norm of the
error is below 2^-8 of the result's."""
import math

import pytest
import torch

from helpers import pkg

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kv", ["bf16", "int8"])
@pytest.mark.parametrize("h,kvh,hd", [(8, 2, 128), (6, 3, 64)])
@pytest.mark.parametrize("lens,S", [([16], 16), ([17, 144], 17), ([127], 127), ([256, 129], 128), ([129], 129), ([385], 257), ([700], 16)])
def test_prompt_attention(kv, h, kvh, hd, lens, S):
    g = torch.Generator(device="cuda").manual_seed(S + hd)
    p = pkg()
    cache = p.KVCache(max(lens), kvh, hd, h, batch=len(lens), dtype=kv)
    for row, n in enumerate(lens):
        k, v = (torch.randn((1, n, kvh, hd), generator=g, device="cuda") for _ in range(2))
        cache.update(k, v, row0=row)
    q = torch.randn((len(lens), S, h, hd), generator=g, device="cuda").to(torch.bfloat16)
    got = p.dispatch.attention_cached(cache, q, hd ** -0.5).double()
    assert p.device_status() == 0
    for row, n in enumerate(lens):
        k, v = (t.cuda().double().repeat_interleave(h // kvh, 1) for t in cache.read(row))  # [n, h, hd]
        s = torch.einsum("thd,khd->htk", q[row].double(), k) / math.sqrt(hd)
        hidden = torch.arange(n, device="cuda")[None] > torch.arange(n - S, n, device="cuda")[:, None]
        want = torch.einsum("htk,khd->thd", torch.softmax(s.masked_fill(hidden, -math.inf), -1), v)
        assert float((got[row] - want).norm()) <= 2.0 ** -8 * float(want.norm()), row


@pytest.mark.parametrize("kv", ["bf16", "int8"])
@pytest.mark.parametrize("hd", [32, 96, 192])
@pytest.mark.parametrize("S", [1, 15, 16, 40])
def test_head_sizes_are_refused_alike(kv, hd, S):
    """A cache whose head size the attention over caches does not serve is refused for any number of queries."""
    p = pkg()
    cache = p.KVCache(S, 2, hd, 4, dtype=kv)
    k, v = (torch.randn((1, S, 2, hd), device="cuda") for _ in range(2))
    cache.append(0, k, v)
    cache.commit(S)
    with pytest.raises(p.Ab2Error, match="head_dim 64 and 128"):
        p.dispatch.attention_cached(cache, torch.randn((1, S, 4, hd), device="cuda").to(torch.bfloat16), hd ** -0.5)


@pytest.mark.parametrize("kv", ["bf16", "int8"])
@pytest.mark.parametrize("h,kvh,hd", [(8, 2, 128), (6, 3, 64)])
@pytest.mark.parametrize("where", ["keys", "values"])
@pytest.mark.parametrize("bad", [math.inf, math.nan])
def test_tokens_that_are_not_finite_stay_behind_the_mask(kv, h, kvh, hd, where, bad):
    """A token with an Inf or NaN in its key or value changes nothing for the queries before it, in its own tile of 128 keys too."""
    n, S, tokens = 500, 300, (230, 499)  # cached tokens, queries, tokens that are not finite: in the middle of a tile and at the end
    g = torch.Generator(device="cuda").manual_seed(hd)
    p = pkg()
    k, v = (torch.randn((1, n, kvh, hd), generator=g, device="cuda") for _ in range(2))
    q = torch.randn((1, S, h, hd), generator=g, device="cuda").to(torch.bfloat16)
    for t in tokens:
        (k if where == "keys" else v)[0, t, 0, 5] = bad
    cache = p.KVCache(n, kvh, hd, h, dtype=kv)
    cache.append(0, k, v)
    cache.commit(n)
    got = p.dispatch.attention_cached(cache, q, hd ** -0.5)[0].double()
    assert p.device_status() == 0
    kc, vc = (t.cuda().double() for t in cache.read(0))
    for head in range(h):
        kh, vh = kc[:, head * kvh // h], vc[:, head * kvh // h]
        for qi in (0, 29, 30, 31, 127, 298, 299):
            seen = n - S + qi + 1
            w = torch.softmax(kh[:seen] @ q[0, qi, head].double() / math.sqrt(hd), 0)
            want, out = w @ vh[:seen], got[qi, head]
            ok = torch.isfinite(want)
            assert torch.equal(ok, torch.isfinite(out)), (head, qi)
            if ok.any():
                assert float((out[ok] - want[ok]).norm()) <= 2.0 ** -8 * float(want[ok].norm()), (head, qi)
