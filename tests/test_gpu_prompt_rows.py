"""Prompts of several sequences in one call, and window layers at the edges of their tiles of 128 keys: lengths of their own,
rings that wrap, sequences picked out of a batch; against 64 bits over what the caches hold.  The weights enter as two bf16
parts (2^-16), the output is rounded once (2^-9 of each value): the norm of the error is below 2^-8 of the result's."""
import ctypes as C
import math

import pytest
import torch

from helpers import pkg
from model_fixtures import SMALL, build_pair

pytestmark = pytest.mark.gpu


def attend(q, k, v, scale, window=0):
    """q [S, H, dim] at the last positions of k [L, G, dim], v [L, G, vdim], in 64 bits."""
    S, L, rep = q.shape[0], k.shape[0], q.shape[1] // k.shape[1]
    k, v = (t.double().repeat_interleave(rep, 1) for t in (k, v))
    back = torch.arange(L - S, L, device="cuda")[:, None] - torch.arange(L, device="cuda")[None]
    hidden = (back < 0) | (back >= (window or L))
    s = torch.einsum("thd,khd->htk", q.double(), k) * scale
    return torch.einsum("htk,khd->thd", torch.softmax(s.masked_fill(hidden, -math.inf), -1), v)


def close(got, want):
    assert float((got.double() - want).norm()) <= 2.0 ** -8 * float(want.norm())


@pytest.mark.parametrize("kv", ["bf16", "int8"])
@pytest.mark.parametrize("h,kvh,hd", [(8, 2, 128), (4, 4, 64)])
@pytest.mark.parametrize("S,lens", [(16, (16, 700, 17, 150)), (40, (300, 40, 41, 168, 129)), (130, (130, 400)), (257, (513, 300, 257))])
def test_prompts_of_several_sequences(kv, h, kvh, hd, S, lens):
    p = pkg()
    g = torch.Generator(device="cuda").manual_seed(S + hd)
    cache = p.KVCache(max(lens) + 5, kvh, hd, h, batch=len(lens) + 2, n_layers=2, dtype=kv)
    for row, n in enumerate(lens):
        k, v = (torch.randn((1, n, kvh, hd), generator=g, device="cuda") for _ in range(2))
        cache.append(1, k, v, row0=row + 1)
        cache.commit(n, row + 1, 1)
    q = torch.randn((len(lens), S, h, hd), generator=g, device="cuda").to(torch.bfloat16)
    got = p.dispatch.attention_cached(cache, q, hd ** -0.5, layer=1, row0=1)
    assert p.device_status() == 0
    for row, n in enumerate(lens):
        k, v = (t.cuda() for t in cache.read(row + 1, 1))
        close(got[row], attend(q[row], k, v, hd ** -0.5))
    alone = torch.cat([p.dispatch.attention_cached(cache, q[i:i + 1], hd ** -0.5, layer=1, row0=i + 1) for i in range(len(lens))])
    close(got, alone.double())


@pytest.mark.parametrize("window", [1, 127, 128, 129, 200])
@pytest.mark.parametrize("H,G,dim,vdim", [(4, 2, 128, 64), (3, 1, 64, 128)])
@pytest.mark.parametrize("S,before", [(129, (0, 0)), (200, (37, 450)), (257, (300, 300)), (400, (700, 5)), (16, (500, 90, 0))])
def test_window_prompts_of_several_sequences(window, H, G, dim, vdim, S, before):
    p = pkg()
    g = torch.Generator(device="cuda").manual_seed(S + window)
    mix = p.AttentionMixer(H, G, dim, vdim, dim ** -0.5, window)
    cfg = p.StackConfig(64, 64, [(mix, None)], 2048)
    cache = p.KVCache.for_stack(cfg, 1400, len(before), 400, "bf16")
    qkv = [torch.randn((n + S, (H + G) * dim + G * vdim), generator=g, device="cuda").to(torch.bfloat16) for n in before]
    for row, n in enumerate(before):
        for a in range(0, n, 390):
            m = min(390, n - a)
            p.dispatch.window_attention(cache, cfg, 0, qkv[row][None, a:a + m].contiguous(), None, 1e-5, row0=row)
            cache.commit(m, row, 1)
    last = torch.stack([t[n:] for t, n in zip(qkv, before)]).contiguous()
    got = p.dispatch.window_attention(cache, cfg, 0, last, None, 1e-5).view(len(before), S, H, vdim)
    assert p.device_status() == 0
    for row, t in enumerate(qkv):
        q, k, v = t.split([H * dim, G * dim, G * vdim], 1)
        close(got[row], attend(q[-S:].reshape(S, H, dim), k.reshape(-1, G, dim), v.reshape(-1, G, vdim), dim ** -0.5, window))


@pytest.mark.parametrize("kv", ["bf16", "int8"])
def test_rows_picked_out_of_a_batch(kv):
    """A prompt for cache rows 3, 0 and 4 of unequal length gives each row what it gets alone."""
    p = pkg()
    cfg = dict(SMALL, d_model=512, ffn_hidden=1024, n_heads=4, n_kv_heads=2, head_dim=128, max_seq=256)
    gpu, _, _ = build_pair(cfg, "w4a16", dtype=torch.bfloat16, max_tokens=256, capacity=8)
    g = torch.Generator().manual_seed(3)
    rows, S, before = (3, 0, 4), 40, (30, 90, 1)
    ids = torch.randint(0, cfg["vocab"], (len(rows), 256), generator=g, dtype=torch.int32)
    cache, single = (gpu.empty_kv_cache_with_capacity(200, batch=5, dtype=kv) for _ in range(2))
    out = torch.empty((len(rows), S, cfg["vocab"]), dtype=torch.bfloat16, device="cuda")
    for c in (cache, single):
        for i, (r, n) in enumerate(zip(rows, before)):
            gpu.forward_with_cache(ids[i:i + 1, :n], 0, c, row=r)
    last = torch.stack([ids[i, n:n + S] for i, n in enumerate(before)]).cuda().contiguous()
    p._lib.check(p._lib.lib.ab2_model_forward_rows(gpu._h, cache._h, last.data_ptr(), S, (C.c_int * len(rows))(*rows), len(rows), 2, out.data_ptr(), None,
                                                   p.qlinear.stream_ptr()))
    for i, (r, n) in enumerate(zip(rows, before)):
        want = gpu.forward_with_cache(ids[i:i + 1, n:n + S], n, single, row=r)[0].double()
        assert float((out[i].double() - want).norm()) < 2e-2 * float(want.norm()), r
        assert cache.seq_len(r) == n + S
