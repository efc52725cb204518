"""Decode attention over INT8 and bf16 caches on tensor cores where the kernel's work changes: contexts at the edges of its blocks of
16 keys and of a row's splits, ragged batches of more rows than a warp has lanes, 1 to 8 query heads a KV head, and whatever a
cache holds past a row's end.  Against 64 bits over what the cache holds."""
import math

import pytest
import torch

from helpers import pkg
from model_fixtures import SMALL, build_pair

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
    (8, 8, [(5 * r) % 24 + 1 for r in range(40)]),      # more short rows than larger CTAs, the shortest over bf16 on CUDA cores
    (8, 8, [(13 * r) % 512 + 1 for r in range(40)]),
    (32, 8, [25 + r % 3 for r in range(64)]),
    (8, 2, [3, 8, 1]),
    (8, 2, [9, 8, 1]),
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


@pytest.mark.parametrize("n", [9, 700])
def test_bf16_values_at_the_ends_of_the_range(n):
    """Infinite values come out infinite; weighted sums of large ones do not overflow; keys whose scores are -inf weigh nothing,
    a whole block of them ahead of the others too."""
    p = pkg()
    gen = torch.Generator(device="cuda").manual_seed(n)
    cache = p.KVCache(n + 3, 2, 128, 8, batch=3, dtype="bf16")
    k, v = (torch.randn((3, n, 2, 128), generator=gen, device="cuda").bfloat16() for _ in range(2))
    q = torch.randn((3, 8, 128), generator=gen, device="cuda").bfloat16()
    q[:, :, 0] = 1
    v[0, n // 2, 0, 5], v[0, n // 3, 1, 77] = math.inf, -math.inf
    # scores that rise by 8 powers of two from one of a warp's blocks to the next; a weighted sum of the values has room for weights of
    # up to 1 of a hundred tokens
    k[1], q[1] = 0, 0
    q[1, :, 1], k[1, :, :, 1] = 1, (torch.arange(n, device="cuda") // 64 * 60)[:, None].bfloat16()
    v[1, :, :, 3] = 3e36
    k[2, :min(n - 1, 80), :, 0] = -math.inf
    for row in range(3):
        cache.append(0, k[row:row + 1], v[row:row + 1], row0=row)
        cache.commit(n, row0=row, nrows=1)
    got = p.dispatch.attention_decode(cache, q, 128 ** -0.5).double().view(3, 8, 128)
    for row in range(3):
        want = attend(q[row], k[row], v[row])
        if row == 0:
            assert (got[0, :4, 5] == math.inf).all() and (got[0, 4:, 77] == -math.inf).all()
            got[0, :4, 5] = got[0, 4:, 77] = want[:4, 5] = want[4:, 77] = 0
        assert torch.isfinite(got[row]).all() and torch.isfinite(want).all()
        for d in range(128):  # a column at a time: one of row 1 is far larger than the others
            assert float((got[row, :, d] - want[:, d]).norm()) <= 2.0 ** -7 * float(want[:, d].norm()) + 2.0 ** -8


@pytest.mark.parametrize("kv,dtype,shift", [("int8", torch.bfloat16, 1), ("bf16", torch.bfloat16, 3), ("int8", torch.float16, 0), ("int8", torch.float32, 0), ("int8", torch.float32, 1)])
def test_queries_of_other_types_and_places(kv, dtype, shift):
    """f32 and f16 queries, queries off 16 bytes, rows from the middle of a cache; rows that are split and rows that are not."""
    p = pkg()
    lens, row0, h, g = [5, 900, 2100, 31, 1500], 2, 12, 4
    gen = torch.Generator(device="cuda").manual_seed(shift)
    cache = p.KVCache(2200, g, 128, h, batch=row0 + len(lens), dtype=kv)
    for row, n in enumerate(lens):
        k, v = (torch.randn((1, n, g, 128), generator=gen, device="cuda").bfloat16() for _ in range(2))
        cache.append(0, k, v, row0=row0 + row)
        cache.commit(n, row0=row0 + row, nrows=1)
    room = torch.randn(len(lens) * h * 128 + shift, generator=gen, device="cuda").bfloat16().to(dtype)
    q = room[shift:].view(len(lens), h, 128)
    got = p.dispatch.attention_decode(cache, q, 128 ** -0.5, row0=row0).double()
    for row in range(len(lens)):
        want = attend(q[row], *cache.read(row0 + row))
        # weights of 11 bits over INT8 rows, and the output's rounding
        assert float((got[row] - want).norm()) <= (2.0 ** -8 if dtype == torch.bfloat16 else 2.0 ** -10) * float(want.norm())


@pytest.mark.parametrize("n", [1, 5, 100, 3000])
@pytest.mark.parametrize("b,h,kvh", [(2, 8, 2), (50, 8, 8)])
def test_one_query_over_keys_and_values_of_the_caller(b, h, kvh, n):
    gen = torch.Generator(device="cuda").manual_seed(n)
    n = min(n, 100) if b > 2 else n
    q, k, v = (torch.randn((b, heads, t, 128), generator=gen, device="cuda").bfloat16() for heads, t in ((h, 1), (kvh, n), (kvh, n)))
    got = pkg().dispatch.attention_forward_causal(q, k, v, 128 ** -0.5).double()
    for row in range(b):
        want = attend(q[row, :, 0], k[row].transpose(0, 1), v[row].transpose(0, 1))
        assert float((got[row, :, 0] - want).norm()) <= 2.0 ** -8 * float(want.norm())


@pytest.mark.parametrize("kv,row0,rows,lens", [("bf16", 40, 1, 2048), ("bf16", 100, 3, 700), ("int8", 230, 20, 900), ("int8", 250, 38, 1024), ("bf16", 0, 2, 2048)])
def test_fixed_scratch_serves_what_it_served(kv, row0, rows, lens):
    """Rows far up in a cache: the most splits of the tensor-core kernel would not fit the fixed array, fewer do."""
    p = pkg()
    gen = torch.Generator(device="cuda").manual_seed(rows)
    h, g = 32, 8
    cache = p.KVCache(lens, g, 128, h, batch=row0 + rows, dtype=kv)
    for row in range(row0, row0 + rows):
        n = lens - 17 * (row - row0)
        k, v = (torch.randn((1, n, g, 128), generator=gen, device="cuda").bfloat16() for _ in range(2))
        cache.append(0, k, v, row0=row)
        cache.commit(n, row0=row, nrows=1)
    q = torch.randn((rows, h, 128), generator=gen, device="cuda").bfloat16()
    got = p.dispatch.attention_decode_static(cache, q, 128 ** -0.5, torch.empty_like(q), row0=row0).double()
    for row in range(rows):
        want = attend(q[row], *cache.read(row0 + row))
        assert float((got[row] - want).norm()) <= 2.0 ** -8 * float(want.norm())
    if row0 == 0:
        assert torch.equal(got, p.dispatch.attention_decode(cache, q, 128 ** -0.5).double())


@pytest.mark.parametrize("rows,n", [(1, 1300), (1, 4000), (2, 300)])
def test_steps_over_int8_rows_whose_scales_have_no_room_in_fp16(rows, n):
    """Values of 10^7: a step takes their scales, times a weight, in f32.  Against an f32 cache of the same values."""
    c = dict(SMALL, n_layers=1, n_heads=4, n_kv_heads=2, head_dim=128, max_seq=4100)
    model, _, _ = build_pair(c, dtype=torch.bfloat16)
    gen = torch.Generator(device="cuda").manual_seed(n)
    k, v = (torch.randn((rows, n, 2, 128), generator=gen, device="cuda").bfloat16() for _ in range(2))
    v = (v.float() * 3e7).bfloat16()
    out = []
    for kv in ("int8", "f32"):
        cache = pkg().KVCache(n + 4, 2, 128, 4, batch=rows, dtype=kv)
        cache.append(0, k, v)
        cache.commit(n)
        ids = torch.arange(1, rows + 1, dtype=torch.int32, device="cuda")
        logits = torch.empty((rows, 1, c["vocab"]), device="cuda", dtype=model.logits_dtype)
        stream = torch.cuda.Stream()
        torch.cuda.synchronize()
        with torch.cuda.stream(stream):
            model.decode_step(ids, cache, logits, None)
        torch.cuda.synchronize()
        out.append(logits.double())
    assert torch.isfinite(out[0]).all() and torch.isfinite(out[1]).all()
    # codes of 7 bits and a sign: a value's error is at most 2^-8 of its token's largest, about 3 standard deviations
    assert float((out[0] - out[1]).norm()) <= 3 * 2.0 ** -8 * float(out[1].norm())
