"""The work that users of this framework have it do, as cases that can be timed and checked.

Four families, each through the public entry points:

* ``dense``: the grouped-query decoder over packed weights (``AarambhModel``), decode steps as a generation loop
  runs them and prompts as a session prefills them.  ``large`` is the 4096-wide class with W4A16 weights and an
  INT8 cache, ``tiny`` the 384-wide f32 class, ``gguf`` a 2048-wide decoder over Q4_K_M-style or INT8 payloads.
* ``tovelix`` and ``vipelix``: layer stacks over bf16 weights, decode steps and prompts.
* ``linear``: ``QuantLinear.forward`` alone on one packed weight.
* ``attention``: ``dispatch.attention_decode`` alone on a filled cache.

A decode pass cuts every row of the cache back to where it stood (as a session that is generated anew does) and
feeds ``steps`` given tokens, one step each, with the logits of every step kept.  A prompt pass cuts the row back and
runs its tokens in one call.  Weights are drawn with the value distributions of quantised checkpoints; cached
prefixes of the dense decoder are N(0, 1) keys and values, those of the layer stacks are prompts run by the model.
"""
import importlib.util
import math
import os
import sys

import torch

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
sys.path.insert(0, ROOT)
from __graft_entry__ import import_package  # noqa: E402

DTYPES = {"bf16": torch.bfloat16, "f32": torch.float32}
LINEARS = ("wq", "wk", "wv", "wo", "w_gate", "w_up", "w_down")
EPS = 1e-5

# sizes of the dense decoder's classes: width, heads, KV heads, head size, feed-forward, vocabulary, tied head
DENSE = {
    "large": (4096, 32, 8, 128, 14336, 32000, False),
    "gguf": (2048, 16, 4, 128, 5632, 8192, False),
    "tiny": (384, 6, 2, 64, 1024, 8192, True),
}
# layer stacks at layer sizes of real models; L lightning attention, A window attention
TOVELIX = {
    "w2048": dict(width=2048, heads=16, kv_heads=4, window=1024, experts=32, top=4, ff=1024),
    "w4096": dict(width=4096, heads=32, kv_heads=8, window=2048, experts=8, top=2, ff=7168),
}
VIPELIX = {
    "w2048": dict(width=2048, heads=16, dim=128, rot=64, vdim=128, rank=512, experts=32, top=3, ff=1024, shared=1024, dense=6144),
    "w4096": dict(width=4096, heads=32, dim=128, rot=64, vdim=128, rank=512, experts=8, top=1, ff=7168, shared=7168, dense=21504),
}
STACK_VOCAB = 32000
CLUSTERS = 64     # groups of tokens that a Tovelix router tells apart


def listed():
    return [
        # the smallest model, one sequence: what a step costs in launches and latency
        dict(name="tiny_generate", family="dense", size="tiny", layers=6, weights="int8", dtype="f32", kv="f32", mode="decode",
             rows=1, ctx=32, steps=16),
        # a Q4_K_M checkpoint reads a prompt of a few hundred tokens
        dict(name="gguf_prompt_300", family="dense", size="gguf", layers=4, weights="q4km", dtype="bf16", kv="bf16", mode="prompt",
             rows=1, ctx=0, tokens=300),
        # the benchmark's headline: one user, the whole 32-layer decoder
        dict(name="large_decode_1", family="dense", size="large", layers=32, weights="w4a16", dtype="bf16", kv="int8", mode="decode",
             rows=1, ctx=512, steps=8),
        # a served batch of ragged sequences
        dict(name="large_decode_32", family="dense", size="large", layers=8, weights="w4a16", dtype="bf16", kv="int8", mode="decode",
             rows=32, ctx=700, steps=8),
        # the benchmark's prompt
        dict(name="large_prompt_512", family="dense", size="large", layers=8, weights="w4a16", dtype="bf16", kv="int8", mode="prompt",
             rows=1, ctx=0, tokens=512),
        # a long document of odd length
        dict(name="large_prompt_3001", family="dense", size="large", layers=4, weights="w4a16", dtype="bf16", kv="int8", mode="prompt",
             rows=1, ctx=0, tokens=3001),
        # a prefill product of an INT8 checkpoint
        dict(name="linear_int8_2048", family="linear", weights="int8", n=14336, k=4096, tokens=2048, dtype="bf16"),
        # decode attention of a batch over long INT8 caches
        dict(name="attention_8x16384", family="attention", rows=8, ctx=16384, heads=32, kv_heads=8, kv="int8", dtype="bf16"),
        # a small batch of a mixture-of-experts stack
        dict(name="tovelix_decode_8", family="tovelix", size="w2048", layers="LLLALLLA", mode="decode", rows=8, ctx=512, steps=8),
        dict(name="tovelix_prompt_2048", family="tovelix", size="w2048", layers="LLLALLLA", mode="prompt", rows=1, ctx=0, tokens=2048),
        # a served batch over latent caches
        dict(name="vipelix_decode_32", family="vipelix", size="w2048", layers=4, loops=2, mode="decode", rows=32, ctx=1500, steps=8),
        dict(name="vipelix_prompt_2048", family="vipelix", size="w4096", layers=4, loops=2, mode="prompt", rows=1, ctx=0, tokens=2048),
    ]


def _log(rng, lo, hi):
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi + 1)))))))


def draw(rng):
    kind = rng.choice(["large", "large", "large", "large", "tiny", "gguf", "tovelix", "tovelix", "vipelix", "vipelix", "linear", "linear", "attention"])
    decode = rng.random() < 0.5
    if kind == "large":
        c = dict(family="dense", size="large", layers=rng.randint(2, 4), weights="w4a16", dtype="bf16", kv=rng.choice(["int8", "int8", "bf16"]))
        if decode:
            return dict(c, mode="decode", rows=_log(rng, 1, 64), ctx=_log(rng, 32, 3000), steps=4)
        return dict(c, mode="prompt", rows=1, ctx=rng.choice([0, 0, _log(rng, 64, 2000)]), tokens=_log(rng, 9, 3000))
    if kind == "tiny":
        c = dict(family="dense", size="tiny", layers=6, weights=rng.choice(["int8", "q4km"]), dtype="f32", kv="f32")
        if decode:
            return dict(c, mode="decode", rows=rng.randint(1, 8), ctx=_log(rng, 8, 400), steps=16)
        return dict(c, mode="prompt", rows=1, ctx=0, tokens=_log(rng, 2, 400))
    if kind == "gguf":
        c = dict(family="dense", size="gguf", layers=rng.randint(2, 4), weights=rng.choice(["q4km", "int8"]), dtype="bf16", kv=rng.choice(["bf16", "int8"]))
        if decode:
            return dict(c, mode="decode", rows=rng.randint(1, 8), ctx=_log(rng, 32, 1000), steps=8)
        return dict(c, mode="prompt", rows=1, ctx=0, tokens=_log(rng, 9, 300))
    if kind in ("tovelix", "vipelix"):
        c = dict(family=kind, size=rng.choice(["w2048", "w2048", "w4096"]))
        c.update(layers=rng.choice(["LLA", "ALLA", "LLLALLLA"] if c["size"] == "w2048" else ["LA", "LLA"])) if kind == "tovelix" else \
            c.update(layers=rng.randint(2, 4), loops=rng.randint(1, 2))
        if decode:
            return dict(c, mode="decode", rows=_log(rng, 1, 32), ctx=_log(rng, 32, 1800), steps=4)
        return dict(c, mode="prompt", rows=1, ctx=rng.choice([0, 0, _log(rng, 32, 800)]), tokens=_log(rng, 9, 2048))
    if kind == "linear":
        n, k = rng.choice([(4096, 4096), (14336, 4096), (4096, 14336), (32000, 4096), (1024, 2048), (3000, 1536)])
        fmt = rng.choice(["w4a16", "awq", "int8", "bf16", "q4km"])
        return dict(family="linear", weights=fmt, n=n, k=k, tokens=_log(rng, 1, 300 if fmt == "q4km" else 2500), dtype="bf16")
    rows = _log(rng, 1, 64)
    heads, kv_heads = rng.choice([(32, 8), (16, 4), (32, 4)])
    return dict(family="attention", rows=rows, ctx=_log(rng, 256, min(32768, 262144 // rows)), heads=heads, kv_heads=kv_heads,
                kv=rng.choice(["int8", "int8", "bf16"]), dtype="bf16")


# ---- weights -----------------------------------------------------------------------------------------------

def _gen(seed):
    return torch.Generator(device="cuda").manual_seed(int(seed) + 1)


def _randn(gen, *shape, dtype=torch.float32):
    return torch.randn(shape, generator=gen, device="cuda", dtype=dtype)


def _nibbles(codes, awq):
    """[rows, 8 n] values of 4 bits -> [rows, n] words, in the order of GPTQ or AWQ checkpoints."""
    if awq:
        codes = codes.view(codes.shape[0], -1, 8)[:, :, [0, 2, 4, 6, 1, 3, 5, 7]].reshape(codes.shape[0], -1)
    return (codes[:, 0::2] | (codes[:, 1::2] << 4)).contiguous().view(torch.int32)


class Weight:
    """A packed weight [n, k] as a checkpoint holds it; its values have a standard deviation of about ``std``."""

    def __init__(self, gen, fmt, n, k, std):
        self.fmt, self.n, self.k = fmt, n, k
        if fmt == "bf16":
            self.codes = _randn(gen, n, k, dtype=torch.bfloat16).mul_(std)
        elif fmt == "int8":
            self.codes = _randn(gen, n, k).mul_(32).round_().clamp_(-127, 127).to(torch.int8)
            self.scales = (torch.rand((n, 1), generator=gen, device="cuda") * 0.5 + 0.75) * (std / 32)
        elif fmt == "q4km":
            blocks = n * k // 256
            self.codes = _randn(gen, blocks, 256).mul_(2.5).add_(7.5).round_().clamp_(0, 15).to(torch.uint8)
            self.scales = ((torch.rand((blocks, 1), generator=gen, device="cuda") * 0.5 + 0.75) * (std / 2.5)).half()
            self.mins = (-7.5 * self.scales.float()).half()
        else:
            g = k // 128
            self.codes = _randn(gen, n, k).mul_(2.5).add_(7.5).round_().clamp_(0, 15).to(torch.uint8)
            self.zeros = torch.randint(6, 10, (n, g), generator=gen, device="cuda", dtype=torch.uint8)
            self.scales = ((torch.rand((n, g), generator=gen, device="cuda") * 0.5 + 0.75) * (std / 2.5)).to(torch.bfloat16)

    def linear(self, pkg):
        Q, n, k = pkg.QuantLinear, self.n, self.k
        if self.fmt == "bf16":
            return Q.from_bf16(self.codes)
        if self.fmt == "int8":
            return Q.from_i8_channel(self.codes, self.scales.flatten(), n, k)
        if self.fmt == "q4km":
            head = torch.cat([self.scales, self.mins], 1).contiguous().view(torch.uint8)
            body = self.codes[:, 0::2] | (self.codes[:, 1::2] << 4)
            return Q.from_q4km_blocks(torch.cat([head, body], 1).contiguous(), n, k)
        awq = self.fmt == "awq"
        zeros = torch.nn.functional.pad(self.zeros, (0, -self.zeros.shape[1] % 8))
        make = Q.from_w4a16_awq if awq else Q.from_w4a16_gptq
        # from_* read the arrays as u32 / u16 words, whatever integer type carries them
        return make(_nibbles(self.codes, awq), self.scales.view(torch.int16), _nibbles(zeros, awq), n, k, 128)

    def dense(self):
        c = self.codes.double()
        if self.fmt == "bf16":
            return c
        if self.fmt == "int8":
            return c * self.scales.double()
        if self.fmt == "q4km":
            return (c * self.scales.double() + self.mins.double()).view(self.n, self.k)
        G = self.k // 128
        return ((c.view(self.n, G, 128) - self.zeros.double()[:, :, None]) * self.scales.double()[:, :, None]).view(self.n, self.k)


# ---- the dense decoder ---------------------------------------------------------------------------------------

def _row_lengths(case):
    """Cached tokens of every row: a batch is ragged."""
    return [max(1, case["ctx"] - (r * 37) % (case["ctx"] // 4 + 1)) if case["ctx"] else 0 for r in range(case["rows"])]


def _dense_seed(seed, *at):
    for a in at:
        seed = (seed * 1000003 + a + 7) % (1 << 40)
    return seed


def _dense_model_weights(case, seed):
    d, _, _, _, _, vocab, tied = DENSE[case["size"]]
    gen = _gen(_dense_seed(seed, 0))
    fmt = case["weights"]
    out = {"embedding": Weight(gen, fmt, vocab, d, 0.5)}
    if not tied:
        out["lm_head"] = Weight(gen, fmt, vocab, d, 0.02)
    return out, 1 + 0.1 * _randn(gen, d)


def _dense_layer(case, seed, layer):
    d, h, g, hd, ffn, _, _ = DENSE[case["size"]]
    shapes = {"wq": (h * hd, d), "wk": (g * hd, d), "wv": (g * hd, d), "wo": (d, h * hd), "w_gate": (ffn, d), "w_up": (ffn, d), "w_down": (d, ffn)}
    gen = _gen(_dense_seed(seed, 1, layer))
    # what goes back to the residual stream is small beside it, as in trained models: without that a random stack
    # of this depth amplifies every rounding, and its logits say little about the arithmetic
    std = 0.02 * math.sqrt(4096 / d)
    w = {n: Weight(gen, case["weights"], *s, std * (0.15 if n in ("wo", "w_down") else 1.0)) for n, s in shapes.items()}
    return w, 1 + 0.1 * _randn(gen, d), 1 + 0.1 * _randn(gen, d)


def _dense_prefix(case, seed, layer, row, n):
    """Keys and values [n, kv_heads, head] that a row holds before the pass."""
    _, _, g, hd, _, _, _ = DENSE[case["size"]]
    gen = _gen(_dense_seed(seed, 2, layer, row))
    dt = DTYPES[case["dtype"]]
    return _randn(gen, n, g, hd).to(dt), _randn(gen, n, g, hd).to(dt)


def _tokens(case, seed, vocab):
    n = case["steps"] if case["mode"] == "decode" else case["tokens"]
    return torch.randint(0, vocab, (case["rows"], n), generator=_gen(_dense_seed(seed, 3)), device="cuda")


def _prepare_dense(pkg, case, seed):
    d, h, g, hd, ffn, vocab, tied = DENSE[case["size"]]
    lens = _row_lengths(case)
    new = case["steps"] if case["mode"] == "decode" else case["tokens"]
    cap = max(lens) + new + 8
    top, final = _dense_model_weights(case, seed)
    weights = {n: w.linear(pkg) for n, w in top.items()}
    weights["final_norm"] = final
    for i in range(case["layers"]):
        w, norm1, norm2 = _dense_layer(case, seed, i)
        weights.update({f"layers.{i}.{n}": w[n].linear(pkg) for n in LINEARS})
        weights[f"layers.{i}.norm1"], weights[f"layers.{i}.norm2"] = norm1, norm2
        del w
    cfg = pkg.ModelConfig(case["layers"], d, h, g, hd, ffn, vocab, cap, EPS, 10000.0, tied)
    model = pkg.AarambhModel(cfg, weights, dtype=DTYPES[case["dtype"]], max_tokens=max(64, case["rows"], new))
    cache = pkg.KVCache(cap, g, hd, h, batch=case["rows"], n_layers=case["layers"], dtype=case["kv"])
    for r, n in enumerate(lens):
        if n:
            for i in range(case["layers"]):
                k, v = _dense_prefix(case, seed, i, r, n)
                cache.append(i, k[None], v[None], row0=r)
            cache.commit(n, row0=r, nrows=1)
    return _model_state(case, seed, model, cache, lens, vocab)


def _model_state(case, seed, model, cache, lens, vocab):
    tokens = _tokens(case, seed, vocab)
    s = dict(case=case, model=model, cache=cache, lens=lens, tokens=tokens, stream=torch.cuda.Stream())
    if case["mode"] == "decode":
        s["steps"] = tokens.t().to(torch.int32).contiguous()
        s["ids"] = torch.empty(case["rows"], dtype=torch.int32, device="cuda")
        s["logits"] = torch.empty((case["rows"], 1, vocab), dtype=model.logits_dtype, device="cuda")
        s["out"] = torch.empty((case["steps"], case["rows"], vocab), dtype=model.logits_dtype, device="cuda")
    else:
        s["tokens"] = tokens.cpu()
    torch.cuda.synchronize()
    return s


def _run_model(s):
    case, model, cache, stream = s["case"], s["model"], s["cache"], s["stream"]
    stream.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(stream):
        for r, n in enumerate(s["lens"]):
            cache.truncate(n, r)
        if case["mode"] == "decode":
            out = s["out"]
            for i in range(case["steps"]):
                s["ids"].copy_(s["steps"][i])
                model.decode_step(s["ids"], cache, s["logits"], None)
                out[i].copy_(s["logits"][:, 0])
        else:
            out = model.forward_with_cache(s["tokens"], s["lens"][0], cache, row=0, last_only=True)
            if case["family"] == "dense":
                out = (out,) + tuple(cache.read(0, case["layers"] - 1))
    torch.cuda.current_stream().wait_stream(stream)
    return out


def _norm64(x, w):
    return x * torch.rsqrt(x.square().mean(-1, keepdim=True) + EPS) * w.double()


def _half_rotation(x, pos):
    """x [T, heads, hd] at positions pos: pairs (i, i + hd / 2)."""
    half = x.shape[-1] // 2
    f = 10000.0 ** (-torch.arange(half, dtype=torch.float64, device=x.device) / half)
    a = pos.double()[:, None, None] * f
    x1, x2 = x[..., :half], x[..., half:]
    return torch.cat([x1 * a.cos() - x2 * a.sin(), x1 * a.sin() + x2 * a.cos()], -1)


def _attend(q, k, v, first, scale, window=0):
    """q [T, H, d] of the positions first..., k, v [P, G, *] of all positions: causal, [T, H, dv]."""
    T, H, _ = q.shape
    P, G, _ = k.shape
    i = torch.arange(first, first + T, device=q.device)[:, None]
    j = torch.arange(P, device=q.device)[None, :]
    hidden = (j > i) | ((j <= i - window) if window else torch.zeros_like(j > i))
    out = []
    for g in range(G):
        s = torch.einsum("thd,pd->htp", q[:, g * H // G:(g + 1) * H // G], k[:, g]) * scale
        s.masked_fill_(hidden, -math.inf)
        out.append(torch.einsum("htp,pd->thd", torch.softmax(s, -1), v[:, g]))
    return torch.cat(out, 1)


def _exact_dense(case, seed):
    d, h, g, hd, ffn, vocab, tied = DENSE[case["size"]]
    lens, tokens = _row_lengths(case), _tokens(case, seed, vocab)
    top, final = _dense_model_weights(case, seed)
    x = top["embedding"].dense()[tokens]
    B, T = tokens.shape
    kv = None
    for i in range(case["layers"]):
        packed, norm1, norm2 = _dense_layer(case, seed, i)
        w = {n: p.dense() for n, p in packed.items()}
        y = _norm64(x, norm1)
        q = (y @ w["wq"].T).view(B, T, h, hd)
        k = (y @ w["wk"].T).view(B, T, g, hd)
        v = (y @ w["wv"].T).view(B, T, g, hd)
        rows = []
        for r, n in enumerate(lens):
            pos = torch.arange(n, n + T, device="cuda")
            kr, vr = _half_rotation(k[r], pos), v[r]
            if n:
                k0, v0 = _dense_prefix(case, seed, i, r, n)
                kr, vr = torch.cat([k0.double(), kr]), torch.cat([v0.double(), vr])
            rows.append(_attend(_half_rotation(q[r], pos), kr, vr, n, hd ** -0.5).reshape(T, h * hd))
        x = x + torch.stack(rows) @ w["wo"].T
        y = _norm64(x, norm2)
        x = x + (torch.nn.functional.silu(y @ w["w_gate"].T) * (y @ w["w_up"].T)) @ w["w_down"].T
        kv = (kr, vr)
    head = top["embedding" if tied else "lm_head"].dense()
    if case["mode"] == "decode":
        return (_norm64(x, final) @ head.T).transpose(0, 1).contiguous()
    return (_norm64(x[:, -1:], final) @ head.T,) + kv


def _format_bytes(fmt, n, k):
    return {"w4a16": n * k // 2 + n * (k // 128) * 5 // 2, "awq": n * k // 2 + n * (k // 128) * 5 // 2, "int8": n * k + 4 * n, "q4km": n * k // 256 * 132, "bf16": 2 * n * k}[fmt]


def _work_dense(case):
    d, h, g, hd, ffn, vocab, tied = DENSE[case["size"]]
    fmt, L = case["weights"], case["layers"]
    shapes = [((h + 2 * g) * hd, d), (d, h * hd), (2 * ffn, d), (d, ffn)]
    per_token = 2 * L * sum(n * k for n, k in shapes)
    weights = L * sum(_format_bytes(fmt, n, k) for n, k in shapes)
    row = 2 * g * ({"int8": hd + 4, "bf16": 2 * hd, "f32": 4 * hd}[case["kv"]])
    lens = _row_lengths(case)
    lsize = 4 if case["dtype"] == "f32" else 2
    if case["mode"] == "decode":
        n = case["steps"]
        keys = sum(n * l + n * (n + 1) // 2 for l in lens)
        return {"bytes": n * (weights + _format_bytes(fmt, vocab, d) + case["rows"] * vocab * lsize) + L * row * (keys + n * case["rows"]),
                "flops": n * case["rows"] * (per_token + 2 * vocab * d) + 4 * L * h * hd * keys}
    T, base = case["tokens"], lens[0]
    keys = T * base + T * (T + 1) // 2
    return {"bytes": weights + _format_bytes(fmt, vocab, d) + L * row * (base + T) + T * d * 4, "flops": T * per_token + 2 * vocab * d + 4 * L * h * hd * keys}


# ---- layer stacks --------------------------------------------------------------------------------------------

def _lin(gen, n, k, gain=1.0):
    return _randn(gen, n, k, dtype=torch.bfloat16).mul_(gain * k ** -0.5)


def _experts(gen, w, q, E, ff, d):
    w[q + "gate"], w[q + "up"], w[q + "down"] = _lin(gen, E * ff, d), _lin(gen, E * ff, d), _lin(gen, E * d, ff)


def _gain(gen, n, g=1.0):
    return g * (1 + 0.1 * _randn(gen, n))


def _tovelix_weights(case, seed):
    """name -> bf16 matrix or f32 vector.  Tokens come in clusters, and a router prefers some experts for a
    cluster by a clear margin, as trained routers do: which experts run does not hang on the last bits."""
    c = TOVELIX[case["size"]]
    d, H, G, E, ff = c["width"], c["heads"], c["kv_heads"], c["experts"], c["ff"]
    gen = _gen(_dense_seed(seed, 10))
    centers = _randn(gen, CLUSTERS, d)
    cluster = torch.arange(STACK_VOCAB, device="cuda") % CLUSTERS
    w = {"embedding": ((centers[cluster] + 0.5 * _randn(gen, STACK_VOCAB, d)) * d ** -0.5).to(torch.bfloat16),
         "embed_norm": _gain(gen, d), "final_norm": _gain(gen, d)}
    levels = torch.cat([3.5 - 0.4 * torch.arange(c["top"]), -1.0 - 1.0 * torch.rand(E - c["top"], generator=torch.Generator().manual_seed(1))]).cuda()
    for i, kind in enumerate(case["layers"]):
        q = f"layers.{i}."
        w[q + "in"] = _lin(gen, 4 * H * 128 if kind == "L" else (H + 2 * G) * 128, d)
        if kind == "L":
            w[q + "mix_norm"] = _gain(gen, H * 128)
        w[q + "out"] = _lin(gen, d, H * 128)
        w[q + "norm1"], w[q + "norm2"] = _gain(gen, d, 0.3), _gain(gen, d, 0.3)
        order = torch.rand((CLUSTERS, E), generator=gen, device="cuda").argsort(1)
        w[q + "router"] = (levels[order].T @ centers / d * 1.2).to(torch.bfloat16)
        _experts(gen, w, q, E, ff, d)
    return w


def _tovelix_config(pkg, case, max_seq):
    c = TOVELIX[case["size"]]
    H = c["heads"]
    ffn = pkg.MoeFfn(c["experts"], c["top"], c["ff"], 7.0)
    decay = tuple(_tovelix_decay(H).tolist())
    layers = [(pkg.LightningMixer(H, 128, 128, decay) if k == "L" else
               pkg.AttentionMixer(H, c["kv_heads"], 128, 128, 0.0884, c["window"], 64, 10000.0, True, True, 0.5), ffn) for k in case["layers"]]
    return pkg.StackConfig(c["width"], STACK_VOCAB, layers, max_seq, EPS)


def _tovelix_decay(H):
    return torch.tensor([1 - 2.0 ** (-2 - 6 * h / H) for h in range(H)], dtype=torch.float32)


def _vipelix_weights(case, seed):
    c = VIPELIX[case["size"]]
    d, H, E, top, ff, sh, r = c["width"], c["heads"], c["experts"], c["top"], c["ff"], c["shared"], c["rank"]
    gen = _gen(_dense_seed(seed, 11))
    w = {"embedding": _lin(gen, STACK_VOCAB, d, d ** 0.5), "final_norm": _gain(gen, d, 0.1)}
    if case["loops"] > 1:
        w["loop_steps"] = 0.5 * _randn(gen, case["loops"], d)
    for i in range(case["layers"]):
        q = f"layers.{i}."
        n = H * (c["dim"] + c["rot"]) + r + c["rot"] + H
        w[q + "in"] = _lin(gen, -(-n // 8) * 8, d)
        w[q + "ukv"], w[q + "out"] = _lin(gen, H * (c["dim"] + c["vdim"]), r), _lin(gen, d, H * c["vdim"])
        w[q + "mix_norm"] = _gain(gen, r)
        for n, g in (("pre1", 1.0), ("norm1", 0.5), ("pre2", 1.0), ("norm2", 0.5)):
            w[q + n] = _gain(gen, d, g)
        if i == 0:
            w[q + "up"], w[q + "down"] = _lin(gen, c["dense"], d), _lin(gen, d, c["dense"])
            continue
        w[q + "table"] = torch.rand((STACK_VOCAB, E), generator=gen, device="cuda").topk(top, 1).indices.to(torch.int32)
        _experts(gen, w, q, E, ff, d)
        w[q + "shared_gate"], w[q + "shared_up"], w[q + "shared_down"] = _lin(gen, sh, d), _lin(gen, sh, d), _lin(gen, d, sh)
    return w


POLY = (0.5, 0.3, 0.2, 0.0)


def _vipelix_loop(case):
    """The layers after the first are looped over."""
    return (1, case["layers"], case["loops"]) if case["loops"] > 1 else None


def _vipelix_config(pkg, case, max_seq):
    c = VIPELIX[case["size"]]
    mix = pkg.LatentMixer(c["heads"], c["dim"], c["rot"], c["vdim"], c["rank"], (c["dim"] + c["rot"]) ** -0.5, 10000.0, True)
    moe = pkg.MoeFfn(c["experts"], c["top"], c["ff"], glu="silu", routing="table", shared_ff=c["shared"])
    layers = [(mix, pkg.PolyFfn(c["dense"], POLY) if i == 0 else moe) for i in range(case["layers"])]
    return pkg.StackConfig(c["width"], STACK_VOCAB, layers, max_seq, EPS, embed_norm=False, pre_norms=True, loop=_vipelix_loop(case), logit_softcap=30.0)


def _stack_prompt(case, seed):
    """What the rows held before the pass: tokens [rows, ctx] that the model has read."""
    return torch.randint(0, STACK_VOCAB, (case["rows"], max(case["ctx"], 1)), generator=_gen(_dense_seed(seed, 4)), device="cuda")


def _prepare_stack(pkg, case, seed):
    new = case["steps"] if case["mode"] == "decode" else case["tokens"]
    max_seq = case["ctx"] + new + 8
    make, config = (_tovelix_weights, _tovelix_config) if case["family"] == "tovelix" else (_vipelix_weights, _vipelix_config)
    tensors = make(case, seed)
    weights = {n: pkg.QuantLinear.from_bf16(t) if t.dtype == torch.bfloat16 else t for n, t in tensors.items()}
    del tensors
    model = pkg.StackModel(config(pkg, case, max_seq), weights, torch.bfloat16, max_tokens=max(64, case["rows"], case["ctx"], new))
    cache = model.empty_kv_cache_with_capacity(max_seq, batch=case["rows"])
    lens = _row_lengths(case)
    prompt = _stack_prompt(case, seed)
    for r, n in enumerate(lens):
        if n:
            model.extend_cache(prompt[r:r + 1, :n], cache, row=r)
        cache.save_row(r)
    return _model_state(case, seed, model, cache, lens, STACK_VOCAB)


def _pair_rotation(x, pos, dims):
    """x [T, heads, n]: adjacent pairs of the first ``dims`` dimensions turn."""
    f = 10000.0 ** (-2.0 * torch.arange(dims // 2, dtype=torch.float64, device=x.device) / dims)
    a = pos.double()[:, None, None] * f
    out = x.clone()
    u, v = x[..., 0:dims:2], x[..., 1:dims:2]
    out[..., 0:dims:2], out[..., 1:dims:2] = u * a.cos() - v * a.sin(), v * a.cos() + u * a.sin()
    return out


def _unit(x):
    return x * torch.rsqrt(x.square().mean(-1, keepdim=True) + EPS)


def _lightning64(q, k, v, decay):
    """q, k, v [T, H, n] of one sequence from its start: sums over j <= i of decay^(i-j) (q_i k_j) v_j."""
    T = q.shape[0]
    i = torch.arange(T, device=q.device, dtype=torch.float64)
    gap = i[:, None] - i[None, :]
    out = torch.empty_like(v)
    for h in range(q.shape[1]):
        m = torch.where(gap >= 0, torch.exp(gap.clamp_min(0) * math.log(decay[h])), 0.0)
        out[:, h] = ((q[:, h] @ k[:, h].T) * m) @ v[:, h]
    return out


def _grouped64(h, w, q, ff, d, chosen, act, weigh_in=None, weigh_out=None):
    """Sum over the chosen experts [T, top] of each token's gated unit."""
    out = torch.zeros_like(h)
    gate, up, down = (w[q + n] for n in ("gate", "up", "down"))
    for e in range(gate.shape[0] // ff):
        t, s = (chosen == e).nonzero(as_tuple=True)
        if not len(t):
            continue
        x = h[t] if weigh_in is None else h[t] * weigh_in[t, s][:, None]
        z = act(x @ gate[e * ff:(e + 1) * ff].double().T, x @ up[e * ff:(e + 1) * ff].double().T) @ down[e * d:(e + 1) * d].double().T
        out.index_add_(0, t, z if weigh_out is None else z * weigh_out)
    return out


def _clamped(g, u):
    g, u = g.clamp_max(7.0), u.clamp(-7.0, 7.0)
    return g * torch.sigmoid(1.702 * g) * (u + 1)


def _tovelix64(case, w, rows):
    """Residual stream [sum of lengths, d] after the stack, for sequences ``rows`` of token ids from their starts."""
    c = TOVELIX[case["size"]]
    d, H, G, E, top, ff = c["width"], c["heads"], c["kv_heads"], c["experts"], c["top"], c["ff"]
    silu = torch.nn.functional.silu
    cuts = [len(r) for r in rows]
    x = _norm64(w["embedding"][torch.cat(rows)].double(), w["embed_norm"])
    decay = _tovelix_decay(H).double().tolist()
    v_first = None
    for i, kind in enumerate(case["layers"]):
        q = f"layers.{i}."
        z = x @ w[q + "in"].double().T
        outs = []
        if kind == "L":
            gate = torch.sigmoid(z[:, 3 * H * 128:])
            z = silu(z[:, :3 * H * 128]).view(-1, 3, H, 128)
            outs = [_lightning64(*(p[:, j] for j in range(3)), decay).reshape(-1, H * 128) for p in z.split(cuts)]
            o = _norm64(torch.cat(outs), w[q + "mix_norm"]) * gate
        else:
            v = z[:, (H + G) * 128:].reshape(-1, G, 128)
            v, v_first = (v, v) if v_first is None else (0.5 * v + 0.5 * v_first, v_first)
            for p, pv in zip(z[:, :(H + G) * 128].reshape(-1, H + G, 128).split(cuts), v.split(cuts)):
                p = _unit(_pair_rotation(p, torch.arange(len(p), device=p.device), 64))
                outs.append(_attend(p[:, :H], p[:, H:], pv, 0, 0.0884, c["window"]).reshape(-1, H * 128))
            o = torch.cat(outs)
        x = x + _norm64(o @ w[q + "out"].double().T, w[q + "norm1"])
        s, chosen = torch.sigmoid(x @ w[q + "router"].double().T).topk(top, 1)
        x = x + _norm64(_grouped64(x, w, q, ff, d, chosen, _clamped, weigh_in=s), w[q + "norm2"])
    return x


def _vipelix64(case, w, rows):
    c = VIPELIX[case["size"]]
    d, H, top, ff, sh, r = c["width"], c["heads"], c["top"], c["ff"], c["shared"], c["rank"]
    dim, rot, vdim = c["dim"], c["rot"], c["vdim"]
    silu = torch.nn.functional.silu
    cuts = [len(t) for t in rows]
    ids = torch.cat(rows)
    x = start = w["embedding"][ids].double()
    loop = _vipelix_loop(case)
    runs = [(i, None) for i in range(case["layers"])] if not loop else \
        [(0, None)] + [(i, t if i == 1 else None) for t in range(case["loops"]) for i in range(1, case["layers"])]
    for i, t in runs:
        q = f"layers.{i}."
        if t is not None:
            x = x + (start if t else 0) + w["loop_steps"][t].double()
        z = _norm64(x, w[q + "pre1"]) @ w[q + "in"].double().T
        n = H * (dim + rot)
        lat = _norm64(z[:, n:n + r], w[q + "mix_norm"])
        kv = (lat @ w[q + "ukv"].double().T).view(-1, H, dim + vdim)
        outs = []
        for pq, pr, pkv in zip(z[:, :n].reshape(-1, H, dim + rot).split(cuts), z[:, n + r:n + r + rot].reshape(-1, 1, rot).split(cuts), kv.split(cuts)):
            pos = torch.arange(len(pq), device=pq.device)
            pq = torch.cat([pq[..., :dim], _pair_rotation(pq[..., dim:], pos, rot)], -1)
            pk = torch.cat([pkv[..., :dim], _pair_rotation(pr, pos, rot).expand(-1, H, -1)], -1)
            outs.append(_attend(pq, pk, pkv[..., dim:], 0, (dim + rot) ** -0.5))
        o = torch.cat(outs) * torch.sigmoid(z[:, n + r + rot:n + r + rot + H])[:, :, None]
        x = x + _norm64(o.reshape(-1, H * vdim) @ w[q + "out"].double().T, w[q + "norm1"])
        y = _norm64(x, w[q + "pre2"])
        if i == 0:
            u = y @ w[q + "up"].double().T
            o = (POLY[0] * _unit(u) + POLY[1] * _unit(u * u) + POLY[2] * _unit(u ** 3) + POLY[3]) @ w[q + "down"].double().T
        else:
            o = _grouped64(y, w, q, ff, d, w[q + "table"][ids], lambda g, u: silu(g) * u, weigh_out=1.0 / top)
            o = o + (silu(y @ w[q + "shared_gate"].double().T) * (y @ w[q + "shared_up"].double().T)) @ w[q + "shared_down"].double().T
        x = x + _norm64(o, w[q + "norm2"])
    return x


def _exact_stack(case, seed):
    tovelix = case["family"] == "tovelix"
    w = (_tovelix_weights if tovelix else _vipelix_weights)(case, seed)
    prompt, tokens, lens = _stack_prompt(case, seed), _tokens(case, seed, STACK_VOCAB), _row_lengths(case)
    out = []
    for r0 in range(0, len(lens), 8):   # some rows at a time, for memory
        rows = [torch.cat([prompt[r, :lens[r]], tokens[r]]) for r in range(r0, min(r0 + 8, len(lens)))]
        x = (_tovelix64 if tovelix else _vipelix64)(case, w, rows)
        n = case["steps"] if case["mode"] == "decode" else 1
        x = torch.stack([p[-n:] for p in x.split([len(t) for t in rows])])
        z = _norm64(x, w["final_norm"]) @ w["embedding"].double().T
        out.append(z if tovelix else 30.0 * torch.tanh(z / 30.0))
    out = torch.cat(out)
    return out.transpose(0, 1).contiguous() if case["mode"] == "decode" else out


def _work_stack(case):
    tovelix = case["family"] == "tovelix"
    c = (TOVELIX if tovelix else VIPELIX)[case["size"]]
    d, H, E, top, ff = c["width"], c["heads"], c["experts"], c["top"], c["ff"]
    n = case["steps"] if case["mode"] == "decode" else 1
    T = case["rows"] if case["mode"] == "decode" else case["tokens"]   # tokens of a step
    hit = E * (1 - (1 - top / E) ** T)
    if case["mode"] == "decode":
        spans = [(l + s, 1) for l in _row_lengths(case) for s in range(n)]
    else:
        spans = [(_row_lengths(case)[0], T)]
    byts = n * (2 * STACK_VOCAB * d + T * 4 * STACK_VOCAB if case["mode"] == "decode" else 2 * STACK_VOCAB * d)
    flops = 2 * STACK_VOCAB * d * (n * T if case["mode"] == "decode" else 1)

    def seen(window):
        pairs = sum(sum(min(l + i + 1, window) for i in range(t)) for l, t in spans)
        return pairs, sum(min(l + t, window + t) for l, t in spans)

    if tovelix:
        G = c["kv_heads"]
        for kind in case["layers"]:
            mats = (5 * H if kind == "L" else 2 * H + 2 * G) * 128 * d + E * d
            byts += n * 2 * (mats + 3 * hit * d * ff)
            flops += 2 * n * T * (mats + 3 * top * d * ff)
            if kind == "L":
                byts += len(spans) * 8 * H * 128 * 128
                flops += n * T * H * 4 * 128 * 128
            else:
                pairs, keys = seen(c["window"])
                byts += keys * 4 * G * 128
                flops += 4 * H * 128 * pairs
        return {"bytes": byts, "flops": flops}
    r, dim, rot, vdim = c["rank"], c["dim"], c["rot"], c["vdim"]
    pairs, keys = seen(1 << 40)
    for i in [0] + [i for _ in range(case["loops"]) for i in range(1, case["layers"])]:
        mats = (H * (dim + rot) + r + rot + H) * d + H * (dim + vdim) * r + H * vdim * d
        ffn_b, ffn_f = (2 * d * c["dense"],) * 2 if i == 0 else (3 * d * (hit * ff + c["shared"]), 3 * d * (top * ff + c["shared"]))
        byts += n * 2 * (mats + ffn_b) + keys * 2 * (r + rot)
        flops += 2 * n * T * (mats + ffn_f) + 2 * H * (dim + rot + vdim) * pairs
    return {"bytes": byts, "flops": flops}


# ---- operators alone -----------------------------------------------------------------------------------------

def _linear_inputs(case, seed):
    gen = _gen(_dense_seed(seed, 20))
    w = Weight(gen, case["weights"], case["n"], case["k"], 0.02)
    return w, _randn(gen, case["tokens"], case["k"]).to(DTYPES[case["dtype"]])


def _attention_rows(case, seed, r):
    gen = _gen(_dense_seed(seed, 21, r))
    n = case["ctx"] - (r * 37) % (case["ctx"] // 4 + 1)
    dt = DTYPES[case["dtype"]]
    return _randn(gen, case["heads"], 128).to(dt), _randn(gen, n, case["kv_heads"], 128).to(dt), _randn(gen, n, case["kv_heads"], 128).to(dt)


def prepare(case, seed):
    pkg = import_package()
    if case["family"] == "dense":
        return _prepare_dense(pkg, case, seed)
    if case["family"] in ("tovelix", "vipelix"):
        return _prepare_stack(pkg, case, seed)
    if case["family"] == "linear":
        w, x = _linear_inputs(case, seed)
        return dict(case=case, weight=w.linear(pkg), x=x)
    cache = pkg.KVCache(case["ctx"], case["kv_heads"], 128, case["heads"], batch=case["rows"], dtype=case["kv"])
    qs = []
    for r in range(case["rows"]):
        q, k, v = _attention_rows(case, seed, r)
        cache.append(0, k[None], v[None], row0=r)
        cache.commit(len(k), row0=r, nrows=1)
        qs.append(q)
    return dict(case=case, pkg=pkg, cache=cache, q=torch.stack(qs))


def run(state):
    family = state["case"]["family"]
    if family == "linear":
        return state["weight"](state["x"])
    if family == "attention":
        return state["pkg"].dispatch.attention_decode(state["cache"], state["q"], 128 ** -0.5)
    return _run_model(state)


def exact(case, seed):
    if case["family"] == "dense":
        return _exact_dense(case, seed)
    if case["family"] in ("tovelix", "vipelix"):
        return _exact_stack(case, seed)
    if case["family"] == "linear":
        w, x = _linear_inputs(case, seed)
        return x.double() @ w.dense().T
    out = []
    for r in range(case["rows"]):
        q, k, v = (t.double() for t in _attention_rows(case, seed, r))
        out.append(_attend(q[None], k, v, len(k) - 1, 128 ** -0.5)[0])
    return torch.stack(out)


def work(case):
    if case["family"] == "dense":
        return _work_dense(case)
    if case["family"] in ("tovelix", "vipelix"):
        return _work_stack(case)
    if case["family"] == "linear":
        n, k, t = case["n"], case["k"], case["tokens"]
        return {"bytes": _format_bytes(case["weights"], n, k) + 2 * t * (n + k), "flops": 2 * t * n * k}
    keys = sum(case["ctx"] - (r * 37) % (case["ctx"] // 4 + 1) for r in range(case["rows"]))
    row = 2 * case["kv_heads"] * (132 if case["kv"] == "int8" else 256)
    return {"bytes": keys * row + case["rows"] * case["heads"] * 128 * 4, "flops": 4 * keys * case["heads"] * 128}


def tolerance(case):
    # f32 models sum in another order; a bf16 linear rounds its output once; decoders round every activation to
    # bf16, and which way a rounding falls carries through the layers
    if case.get("dtype") == "f32":
        return {"rel": 1e-5, "max": 1e-3}
    if case["family"] == "linear":
        return {"rel": 4e-3, "max": 2e-2}
    if case["family"] == "attention":
        return {"rel": 8e-3, "max": 5e-2}
    return {"rel": 2.5e-2, "max": 0.3}
