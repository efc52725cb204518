"""bf16 GEMMs of many tokens on pairs of CTAs, at the edges of their tiles: 256 channels x 256 tokens (gate and up products: 128), a
second CTA without channels, K that ends inside a stage, experts with more and fewer rows than a tile."""
import numpy as np
import pytest
import torch

import vipelix_fixtures as fx
from helpers import pkg

pytestmark = pytest.mark.gpu


# short K by single CTAs, and by pairs where there are rounds enough
@pytest.mark.parametrize("N,K,M", [(N, K, M) for N, K in [(74 * 256, 1024), (75 * 256 - 128, 1000), (75 * 256 - 120, 200), (38 * 256 + 8, 64)]
                                   for M in (257, 400, 512, 513, 800)] +
                         [(74 * 256, 4096, 257), (75 * 256 - 128, 4104, 513), (38 * 256 + 8, 4200, 400), (75 * 256 - 120, 1000, 801), (74 * 256 - 8, 200, 4100), (74 * 256, 136, 5890)])
def test_linear(N, K, M):
    gen = torch.Generator("cuda").manual_seed(N + K + M)
    w = (torch.randn((N, K), generator=gen, device="cuda") * K ** -0.5).bfloat16()
    x = torch.randn((M, K), generator=gen, device="cuda").bfloat16()
    want = x.double() @ w.double().T
    # one rounding to bf16; f32 sums of K products: at most K roundings of 2^-24 of the sum of magnitudes, in practice its root
    bound = 2.0 ** -8 * want.abs() + K ** 0.5 * 2.0 ** -23 * (x.double().abs() @ w.double().abs().T)
    lin = pkg().QuantLinear.from_bf16(w)
    for _ in range(3):
        assert ((lin(x).double() - want).abs() <= bound).all()
    assert pkg().device_status() == 0


@pytest.mark.parametrize("E,top,ff,d,T", [(16, 2, 1024, 1024, 2000), (5, 1, 2184, 2056, 1500), (40, 4, 520, 520, 1100)])
def test_experts(E, top, ff, d, T):
    p = pkg()
    gen = torch.Generator("cuda").manual_seed(E + T)
    w = {n: (torch.randn(s, generator=gen, device="cuda") * s[1] ** -0.5).bfloat16() for n, s in
         {"r": (E, d), "g": (E * ff, d), "u": (E * ff, d), "d": (E * d, ff)}.items()}
    x = torch.randn((T, d), generator=gen, device="cuda").bfloat16()
    limit = 0.8
    got = p.dispatch.MoeExperts(p.MoeFfn(E, top, ff, limit), *(p.QuantLinear.from_bf16(w[n]) for n in "rgud"))(x).double()
    z = x.double() @ w["r"].double().T
    score, chosen = torch.sigmoid(z).topk(top, 1)
    # f32 sums may turn two experts whose logits are this close around
    order = z.sort(1, descending=True).values
    clear = (order[:, :top] - order[:, 1:top + 1] > 1e-4).all(1)
    assert clear.float().mean() > 0.9
    for e in range(E):
        t, s = ((chosen == e) & clear[:, None]).nonzero(as_tuple=True)
        h = x[t].double() * score[t, s][:, None]
        gate = (h @ w["g"][e * ff:(e + 1) * ff].double().T).clamp_max(limit)
        up = (h @ w["u"][e * ff:(e + 1) * ff].double().T).clamp(-limit, limit)
        want = (gate * torch.sigmoid(1.702 * gate) * (up + 1)) @ w["d"][e * d:(e + 1) * d].double().T
        # the gated unit is rounded to bf16 once: 2^-9 of each term of the sum, whose errors add up as their root
        assert (got[t, s] - want).norm() <= 2.0 ** -8 * want.norm()
    assert p.device_status() == 0


def test_shared_expert_of_a_prompt(tmp_path):
    """A latent stack whose shared expert's gate and up products and head of every token run on pairs."""
    vocab = 9600
    cfg = fx.config([(fx.latent(8, 64, 32, 64, 128), fx.moe(4, 2, 256, 9480))], width=512, vocab=vocab, loop=None)
    w = fx.weights(cfg, 7)
    model = fx.load(tmp_path, cfg, w, torch.bfloat16, 400, 400)
    tokens = np.random.default_rng(4).integers(0, vocab, 400)
    cache = model.empty_kv_cache_with_capacity(400, batch=1)
    got = model.forward_with_cache(torch.from_numpy(tokens)[None], 0, cache, row=0, last_only=False).double().cpu().numpy().reshape(400, vocab)
    want = fx.expected(cfg, w, tokens.tolist())
    assert np.linalg.norm(got - want) < 2e-2 * np.linalg.norm(want)
    assert pkg().device_status() == 0


def test_many_launches_of_pairs():
    """Launch after launch: CTAs of one come and go while others of their pairs still set up or give back tensor memory."""
    lins = [pkg().QuantLinear.from_bf16((torch.randn((n, k), device="cuda") * k ** -0.5).bfloat16()) for n, k in ((74 * 256, 256), (38 * 256 + 8, 1000))]
    xs = [torch.randn((m, lin.in_features), device="cuda").bfloat16() for lin, m in zip(lins, (4096, 2600))]
    first = [lin(x) for lin, x in zip(lins, xs)]
    stream = torch.cuda.Stream()
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=stream):
        for _ in range(50):
            got = [lin(x) for lin, x in zip(lins, xs)]
    for _ in range(100):
        graph.replay()
    torch.cuda.synchronize()
    assert all(torch.equal(a, b) for a, b in zip(got, first)) and pkg().device_status() == 0
