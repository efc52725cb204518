"""A prompt of one row of which only the last logits are wanted runs the rest of the last layer, after its attention,
on the last token: its logits are those of the prompt with all logits kept (f32: to sums in another order, 2^-24 a term
over 6 layers of at most 1024 terms), and the cache holds the same keys and values."""
import importlib

import numpy as np
import pytest
import torch

from model_fixtures import TINY, build_pair

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("method", ["int8_channel", "q4_k_m"])
@pytest.mark.parametrize("before,S", [(0, 2), (0, 9), (5, 17), (0, 64), (1, 63)])
def test_last_token_alone(method, before, S):
    gpu, _, _ = build_pair(TINY, method, max_tokens=64)
    ids = np.random.default_rng(S).integers(0, TINY["vocab"], (1, before + S))
    caches = [gpu.empty_kv_cache_with_capacity(160) for _ in range(2)]
    outs = []
    for cache, last in zip(caches, (True, False)):
        if before:
            gpu.forward_with_cache(ids[:, :before], 0, cache)
        outs.append(gpu.forward_with_cache(ids[:, before:], before, cache, last_only=last).double())
    assert outs[0].shape == (1, 1, TINY["vocab"])
    assert float((outs[0][0, 0] - outs[1][0, -1]).norm()) <= 6 * 1024 * 2.0 ** -24 * float(outs[1][0, -1].norm())
    for layer in range(gpu.cfg.n_layers):
        for a, b in zip(caches[0].read(0, layer), caches[1].read(0, layer)):
            assert torch.equal(a, b)


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("family,stack", [("tovelix", "VARIED"), ("tovelix", "STEADY"), ("vipelix", "VARIED"), ("vipelix", "ROUND"), ("vipelix", "PLAIN")])
@pytest.mark.parametrize("before,S", [(0, 2), (0, 70), (6, 33)])
def test_last_token_alone_in_stacks(tmp_path, family, stack, dtype, before, S):
    """The same for layer stacks; bf16 rounds what the sublayers read, where other sums may fall on the other side."""
    fx = importlib.import_module(family + "_fixtures")
    cfg = getattr(fx, stack)
    model = fx.load(str(tmp_path), cfg, fx.weights(cfg), dtype)
    ids = np.random.default_rng(S).integers(0, cfg["vocab"] if isinstance(cfg, dict) else cfg.vocab, (1, before + S))
    outs = []
    for last in (True, False):
        cache = model.empty_kv_cache_with_capacity(160)
        if before:
            model.forward_with_cache(ids[:, :before], 0, cache)
        outs.append(model.forward_with_cache(ids[:, before:], before, cache, last_only=last).double())
    limit = 1e-4 if dtype == torch.float32 else 2e-2
    assert float((outs[0][0, 0] - outs[1][0, -1]).norm()) <= limit * float(outs[1][0, -1].norm())
