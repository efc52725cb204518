"""Recorded launches of the Q4_K_M GEMM, which leases memory: decode steps of 9 to 40 rows, whose launches are chained, and a linear in
a caller's graph.  Every case runs in a process of its own, so that its first lease is taken while a graph is recorded.  Replayed
steps are compared with the step as plain launches (the same kernels, the attention cut by another bound of the context)."""
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu


def run(rows):
    import torch
    from helpers import pkg
    from model_fixtures import SMALL, build_pair
    cfg = dict(SMALL, d_model=256, ffn_hidden=512, n_heads=4, n_kv_heads=2, head_dim=64)
    gpu, _, _ = build_pair(cfg, "q4_k_m", dtype=torch.bfloat16, max_tokens=64, capacity=8)
    g = torch.Generator().manual_seed(rows)
    ids = torch.randint(0, cfg["vocab"], (4, rows), generator=g, dtype=torch.int32).cuda()
    stepped, plain = (gpu.empty_kv_cache_with_capacity(16, batch=rows, dtype="bf16") for _ in range(2))
    logits = torch.empty((rows, cfg["vocab"]), dtype=torch.bfloat16, device="cuda")
    side, got = torch.cuda.Stream(), []
    torch.cuda.synchronize()
    held = torch.empty_like(ids[0])
    with torch.cuda.stream(side):
        for step in range(4):
            held.copy_(ids[step])
            gpu.decode_step(held, stepped, logits, None)
            got.append(logits.clone())
    torch.cuda.synchronize()
    for step in range(4):
        want = gpu.forward_decode_batch(ids[step][:, None], [step] * rows, plain)[:, 0].double()
        assert float((got[step].double() - want).norm()) < 1e-2 * float(want.norm()), step
    assert pkg().device_status() == 0


def record_a_linear():
    import torch
    from helpers import pkg
    g = torch.Generator(device="cuda").manual_seed(3)
    lin = pkg().QuantLinear.quantise(torch.randn((1024, 1024), generator=g, device="cuda"), "q4_k_m")
    x = torch.randn((40, 1024), generator=g, device="cuda").to(torch.bfloat16)
    graph = torch.cuda.CUDAGraph()
    torch.cuda.synchronize()
    with torch.cuda.graph(graph):
        y = lin(x)
    for _ in range(3):
        graph.replay()
    torch.cuda.synchronize()
    assert torch.equal(y, lin(x)) and pkg().device_status() == 0


@pytest.mark.parametrize("rows", [0, 9, 16, 17, 33, 40])  # 0: the linear
def test_recorded_in_a_new_process(rows):
    r = subprocess.run([sys.executable, os.path.abspath(__file__), str(rows)], capture_output=True, text=True, timeout=200)
    assert r.returncode == 0, r.stdout[-2000:] + r.stderr[-3000:]


if __name__ == "__main__":
    rows = int(sys.argv[1])
    run(rows) if rows else record_a_linear()
