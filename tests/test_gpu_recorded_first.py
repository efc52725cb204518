"""A call that is the first of its kind in the process may be one that is recorded into a graph: nothing it needs is allocated then.  Each
runs in a process of its own."""
import os
import subprocess
import sys

import pytest

from helpers import ROOT

pytestmark = pytest.mark.gpu

HEAD = """
import torch
from helpers import pkg
p, stream, graph, same = pkg(), torch.cuda.Stream(), torch.cuda.CUDAGraph(), True
gen = torch.Generator("cuda").manual_seed(1)
randn = lambda *s: torch.randn(s, generator=gen, device="cuda").bfloat16()

def check(call, want):
    torch.cuda.synchronize()
    with torch.cuda.graph(graph, stream=stream):
        got = call()
    graph.replay()
    torch.cuda.synchronize()
    assert float((got.double() - want).norm()) <= 2.0 ** -8 * float(want.norm())
    assert torch.equal(call(), got) or not same  # recorded or not, one kernel
    assert p.device_status() == 0
"""
ATTENTION = """
cache = p.KVCache({n} + 4, 4, 128, 8, batch=2, dtype="{kv}")
k, v, q = randn(2, {n}, 4, 128), randn(2, {n}, 4, 128), randn(2, 8, 128)
cache.append(0, k, v)
cache.commit({n})
if "{kv}" == "int8":
    k, v = (torch.stack(t) for t in zip(cache.read(0), cache.read(1)))
k, v = (t.double().repeat_interleave(2, 2) for t in (k, v))
w = torch.softmax(torch.einsum("bhd,bnhd->bhn", q.double(), k) * 128 ** -0.5, -1)
check(lambda: p.dispatch.attention_decode(cache, q, 128 ** -0.5), torch.einsum("bhn,bnhd->bhd", w, v))
"""
LINEAR = """
w, x = randn({N}, {K}) * {K} ** -0.5, randn({M}, {K})
lin = p.QuantLinear.from_bf16(w.contiguous())
check(lambda: lin(x), x.double() @ w.double().T)
"""


def alone(code, **more):
    env = dict(os.environ, PYTHONPATH=os.path.join(ROOT, "tests"), **more)
    r = subprocess.run([sys.executable, "-c", HEAD + code], cwd=ROOT, env=env, capture_output=True, text=True, timeout=120)
    assert r.returncode == 0, r.stdout[-2000:] + r.stderr[-3000:]


@pytest.mark.parametrize("kv,n", [("bf16", 300), ("int8", 3000)])
def test_decode_attention(kv, n):
    alone(ATTENTION.format(kv=kv, n=n))


@pytest.mark.parametrize("N,K,M", [(2560, 2048, 20), (250 * 128, 1024, 32), (149 * 128, 1024, 32), (80 * 128, 4096, 9), (4096, 4096, 300)])
def test_bf16_linears(N, K, M):
    alone(LINEAR.format(N=N, K=K, M=M))


def test_refused_scratch_while_recording():
    alone("same = False" + LINEAR.format(N=149 * 128, K=1024, M=32), AB2_SCRATCH_MAX_BYTES="0")
