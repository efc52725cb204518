"""Linears over bf16 weights of 5 to 32 tokens where the decode GEMM's shape changes: clusters of 8, 4 and 2 CTAs a tile, ranges
that cut tiles, whole tiles, K and channels that do not fill theirs, and what a stream without its scratch memory takes."""
import ctypes
import threading

import numpy as np
import pytest
import torch

import vipelix_fixtures as fx
from helpers import pkg

pytestmark = pytest.mark.gpu


def data(N, K, M):
    gen = torch.Generator("cuda").manual_seed(N + K + M)
    w = (torch.randn((N, K), generator=gen, device="cuda") * K ** -0.5).bfloat16()
    x = torch.randn((M, K), generator=gen, device="cuda").bfloat16()
    want = x.double() @ w.double().T
    # one rounding to bf16; f32 sums of K products: at most K roundings of 2^-24 of the sum of magnitudes, in practice its root
    return w, x, want, 2.0 ** -8 * want.abs() + K ** 0.5 * 2.0 ** -23 * (x.double().abs() @ w.double().abs().T)


@pytest.mark.parametrize("N,K,M", [(N, K, M) for N, K in [(1000, 4200), (2048, 2048), (4104, 4096), (74 * 128, 1024), (75 * 128, 1800), (95 * 128 + 8, 1800),
                                                         (12288, 1400), (149 * 128, 1024), (219 * 128 + 40, 640), (250 * 128, 544), (40000, 512), (8200, 8192),
                                                         (1536, 4096), (2560, 2048), (2048, 2560)]
                                   for M in (17, 31, 32)] +
                         [(N, K, M) for N, K in [(1000, 17000), (4096, 4200), (149 * 128, 1024), (9600, 4100 // 8 * 8), (149 * 128, 1400), (7168, 4096), (5120, 4096)]
                          for M in (5, 8, 9, 15, 16)] +
                         [(N, K, M) for N, K in [(4096, 7168), (10240, 4160), (14336, 4096)] for M in (5, 6, 7, 8)])
def test_linear(N, K, M):
    w, x, want, bound = data(N, K, M)
    lin = pkg().QuantLinear.from_bf16(w)
    got = lin(x)
    assert ((got.double() - want).abs() <= bound).all()
    for _ in range(3):  # contributors are added in one order, whatever the order they arrive in
        assert torch.equal(lin(x), got)
    assert pkg().device_status() == 0


@pytest.mark.parametrize("N,K", [(2048, 2560), (149 * 128, 1024), (250 * 128, 544)])
def test_rows_that_are_not_finite_stay_alone(N, K):
    w, x, want, bound = data(N, K, 32)
    x[3], x[31, 5] = float("nan"), float("inf")
    got = pkg().QuantLinear.from_bf16(w)(x).double()
    rest = [r for r in range(32) if r not in (3, 31)]
    assert got[3].isnan().all() and not got[31].isfinite().any()
    assert ((got[rest] - want[rest]).abs() <= bound[rest]).all()


@pytest.mark.parametrize("N,K", [(2048, 2560), (149 * 128, 1024), (250 * 128, 544)])
def test_recorded_and_on_several_streams(N, K):
    """A recorded call replays beside eager calls on the stream it was recorded on; streams have parts of their own."""
    w, x, want, bound = data(N, K, 32)
    lin = pkg().QuantLinear.from_bf16(w)
    streams = [torch.cuda.Stream() for _ in range(3)]
    torch.cuda.synchronize()
    with torch.cuda.stream(streams[0]):
        lin(x)
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph, stream=streams[0]):
            recorded = lin(x)
    torch.cuda.synchronize()
    outs = []
    for _ in range(20):
        with torch.cuda.stream(streams[1]):
            graph.replay()
        for s in (streams[0], streams[2]):
            with torch.cuda.stream(s):
                outs.append(lin(x))
    torch.cuda.synchronize()
    for got in outs + [recorded]:
        assert ((got.double() - want).abs() <= bound).all()
        assert torch.equal(got, outs[0])  # recorded or not, one kernel


def test_a_stream_handle_that_is_used_again():
    """A stream with launches still to run is destroyed, and another may get its handle."""
    w, x, want, bound = data(149 * 128, 1024, 32)
    lin, lib, cudart = pkg().QuantLinear.from_bf16(w), pkg()._lib.lib, ctypes.CDLL("libcudart.so.12")
    eager = lin(x)
    outs = [torch.full_like(eager, float("nan")) for _ in range(6)]
    side, event, codes = torch.cuda.Stream(), torch.cuda.Event(), []
    torch.cuda.synchronize()
    for out in outs:
        stream = ctypes.c_void_p()
        codes.append(cudart.cudaStreamCreateWithFlags(ctypes.byref(stream), 1))
        codes.append(lib.ab2_qlinear_forward(lin._h, x.data_ptr(), 32, 2, out.data_ptr(), stream))
        if out is outs[0]:
            with torch.cuda.stream(side):
                torch.cuda._sleep(100_000_000)
                event.record()
        codes.append(cudart.cudaStreamWaitEvent(stream, ctypes.c_void_p(event.cuda_event), 0))
        codes.append(lib.ab2_qlinear_forward(lin._h, x.data_ptr(), 32, 2, out.data_ptr(), stream))
        codes.append(cudart.cudaStreamDestroy(stream))
    torch.cuda.synchronize()
    assert not any(codes) and all(torch.equal(out, eager) for out in outs)


@pytest.mark.parametrize("N,K", [(149 * 128, 1024), (80 * 128, 1800)])
def test_per_thread_stream(N, K):
    """Cut tiles on the stream whose handle every thread shares: parts are leased for each launch."""
    w, x, want, bound = data(N, K, 32)
    lin = pkg().QuantLinear.from_bf16(w)
    eager = lin(x)
    torch.cuda.synchronize()
    outs = [torch.full((32, N), float("nan"), device="cuda", dtype=torch.bfloat16) for _ in range(8)]
    torch.cuda.synchronize()
    lib, codes = pkg()._lib.lib, []

    def work(mine):
        for out in mine:
            codes.append(lib.ab2_qlinear_forward(lin._h, x.data_ptr(), 32, 2, out.data_ptr(), ctypes.c_void_p(2)))

    threads = [threading.Thread(target=work, args=(outs[i::2],)) for i in range(2)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    torch.cuda.synchronize()
    assert codes == [0] * 8 and all(torch.equal(out, eager) for out in outs)


def test_gated_unit_and_capped_head_of_a_stack(tmp_path):
    """A latent stack whose shared expert, projections and head are wide enough, 20 rows a step."""
    vocab = 9640
    cfg = fx.config([(fx.latent(8, 64, 32, 64, 128), fx.dense(4096)), (fx.latent(8, 64, 32, 64, 128), fx.moe(4, 2, 256, 4104))], width=1024, vocab=vocab, loop=None)
    w = fx.weights(cfg, 5)
    model = fx.load(tmp_path, cfg, w, torch.bfloat16, 64, 16)
    tokens = np.random.default_rng(3).integers(0, vocab, (20, 4))

    def steps(rows):
        cache = model.empty_kv_cache_with_capacity(16, batch=len(rows))
        logits = torch.empty((len(rows), 1, vocab), device="cuda", dtype=model.logits_dtype)
        out = []
        with torch.cuda.stream(torch.cuda.Stream()):
            for i in range(4):
                model.decode_step(torch.from_numpy(tokens[rows, i].astype(np.int32)).cuda(), cache, logits, None)
                out.append(logits[:, 0].double().cpu().numpy())
        return np.stack(out, 1)

    got = steps(list(range(20)))
    for r in (0, 7, 19):
        want = fx.expected(cfg, w, tokens[r].tolist())
        many, one = (np.linalg.norm(x - want) / np.linalg.norm(want) for x in (got[r], steps([r])[0]))
        # the roundings of activations to bf16, which both have, fall differently: the GEMV's error is the measure
        assert many < 1.3 * one + 1e-3 and one < 3e-2, (many, one)
    assert pkg().device_status() == 0


@pytest.mark.parametrize("ff,rows", [(149 * 128 + 8, 17), (149 * 128 + 8, 32), (149 * 128 + 8, 9), (12800, 20), (80 * 128, 31), (66 * 128 - 8, 12)])
def test_gated_unit_over_cut_and_whole_tiles(tmp_path, ff, rows):
    """The gate and up products of a dense feed-forward in every form of more tiles than a cluster serves (and one that it does).  Rows
    hold the same tokens, so that each has to be the others' equal to the bit."""
    vocab = 512
    cfg = fx.config([(fx.latent(8, 64, 32, 64, 128), fx.dense(ff))], width=1032, vocab=vocab, loop=None)
    w = fx.weights(cfg, ff)
    model = fx.load(tmp_path, cfg, w, torch.bfloat16, 64, 16)
    tokens = np.random.default_rng(rows).integers(0, vocab, 3)

    def steps(n):
        cache = model.empty_kv_cache_with_capacity(16, batch=n)
        logits = torch.empty((n, 1, vocab), device="cuda", dtype=model.logits_dtype)
        out = []
        with torch.cuda.stream(torch.cuda.Stream()):
            for t in tokens:
                model.decode_step(torch.full((n,), int(t), dtype=torch.int32, device="cuda"), cache, logits, None)
                out.append(logits[:, 0].clone())
        torch.cuda.synchronize()
        return torch.stack(out, 1)

    got = steps(rows)
    assert torch.equal(got, got[:1].expand_as(got)) and torch.equal(steps(rows), got)
    want = fx.expected(cfg, w, tokens.tolist())
    many, one = (np.linalg.norm(x[0].double().cpu().numpy() - want) / np.linalg.norm(want) for x in (got, steps(1)))
    assert many < 1.3 * one + 1e-3 and one < 3e-2, (many, one)  # as above
    assert pkg().device_status() == 0
