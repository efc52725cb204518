"""Cutting a row does not wait for the GPU: it takes its place in its stream, and calls on the cache from other streams come after it."""
import ctypes
import threading

import pytest
import torch

from helpers import pkg

pytestmark = pytest.mark.gpu


def filled(rows, n):
    gen = torch.Generator(device="cuda").manual_seed(n)
    cache = pkg().KVCache(n + 8, 2, 128, 4, batch=rows, dtype="bf16")
    k, v = (torch.randn((rows, n, 2, 128), generator=gen, device="cuda").bfloat16() for _ in range(2))
    cache.append(0, k, v)
    cache.commit(n, row0=0, nrows=rows)
    return cache, k, v


def test_a_cut_takes_its_place_in_the_stream():
    cache, k, _ = filled(3, 40)
    side = torch.cuda.Stream()
    torch.cuda.synchronize()
    with torch.cuda.stream(side):
        torch.cuda._sleep(200_000_000)       # the cut below is still to come when the call returns
        cache.truncate(7, 1)
    assert cache.seq_len(1) == 7 and not side.query()
    new = torch.ones((1, 1, 2, 128), device="cuda", dtype=torch.bfloat16)
    cache.append(0, new, new, row0=1)        # another stream: after the cut
    cache.commit(1, row0=1, nrows=1)
    got = cache.read(1)[0]
    assert got.shape[0] == 8 and torch.equal(got[:7].bfloat16(), k[1, :7]) and (got[7] == 1).all()
    q = torch.randn((3, 4, 128), device="cuda", dtype=torch.bfloat16)
    assert torch.isfinite(pkg().dispatch.attention_decode(cache, q, 0.1).float()).all()
    assert [cache.seq_len(r) for r in range(3)] == [40, 8, 40]


def test_many_cuts_in_a_row():
    cache, k, _ = filled(33, 50)
    for n in (49, 20, 3):
        for r in range(33):
            cache.truncate(n if r % 2 else 50 if n == 49 else n + 1, r)
    for r in (0, 1, 32):
        n = 3 if r % 2 else 4
        assert torch.equal(cache.read(r)[0].bfloat16(), k[r, :n])


def row_after_a_cut(cache, k, row=0):
    """The row was cut to 7 tokens and given a token of ones behind them."""
    got = cache.read(row)[0]
    assert got.shape[0] == 8 and torch.equal(got[:7].bfloat16(), k[row, :7]) and (got[7] == 1).all()


def ones():
    new = torch.ones((1, 1, 2, 128), device="cuda", dtype=torch.bfloat16)
    torch.cuda.synchronize()
    return new


def busy_event():
    """An event that is reached in about 0.1 s."""
    side, event = torch.cuda.Stream(), torch.cuda.Event()
    with torch.cuda.stream(side):
        torch.cuda._sleep(200_000_000)
        event.record()
    return event


def test_the_per_thread_stream_of_two_threads():
    """One handle, two streams: a cut by one thread, then an append by another."""
    lib, cudart, per_thread = pkg()._lib.lib, ctypes.CDLL("libcudart.so.12"), ctypes.c_void_p(2)
    cache, k, _ = filled(1, 40)
    new, event = ones(), busy_event()
    cut, done, codes = threading.Event(), threading.Event(), []

    def first():
        codes.append(cudart.cudaStreamWaitEvent(per_thread, ctypes.c_void_p(event.cuda_event), 0))
        codes.append(lib.ab2_kv_truncate(cache._h, 0, 7, per_thread))
        cut.set()
        done.wait(60)

    def second():
        cut.wait(60)
        codes.append(lib.ab2_kv_append(cache._h, 0, new.data_ptr(), new.data_ptr(), 1, 0, 1, 2, None, None, None, 0, per_thread))
        codes.append(lib.ab2_kv_commit(cache._h, 1, 0, 1, per_thread))
        done.set()

    threads = [threading.Thread(target=f) for f in (first, second)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    torch.cuda.synchronize()
    assert codes == [0, 0, 0, 0]
    row_after_a_cut(cache, k)


def test_a_handle_that_is_used_again():
    """The cut's stream is destroyed while the cut is still to come; a new stream may get its handle."""
    lib, cudart = pkg()._lib.lib, ctypes.CDLL("libcudart.so.12")
    cache, k, _ = filled(1, 40)
    new, event = ones(), busy_event()
    streams = [ctypes.c_void_p() for _ in range(9)]
    codes = [cudart.cudaStreamCreateWithFlags(ctypes.byref(streams[0]), 1), cudart.cudaStreamWaitEvent(streams[0], ctypes.c_void_p(event.cuda_event), 0),
             lib.ab2_kv_truncate(cache._h, 0, 7, streams[0]), cudart.cudaStreamDestroy(streams[0])]
    codes += [cudart.cudaStreamCreateWithFlags(ctypes.byref(s), 1) for s in streams[1:]]
    again = next((s for s in streams[1:] if s.value == streams[0].value), streams[1])
    codes.append(lib.ab2_kv_append(cache._h, 0, new.data_ptr(), new.data_ptr(), 1, 0, 1, 2, None, None, None, 0, again))
    codes.append(lib.ab2_kv_commit(cache._h, 1, 0, 1, again))
    torch.cuda.synchronize()
    codes += [cudart.cudaStreamDestroy(s) for s in streams[1:]]
    assert not any(codes)
    row_after_a_cut(cache, k)


def recorded_append(cache, new, stream):
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.stream(stream):
        graph.capture_begin(capture_error_mode="thread_local")
        cache.append(0, new, new, row0=0)
        graph.capture_end()
    return graph


def test_a_recording_after_a_cut():
    """Recorded on the cut's own stream while the cut is still to come, launched on another."""
    cache, k, _ = filled(1, 40)
    new, side, other = ones(), torch.cuda.Stream(), torch.cuda.Stream()
    with torch.cuda.stream(side):
        torch.cuda._sleep(200_000_000)
        cache.truncate(7, 0)
    graph = recorded_append(cache, new, side)
    with torch.cuda.stream(other):
        graph.replay()
        cache.commit(1, row0=0, nrows=1)
    torch.cuda.synchronize()
    row_after_a_cut(cache, k)


def test_a_cut_after_a_recording():
    """A graph recorded ahead of the cut and launched after it, on another stream."""
    cache, k, _ = filled(1, 40)
    new, side, other = ones(), torch.cuda.Stream(), torch.cuda.Stream()
    graph = recorded_append(cache, new, other)
    with torch.cuda.stream(side):
        torch.cuda._sleep(200_000_000)
        cache.truncate(7, 0)
    with torch.cuda.stream(other):
        graph.replay()
        cache.commit(1, row0=0, nrows=1)
    torch.cuda.synchronize()
    row_after_a_cut(cache, k)
