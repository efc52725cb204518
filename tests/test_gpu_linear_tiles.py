"""Linears of many tokens over the reference's formats: the tcgen05 GEMM over Q4_K_M-style blocks (bf16, from 9 tokens
on) and the tiled CUDA-core GEMM (every other format and type from 9 tokens on), against the product with the
dequantised weight in 64 bits.  An f32 sum of n terms is within n 2^-24 of the sum of their magnitudes, a bf16
output within 2^-8 of itself."""
import pytest
import torch

from helpers import pkg

pytestmark = pytest.mark.gpu


def check(lin, x, terms, weight=None):
    """The linear's outputs, within the rounding of `terms` f32 operations, against the product with `weight` (default: its own weights)."""
    y = lin(x).double()
    w = (lin.dequantise() if weight is None else weight).double()
    ref, size = x.double() @ w.T, x.double().abs() @ w.abs().T
    rounding = {torch.float32: 0.0, torch.bfloat16: 2.0 ** -8, torch.float16: 2.0 ** -11}[x.dtype]
    assert torch.isfinite(y).all()
    assert bool(((y - ref).abs() <= rounding * ref.abs() + terms * 2.0 ** -24 * size + 1e-30).all())
    assert pkg().device_status() == 0


# tiles of 128 channels and 32, 64 or 128 tokens, one and several blocks of 256 per row, K split or not (N % 8)
@pytest.mark.parametrize("M", [9, 31, 33, 64, 65, 128, 129, 300])
@pytest.mark.parametrize("N,K", [(128, 256), (7, 512), (1028, 768), (200, 5632), (2048, 2048)])
def test_q4km_many_tokens(M, N, K):
    g = torch.Generator(device="cuda").manual_seed(M + N)
    w = torch.randn((N, K), generator=g, device="cuda") * torch.rand((N, 1), generator=g, device="cuda") + 0.1
    lin = pkg().QuantLinear.quantise(w, "q4_k_m")
    x = (torch.randn((M, K), generator=g, device="cuda") * 3 + 0.5).to(torch.bfloat16)
    # the sums of a block and of its activations are within 256 terms each, the blocks' within K / 256, and the part
    # with the minimum enters beside the codes': both are at most 16 times the sum of the weights' magnitudes here
    check(lin, x, 16 * (512 + K // 256))
    assert torch.equal(lin(x), lin(x))


def test_q4km_many_tokens_streams_and_capture():
    """Two streams at once and a captured call give the bits of a call alone."""
    g = torch.Generator(device="cuda").manual_seed(3)
    lin = pkg().QuantLinear.quantise(torch.randn((1024, 1024), generator=g, device="cuda"), "q4_k_m")
    xs = [torch.randn((40, 1024), generator=g, device="cuda").to(torch.bfloat16) for _ in range(2)]
    alone = [lin(x).clone() for x in xs]
    streams = [torch.cuda.Stream() for _ in xs]
    torch.cuda.synchronize()
    for _ in range(20):
        outs = []
        for x, s in zip(xs, streams):
            with torch.cuda.stream(s):
                outs.append(lin(x))
        torch.cuda.synchronize()
        assert all(torch.equal(o, a) for o, a in zip(outs, alone))
    with torch.cuda.stream(streams[0]):
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph, stream=streams[0]):
            y = lin(xs[0])
        for _ in range(3):
            graph.replay()
    torch.cuda.synchronize()
    assert torch.equal(y, alone[0])


def expected(lin, method, K, M):
    """Weights that a tensor-core linear multiplies, and the f32 operations its outputs may be off by."""
    w = lin.dequantise()
    if method == "w4a16" and M > 64:
        return w.to(torch.bfloat16).float(), 2 * K  # its operand is the rounded weight; up to 64 tokens codes are, and the scale is f32's
    return w, 16 * (512 + K // 256) if method == "q4_k_m" else 2 * K


# tiles of 128 channels and 32, 128, 192 or 256 tokens, their edges; K split or not; rows stored in 16-byte pieces (N % 8 == 0,
# y on a 16-byte boundary) or element by element.
@pytest.mark.parametrize("M", [9, 32, 33, 40, 64, 65, 128, 129, 192, 193, 257, 385, 520, 1100])
@pytest.mark.parametrize("method,N,K", [("w4a16", 256, 512), ("w4a16", 2000, 1024), ("w4a16", 1004, 2048), ("w4a16", 4096, 384),
                                        ("int8_channel", 130, 128), ("int8_channel", 2000, 1024), ("int8_channel", 6144, 256),
                                        ("bf16", 136, 64), ("bf16", 2004, 512), ("bf16", 5120, 256)])
def test_tensor_core_tiles(method, N, K, M):
    g = torch.Generator(device="cuda").manual_seed(M + N)
    w = torch.randn((N, K), generator=g, device="cuda")
    lin = pkg().QuantLinear.from_bf16(w.to(torch.bfloat16)) if method == "bf16" else pkg().QuantLinear.quantise(w, method, 128)
    x = torch.randn((M, K), generator=g, device="cuda").to(torch.bfloat16)
    weight, terms = expected(lin, method, K, M)
    check(lin, x, terms, weight)
    assert torch.equal(lin(x), lin(x))


# tiles of 64 x 64 and 32 x 32 outputs, steps of 32 columns
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16, torch.float16])
@pytest.mark.parametrize("method", ["int8_channel", "int4", "q4_k_m", "w4a16"])
@pytest.mark.parametrize("M,N,K", [(9, 33, 128), (32, 384, 384), (70, 1000, 256), (200, 8192, 384)])
def test_generic_tiles(dtype, method, M, N, K):
    g = torch.Generator(device="cuda").manual_seed(K)
    lin = pkg().QuantLinear.quantise(torch.randn((N, K), generator=g, device="cuda"), method, 64 if method == "w4a16" else 128)
    check(lin, torch.randn((M, K), generator=g, device="cuda").to(dtype), 16 * (K // 32 + 34))


@pytest.mark.parametrize("method", ["int8_channel", "int4"])
def test_generic_tiles_short_rows(method):
    """Rows that end inside a step, and groups that straddle rows."""
    g = torch.Generator(device="cuda").manual_seed(1)
    lin = pkg().QuantLinear.quantise(torch.randn((50, 72), generator=g, device="cuda"), method, 16)
    check(lin, torch.randn((35, 72), generator=g, device="cuda"), 64)


# y need only lie on an element: few tiles, for which a y on 16 bytes would have its K split and reduced in 16-byte pieces, and many
@pytest.mark.parametrize("M", [9, 40, 65, 130, 300])
@pytest.mark.parametrize("method,N,K", [("q4_k_m", 128, 2048), ("q4_k_m", 4096, 512), ("w4a16", 256, 4096), ("w4a16", 4096, 512),
                                        ("int8_channel", 256, 512)])
def test_output_off_a_16_byte_boundary(method, N, K, M):
    g = torch.Generator(device="cuda").manual_seed(M + N)
    p = pkg()
    lin = p.QuantLinear.quantise(torch.randn((N, K), generator=g, device="cuda"), method, 128)
    x = torch.randn((M, K), generator=g, device="cuda").to(torch.bfloat16)
    for off in (1, 4):
        buf = torch.full((M * N + 16,), 7.0, dtype=torch.bfloat16, device="cuda")
        assert buf.data_ptr() % 16 == 0
        y = buf[off:off + M * N].view(M, N)
        p._lib.check(p._lib.lib.ab2_qlinear_forward(lin._h, x.data_ptr(), M, p.qlinear.dtype_code(x.dtype), y.data_ptr(), p.qlinear.stream_ptr()))
        assert bool((buf[:off] == 7).all()) and bool((buf[off + M * N:] == 7).all())
        weight, terms = expected(lin, method, K, M)
        check(lambda _: y, x, terms, weight)


@pytest.mark.parametrize("M", [9, 40, 130])
def test_q4km_codes_cancel_exactly(M):
    """Weights scale * (code - 8) whose products with the activations, small integers, sum to 0 in every block: the part with the minimum and the
    part with the codes have nothing to cancel, and the output is 0 to the last bit.  (scale * sum of codes is 27 bits long.)"""
    scale = 2047 / 2 ** 17  # all 11 bits of an f16
    groups = [(-8, 7, 1)] + [(k, -k) for k in range(1, 8)] * 18 + [(0,)]
    codes = torch.tensor([c for group in groups for c in group])
    assert codes.numel() == 256
    w = (codes.repeat(128, 2) * scale).cuda()
    lin = pkg().QuantLinear.quantise(w, "q4_k_m")
    assert torch.equal(lin.dequantise(), w)
    each = torch.randint(1, 256, (M, 2, len(groups)), generator=torch.Generator().manual_seed(M))
    x = each.repeat_interleave(torch.tensor([len(group) for group in groups]), -1).reshape(M, 512)
    assert bool((x.view(M, 2, 256) * codes).sum(-1).eq(0).all())
    assert bool((lin(x.to(torch.bfloat16).cuda()) == 0).all())


# more tokens than a grid has rows of tiles (65535): blocks of 8 tokens of the Q4_K_M preparation, tiles of 64 of the CUDA-core GEMM
@pytest.mark.parametrize("method,dtype,K,M", [("q4_k_m", torch.bfloat16, 256, 8 * 65535 + 37), ("int8_channel", torch.float32, 8, 64 * 65535 + 100)])
def test_more_tokens_than_rows_of_a_grid(method, dtype, K, M):
    g = torch.Generator(device="cuda").manual_seed(1)
    lin = pkg().QuantLinear.quantise(torch.randn((8, K), generator=g, device="cuda"), method, 128)
    x = torch.randn((M, K), generator=g, device="cuda").to(dtype)
    y = lin(x)
    for part in (slice(0, 200), slice(M - 300, M)):
        check(lambda _: y[part], x[part], 16 * (512 + K // 256), lin.dequantise())
