"""The W4A16 decode GEMM (9 to 64 tokens) where its shape changes: token counts at the edges of 16, 32 and 64, channel tiles with
CTAs of their own and equal shares of the units, one group, rows that do not fill a tile, results off 16-byte boundaries."""
import numpy as np
import pytest
import torch

from helpers import make_w4a16, pack_w4, pkg
from oracle import oracle as orc

pytestmark = pytest.mark.gpu


def linear(weight, x, N, offset):
    """x . W^T by the C entry, the result `offset` elements off a 256-byte boundary."""
    y = torch.full((x.shape[0] * N + offset + 64,), 7.0, device="cuda", dtype=torch.bfloat16)
    out = y[offset:offset + x.shape[0] * N]
    q = pkg().qlinear
    q.check(q.lib.ab2_qlinear_forward(weight._h, x.data_ptr(), x.shape[0], q.dtype_code(x.dtype), out.data_ptr(), q.stream_ptr()))
    assert (y[:offset] == 7).all() and (y[offset + x.shape[0] * N:] == 7).all()
    return out.view(x.shape[0], N)


# tiles x groups: four CTAs a tile, shares that cut tiles (more tiles than SMs; long K over few tiles), whole tiles, one group, remainders
@pytest.mark.parametrize("N,K", [(4096, 4096), (148 * 128 + 16, 640), (2560, 4096), (14336, 512), (384, 128), (40, 1152), (3000, 1536)])
@pytest.mark.parametrize("M", [9, 16, 17, 32, 33, 48, 64, 65])
def test_linear(N, K, M):
    rng = np.random.default_rng(N + K + M)
    weight = pkg().QuantLinear.from_w4a16_gptq(*make_w4a16(rng, N, K), N, K, 128)
    x = torch.randn((M, K), generator=torch.Generator("cuda").manual_seed(M), device="cuda").bfloat16()
    dense = weight.dequantise(torch.float32).double()
    want = x.double() @ dense.T
    # one rounding to bf16; f32 sums of K products: at most K roundings of 2^-24 of the sum of magnitudes, in practice its root
    bound = 2.0 ** -8 * want.abs() + K ** 0.5 * 2.0 ** -23 * (x.double().abs() @ dense.abs().T)
    if M > 64:  # the GEMM of many tokens rounds every weight to bf16
        bound += 2.0 ** -8 * (x.double().abs() @ dense.abs().T)
    for offset in (0, 1, 8):
        assert ((linear(weight, x, N, offset).double() - want).abs() <= bound).all()


@pytest.mark.parametrize("M", [9, 40])
def test_every_code_and_zero_point(M):
    """A token of one element 1 has the weight itself, rounded once, as its result: exact for all pairs of code and zero point."""
    N, K = 256, 256
    codes = np.arange(N * K, dtype=np.uint32).reshape(N, K) * 7 // 3 % 16
    zeros = (np.arange(N * 2).reshape(N, 2) % 16).astype(np.uint32)
    scales = orc.bf16_bits(np.random.default_rng(1).uniform(0.005, 0.02, (N, 2)).astype(np.float32))
    weight = pkg().QuantLinear.from_w4a16_gptq(pack_w4(codes), scales, pack_w4(zeros), N, K, 128)
    dense = weight.dequantise(torch.float32)
    for k0 in range(0, K, M):
        n = min(M, K - k0)
        x = torch.zeros((M, K), device="cuda", dtype=torch.bfloat16)
        x[torch.arange(n), k0 + torch.arange(n)] = 1
        assert torch.equal(linear(weight, x, N, 0)[:n], dense[:, k0:k0 + n].T.bfloat16())
