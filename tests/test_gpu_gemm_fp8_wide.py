"""The 128 x 256 tiles of the fp8 product: sizes whose wave counts choose them, remainders of rows and columns, both scale forms,
against fp64 products.  Bound: half a bf16 ulp and fp32 sums of K terms."""
import pytest
import torch

from vllm_ascend_b200 import _native
from vllm_ascend_b200.quantization import schemes

pytestmark = pytest.mark.gpu
DEV = "cuda"


def _fp8(*shape, g):
    return (torch.randn(*shape, device=DEV, generator=g) * 60).clamp(-448, 448).to(torch.float8_e4m3fn)


@pytest.mark.parametrize("M,N,K", [(300, 32000, 256), (1000, 8200, 384), (2048, 10240, 128), (129, 57344, 640)])
def test_block_scales(M, N, K):
    g = torch.Generator(device=DEV).manual_seed(N)
    a, w = _fp8(M, K, g=g), _fp8(N, K, g=g)
    sa = torch.rand(M, K // 128, device=DEV, generator=g) * 0.02 + 0.001
    sw = torch.rand((N + 127) // 128, K // 128, device=DEV, generator=g) * 1e-3 + 1e-4
    out = schemes.fp8_block_linear(None, w, sw, quant=(a, sa))
    ad = a.double() * sa.double().repeat_interleave(128, 1)
    wd = w.double() * sw.double().repeat_interleave(128, 0)[:N].repeat_interleave(128, 1)
    want, absum = ad @ wd.t(), ad.abs() @ wd.abs().t()
    assert ((out.double() - want).abs() <= want.abs() * 2.0 ** -8 + absum * (8 * 2.0 ** -24 * K ** 0.5) + 1e-6).all()
    _native.check_status(torch.device(DEV))


def test_channel_scales():
    M, N, K = 300, 32008, 256
    g = torch.Generator(device=DEV).manual_seed(1)
    x = torch.randn(M, K, device=DEV, generator=g).bfloat16()
    w, sw = _fp8(N, K, g=g), torch.rand(N, device=DEV, generator=g) * 1e-3
    bias = torch.randn(N, device=DEV, generator=g).bfloat16()
    out = schemes.fp8_channel_linear(x, w, sw, bias)
    from vllm_ascend_b200 import ops
    q, s = ops.quant_fp8_per_token(x)
    ad, wd = q.double() * s.double().view(-1, 1), w.double() * sw.double().view(-1, 1)
    want = ad @ wd.t() + bias.double()
    assert ((out.double() - want).abs() <= want.abs() * 2.0 ** -8 + (ad.abs() @ wd.abs().t() + 4) * (8 * 2.0 ** -24 * K ** 0.5) + 1e-6).all()
    _native.check_status(torch.device(DEV))
