"""Block scales of the fp8 product in shared memory, eight K blocks at a time: last groups of one to eight blocks, rows of scales that
take 16-byte loads (a multiple of four blocks) and others, scales that start off 16 bytes, both tile widths and groups of rows."""
import pytest
import torch

from vllm_ascend_b200 import _native
from vllm_ascend_b200.quantization import schemes

pytestmark = pytest.mark.gpu
DEV = "cuda"


def _case(M, N, K, shift, seed):
    g = torch.Generator(device=DEV).manual_seed(seed)
    a, w = ((torch.randn(n, K, device=DEV, generator=g) * 60).clamp(-448, 448).to(torch.float8_e4m3fn) for n in (M, N))
    sa = torch.empty(M * (K // 128) + shift, device=DEV)[shift:].view(M, K // 128)
    sa.copy_(torch.rand(M, K // 128, device=DEV, generator=g) * 0.02 + 0.001)
    sw = torch.rand((N + 127) // 128, K // 128, device=DEV, generator=g) * 1e-3 + 1e-4
    out = schemes.fp8_block_linear(None, w, sw, quant=(a, sa))
    _native.check_status(torch.device(DEV))
    ad, wd = a.double() * sa.double().repeat_interleave(128, 1), w.double() * sw.double().repeat_interleave(128, 0)[:N].repeat_interleave(128, 1)
    want, absum = ad @ wd.t(), ad.abs() @ wd.abs().t()
    # half a bf16 ulp and fp32 sums of K terms
    assert ((out.double() - want).abs() <= want.abs() * 2.0 ** -8 + absum * (8 * 2.0 ** -24 * K ** 0.5) + 1e-6).all()


@pytest.mark.parametrize("M,N", [(300, 32000), (130, 264)])            # tiles of 256 columns over several waves, of 128 in one
@pytest.mark.parametrize("blocks", [1, 4, 7, 8, 9, 12, 16, 17])
@pytest.mark.parametrize("shift", [0, 1])
def test_groups_of_scales(M, N, blocks, shift):
    _case(M, N, blocks * 128, shift, 10 * blocks + shift)
