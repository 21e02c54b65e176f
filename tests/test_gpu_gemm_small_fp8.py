"""Few-row block-scaled fp8 GEMM: every accumulator width, remainders of its tiles, splits and K blocks (more than one stage of
scales), against fp64 products of the same fp8 values.  Bound: half a bf16 ulp of the result and fp32 sums, as for the bf16 form."""
import pytest
import torch

from vllm_ascend_b200 import _native
from vllm_ascend_b200.quantization import schemes

pytestmark = pytest.mark.gpu
DEV = "cuda"


def _make(M, N, K, seed):
    g = torch.Generator(device=DEV).manual_seed(seed)
    a = (torch.randn(M, K, device=DEV, generator=g) * 60).clamp(-448, 448).to(torch.float8_e4m3fn)
    w = (torch.randn(N, K, device=DEV, generator=g) * 60).clamp(-448, 448).to(torch.float8_e4m3fn)
    sa = torch.rand(M, K // 128, device=DEV, generator=g) * 0.02 + 0.001
    sw = torch.rand((N + 127) // 128, K // 128, device=DEV, generator=g) * 1e-3 + 1e-4
    ad = a.double() * sa.double().repeat_interleave(128, 1)
    wd = w.double() * sw.double().repeat_interleave(128, 0)[:N].repeat_interleave(128, 1)
    return a, w, sa, sw, ad, wd


def _check(out, want, absum, K):
    assert ((out.double() - want).abs() <= want.abs() * 2.0 ** -8 + absum * (8 * 2.0 ** -24 * K ** 0.5) + 1e-6).all()


@pytest.mark.parametrize("M,N,K", [(1, 128, 128), (1, 4096, 4096), (17, 200, 2048), (32, 1024, 8192), (33, 136, 1152), (64, 640, 5120),
                                   (65, 128, 2176), (128, 1536, 4096), (100, 32000, 2048)])
def test_against_fp64(M, N, K):
    a, w, sa, sw, ad, wd = _make(M, N, K, M + N)
    bias = torch.randn(N, device=DEV).bfloat16()
    out = schemes.fp8_block_linear(None, w, sw, bias, quant=(a, sa))
    _check(out, ad @ wd.t() + bias.double(), ad.abs() @ wd.abs().t() + 4, K)
    assert torch.equal(out, schemes.fp8_block_linear(None, w, sw, bias, quant=(a, sa)))
    _native.check_status(torch.device(DEV))


@pytest.mark.parametrize("M", [5, 50, 128])
@pytest.mark.parametrize("splits", [1, 3, 8])
def test_every_split(M, splits):
    N, K = 264, 41 * 128
    a, w, sa, sw, ad, wd = _make(M, N, K, splits)
    out = torch.full((M, N), float("nan"), device=DEV, dtype=torch.bfloat16)
    _native.check(_native.lib().b200_gemm_small_fp8(
        a.data_ptr(), sa.data_ptr(), w.data_ptr(), sw.data_ptr(), out.data_ptr(), None, M, N, K, K, K, N, splits,
        _native.status_word(a.device).data_ptr(), _native.stream_ptr()), "gemm_small_fp8")
    _check(out, ad @ wd.t(), ad.abs() @ wd.abs().t(), K)
    _native.check_status(torch.device(DEV))


@pytest.mark.parametrize("M,N,K,few", [(32, 128, 1024, True), (32, 128, 896, False), (33, 640, 2048, True), (64, 16384, 4096, False), (64, 16384, 8192, True),
                                       (128, 2048, 4096, True), (128, 28672, 8192, False), (128, 128, 2048, False), (129, 128, 8192, False)])
def test_which_products_split_k(monkeypatch, M, N, K, few):
    """The kernel that the rule chooses, and products of a tile, a remainder and a part of K on both sides of the rule's lines."""
    assert (M <= schemes._FP8_FEW_ROWS and schemes._fp8_few_rows_faster(M, N, K)) == few
    N = min(N, 264)
    a, w, sa, sw, ad, wd = _make(M, N, K, M)
    for choice in (True, False):
        monkeypatch.setattr(schemes, "_fp8_few_rows_faster", lambda *size: choice)
        out = schemes.fp8_block_linear(None, w, sw, None, quant=(a, sa))
        _check(out, ad @ wd.t(), ad.abs() @ wd.abs().t(), K)
    _native.check_status(torch.device(DEV))
