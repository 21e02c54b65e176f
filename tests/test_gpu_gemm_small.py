"""Few-row GEMM: edges of its tiles (16 tokens, 128 weight rows, 64 columns of K), every split, both epilogues, against
fp64 products.  Bound: half a bf16 ulp of the result (2^-9) plus fp32 sums of K terms, 2^-24 sqrt(K) of the absolute sum
for random signs, taken eight times."""
import pytest
import torch

from vllm_ascend_b200 import _native, ops

pytestmark = pytest.mark.gpu
DEV = "cuda"


def _check(got, want, absum, K):
    bound = want.abs() * 2.0 ** -8 + absum * (8 * 2.0 ** -24 * K ** 0.5) + 1e-6
    assert ((got.double() - want).abs() <= bound).all()


@pytest.mark.parametrize("M,N,K", [(1, 8, 8), (1, 4096, 4096), (15, 136, 2048), (16, 128, 2056), (17, 640, 4096), (128, 200, 2048),
                                   (129, 4096, 4096), (255, 1536, 2112), (256, 5120, 2048), (1, 32000, 2048)])
def test_linear_step_against_fp64(M, N, K):
    g = torch.Generator(device=DEV).manual_seed(M + N + K)
    wide = torch.randn(M, K + 8, device=DEV, generator=g).bfloat16()
    x = wide[:, :K]                                              # rows with a stride of their own
    w = (torch.randn(N, K, device=DEV, generator=g) * 0.05).bfloat16()
    b = torch.randn(N, device=DEV, generator=g).bfloat16()
    r = torch.randn(M, N, device=DEV, generator=g).bfloat16()
    want = x.double() @ w.double().t()
    absum = x.double().abs() @ w.double().abs().t() + 8
    _check(ops.linear_step(x, w), want, absum, K)
    got = ops.linear_step(x, w, b, r)
    _check(got, want + b.double() + r.double(), absum, K)
    assert torch.equal(got, ops.linear_step(x, w, b, r))         # sums have one order
    _native.check_status(torch.device(DEV))


@pytest.mark.parametrize("splits", [1, 2, 3, 5, 8])
def test_every_split_and_the_gates(splits):
    g = torch.Generator(device=DEV).manual_seed(splits)
    M, I, K = 37, 328, 1000
    x = torch.randn(M, K, device=DEV, generator=g).bfloat16()
    w = (torch.randn(2 * I, K, device=DEV, generator=g) * 0.05).bfloat16()
    gate, up = (x.double() @ w.double().t()).split(I, 1)
    for alpha, limit in ((0.0, 0.0), (1.702, 0.7)):
        out = torch.full((M, I), float("nan"), device=DEV, dtype=torch.bfloat16)
        _native.check(_native.lib().b200_gemm_small_bf16(
            x.data_ptr(), w.data_ptr(), out.data_ptr(), None, None, M, I, K, K, K, I, 1, alpha, limit, splits,
            _native.status_word(x.device).data_ptr(), _native.stream_ptr()), "gemm_small")
        if alpha:
            gc = gate.clamp(max=limit)
            want = gc * torch.sigmoid(alpha * gc) * (up.clamp(-limit, limit) + 1)
        else:
            want = torch.nn.functional.silu(gate) * up
        # the fast exponential adds 2^-21 of the gate, the products' fp32 sums far less
        assert ((out.double() - want).abs() <= want.abs() * 2.0 ** -8 + 2e-4).all()
    _native.check_status(torch.device(DEV))


def test_rows_do_not_depend_on_the_row_count_within_a_tile():
    g = torch.Generator(device=DEV).manual_seed(3)
    x = torch.randn(128, 4096, device=DEV, generator=g).bfloat16()
    w = (torch.randn(6144, 4096, device=DEV, generator=g) * 0.05).bfloat16()
    full = ops.linear_step(x, w)
    for m in (1, 16, 33, 100):
        assert torch.equal(ops.linear_step(x[:m], w), full[:m])


@pytest.mark.parametrize("M,N,K", [(1, 128, 2048), (256, 4096, 2048), (130, 1000, 4096)])
def test_row_statistics_are_those_of_the_stored_rows(M, N, K):
    g = torch.Generator(device=DEV).manual_seed(N)
    x = torch.randn(M, K, device=DEV, generator=g).bfloat16()
    w = (torch.randn(N, K, device=DEV, generator=g) * 0.05).bfloat16()
    res = torch.randn(M, N, device=DEV, generator=g).bfloat16()
    ss = ops.alloc_row_stats(300, 4096, torch.device(DEV))
    want = ops.linear_step(x, w, None, res)
    out = ops.linear_norm_folded(x, w, residual=res, out=res, ss_out=ss)       # in place on the stream
    assert out is res and torch.equal(out, want)
    parts = int(ss[32 * 300:32 * 300 + 1].view(torch.int32))
    assert parts == (N + 127) // 128
    got = ss[:parts * 300].view(parts, 300)[:, :M]
    sq = torch.nn.functional.pad(out.double() ** 2, (0, parts * 128 - N)).view(M, parts, 128).sum(-1).t()
    assert ((got.double() - sq).abs() <= sq * 2.0 ** -20).all()
    # the next product reads them
    w2 = (torch.randn(256, N, device=DEV, generator=g) * 0.05).bfloat16()
    y = ops.linear_norm_folded(out, w2, ss_in=ss, norm_dim=N, eps=1e-6)
    ref = (out.double() @ w2.double().t()) * torch.rsqrt((out.double() ** 2).mean(-1, keepdim=True) + 1e-6)
    assert ((y.double() - ref).abs() <= ref.abs() * 2.0 ** -8 + 1e-3).all()
    _native.check_status(torch.device(DEV))


@pytest.mark.parametrize("M,N,K", [(33, 12288, 2048), (40, 5120, 2048), (64, 6144, 2112), (130, 3072, 2048), (250, 2040, 2048)])
def test_splits_that_fit_one_wave(M, N, K):
    """Tile counts at which a part more per tile would leave clusters for a second wave."""
    g = torch.Generator(device=DEV).manual_seed(N)
    x = torch.randn(M, K, device=DEV, generator=g).bfloat16()
    w = (torch.randn(N, K, device=DEV, generator=g) * 0.05).bfloat16()
    assert ops._few_rows(M, N, K) == (N != 12288)
    out = torch.full((M, N), float("nan"), device=DEV, dtype=torch.bfloat16)
    ops._gemm_small(x, w, out, None, None, N, False)
    _check(out, x.double() @ w.double().t(), x.double().abs() @ w.double().abs().t(), K)
    _native.check_status(torch.device(DEV))


def test_splits_and_the_choice_of_kernel():
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    for M in (1, 16, 64, 128, 129, 256):
        for N in (8, 128, 2048, 5120, 6144, 12288, 18944, 60000, 151936):
            for K in (8, 2040, 2048, 4096, 28672):
                for glu in (0, 1):
                    s = _native.lib().b200_gemm_small_splits(M, N, K, glu)
                    tiles, blocks = -(-N // (64 if glu else 128)), -(-K // 64)
                    assert 1 <= s <= min(8, max(1, blocks // 4)) and (s == 1 or blocks >= 32)
                    assert s == 1 or s * tiles <= sms * (2 if M <= 128 else 1), (M, N, K, glu, s)
    assert _native.lib().b200_gemm_small_splits(257, 128, 4096, 0) < 0
    # K that is not split, products wide enough for the general kernels, few rows
    few = ops._few_rows
    assert few(1, 4096, 512) and few(32, 151936, 2048) and few(128, 4096, 2048) and few(256, 4096, 4096) and few(64, 12288, 4096)
    assert not few(33, 4096, 1536) and not few(256, 6144, 4096) and not few(128, 12288, 4096) and not few(64, 12288, 2048)
    assert few(100, 28672, 2048, True) and not few(128, 28672, 2048, True) and not few(200, 768, 1024, True)
