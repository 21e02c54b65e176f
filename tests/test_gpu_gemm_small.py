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
