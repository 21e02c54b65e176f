"""Gated products of 129 to 192 rows on both sides of the rule that gives them to the few-row kernel: one wave of its blocks, tiles with
remainders, one row past a limit."""
import pytest
import torch

from vllm_ascend_b200 import _native, ops

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("M,N,K,few", [(129, 6144, 2048, True), (160, 5704, 2056, True), (161, 6144, 2048, False), (192, 7112, 2048, True),
                                       (193, 8192, 2048, False), (137, 9472, 2048, True), (137, 9480, 2048, False), (137, 6144, 1024, False)])
def test_gated_rows(M, N, K, few):
    if torch.cuda.get_device_properties(0).multi_processor_count == 148:
        assert ops._few_rows(M, N, K, True) == few
    g = torch.Generator(device="cuda").manual_seed(M + N)
    x = torch.randn(M, K, device="cuda", generator=g).bfloat16()
    w = (torch.randn(2 * N, K, device="cuda", generator=g) * K ** -0.5).bfloat16()
    got = ops.linear_swiglu_step(x, w).double()
    xd = x.double()
    gate, up = xd @ w[:N].double().t(), xd @ w[N:].double().t()
    # fp32 sums of K products in any order: K 2^-24 of the sum of magnitudes; silu's slope is at most 1.1; the result is rounded to bf16
    mag = K * 2.0 ** -24
    eg, eu = (xd.abs() @ w[:N].double().abs().t()) * mag, (xd.abs() @ w[N:].double().abs().t()) * mag
    want = torch.nn.functional.silu(gate) * up
    bound = 1.1 * eg * (up.abs() + eu) + gate.abs() * eu + want.abs() * (2.0 ** -8 + 2.0 ** -20) + 1e-6
    assert ((got - want).abs() - bound).max().item() <= 0
    _native.check_status(torch.device("cuda"))
