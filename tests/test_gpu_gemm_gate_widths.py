"""Gated products of the paired-CTA kernel in every tile width that the rule picks."""
import pytest
import torch

from vllm_ascend_b200 import _native, ops

pytestmark = pytest.mark.gpu


# rows, gate columns -> 128, 160, 192, 224 and 256 columns a tile on 148 SMs; last tiles that hold 64 to 8 gate columns, last row tiles
# of 1 to 256 rows
@pytest.mark.parametrize("M,I", [(300, 1536), (300, 2944), (257, 6400), (520, 5120), (512, 128), (150, 9728), (137, 12288), (256, 12288)])
@pytest.mark.parametrize("limit", [None, 7.0])
def test_gate_widths(M, I, limit):
    K = 512
    g = torch.Generator(device="cuda").manual_seed(M + I)
    x = torch.randn(M, K, device="cuda", generator=g).bfloat16()
    w = (torch.randn(2 * I, K, device="cuda", generator=g) * K ** -0.5).bfloat16()
    out = ops.linear_swiglu(x, w, two_cta=True, limit=limit).float()
    _native.check_status(x.device)
    h = x.double() @ w.double().t()
    gate, up = h[:, :I], h[:, I:]
    if limit is None:
        exp = gate * torch.sigmoid(gate) * up
    else:
        gate, up = gate.clamp(max=limit), up.clamp(-limit, limit) + 1
        exp = gate * torch.sigmoid(ops.CLAMPED_GATE_ALPHA * gate) * up
    # one rounding to bf16 (2^-9 of the value), and fp32 sums of 512 products of about 1 / 512 and an exponential (below 2^-14 of gate times up)
    assert bool(((out - exp).abs() <= 2.0 ** -8 * exp.abs() + 2.0 ** -12 * (1 + up.abs()) * (1 + gate.abs())).all())
