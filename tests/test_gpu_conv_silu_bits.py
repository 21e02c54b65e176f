"""The convolution's SiLU, whose quotient is approximate away from the places where bf16 rounds the other way: equal to the exact
quotient's bits, which other kernels of the library return for the same sums."""
import pytest
import torch

from vllm_ascend_b200 import ops
from vllm_ascend_b200.ops import linear_attn as la

pytestmark = pytest.mark.gpu
DEV = "cuda"


def _conv(x, w):
    T, C, K = *x.shape, w.shape[1]
    state = torch.zeros(1, K - 1, C, dtype=x.dtype, device=DEV)
    one = dict(dtype=torch.int32, device=DEV)
    return la.causal_conv1d(x, w, None, state, torch.tensor([0, T], **one), torch.zeros(1, **one), torch.zeros(1, **one))


@pytest.mark.parametrize("K,C", [(4, 256), (3, 256), (5, 256), (4, 63)])
def test_every_bf16_sum(K, C):
    """One tap of one: the sums are all bf16 values, among them subnormal ones, infinities, NaN, and those whose exponential is above
    2^126 or infinite."""
    bits = torch.arange(65536, device=DEV).to(torch.uint16).view(torch.bfloat16)
    T = -(-65536 // C)
    x = torch.zeros(T * C, dtype=torch.bfloat16, device=DEV)
    x[:65536] = bits
    # a NaN or infinity meets the other taps' zeros in the rows behind it: rows of zeros in between
    rows = torch.zeros(K * T, C, dtype=torch.bfloat16, device=DEV)
    rows[::K] = x.view(T, C)
    w = torch.zeros(C, K, dtype=torch.bfloat16, device=DEV)
    w[:, K - 1] = 1
    got = _conv(rows, w)[::K].reshape(-1)[:65536]
    sums = (bits.float() + 0).bfloat16()                         # minus zero added to zeros is zero
    # the gated activation of the sum and a one, in 16 bits with the exact quotient
    want = ops.activation(torch.cat([sums, torch.ones_like(bits)]).view(2, 65536).t().contiguous(), "silu", gated=True).view(-1)
    assert torch.equal(got.isnan(), want.isnan()) and torch.equal(got.view(torch.int16)[~got.isnan()], want.view(torch.int16)[~want.isnan()])


@pytest.mark.parametrize("scale", [2.0 ** -26, 2.0 ** -20, 2.0 ** -18, 2.0 ** -15])
def test_sums_of_22_bits(scale):
    """Sums of two products that are whole numbers below 2^22 times a power of two, so that the convolution's and a matrix product's
    are the same: its gated epilogue divides exactly."""
    T, C = 4096, 4096
    g = torch.Generator(device=DEV).manual_seed(int(-torch.log2(torch.tensor(scale))))
    s = torch.randint(-127, 128, (T,), device=DEV, generator=g).float()
    taps = torch.randint(-127, 128, (C, 2), device=DEV, generator=g).float()
    w = torch.zeros(C, 4, device=DEV)
    w[:, 3], w[:, 2] = taps[:, 0] * 128 * scale, taps[:, 1] * scale
    got = _conv(s.bfloat16()[:, None].expand(T, C).contiguous(), w.bfloat16())
    x = torch.zeros(T, 8, device=DEV)
    x[:, 0], x[1:, 1], x[:, 2] = s, s[:-1], 1
    both = torch.zeros(2 * C, 8, device=DEV)
    both[:C, 0], both[:C, 1], both[C:, 2] = w[:, 3], w[:, 2], 1
    want = ops.linear_swiglu(x.bfloat16(), both.bfloat16())
    assert torch.equal(got.view(torch.int16), want.view(torch.int16))
