"""Causal convolution of steps whose blocks take 32 rows (2048 tokens and more) or 16, at the edges of both."""
import pytest
import torch

from vllm_ascend_b200.ops import linear_attn as la

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("lens", [[31, 32, 33, 64, 1, 2, 1885], [2048], [15, 16, 17, 1999], [1, 2050]])
@pytest.mark.parametrize("K,C", [(4, 264), (3, 256), (2, 72), (5, 64)])
def test_tiles(lens, K, C):
    gen = torch.Generator(device="cuda").manual_seed(sum(lens) + K)
    T, B = sum(lens), len(lens)
    x, w = torch.randn(T, C, device="cuda", generator=gen).bfloat16(), torch.randn(C, K, device="cuda", generator=gen).bfloat16()
    state = torch.randn(B, K - 1, C, device="cuda", generator=gen).bfloat16()
    cu = torch.tensor([sum(lens[:i]) for i in range(B + 1)], dtype=torch.int32, device="cuda")
    slots, init = torch.arange(B, dtype=torch.int32, device="cuda"), torch.tensor([i % 2 for i in range(B)], dtype=torch.int32, device="cuda")
    st_ref, st = state.double(), state.clone()
    y = la.causal_conv1d(x, w, None, st, cu, slots, init)
    want = la.causal_conv1d_ref(x.double(), w.double(), None, st_ref, cu, slots, init)
    # one rounding to bf16; in fp32 a sum of five products below 64 (2^-24 of each) and a sigmoid
    assert bool(((y.double() - want).abs() <= 2.0 ** -8 * want.abs() + 2.0 ** -16).all())
    assert torch.equal(st.double(), st_ref)
