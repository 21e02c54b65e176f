"""Chunked delta rule with keys that are not normalised: writes that grow from token to token, behind tokens that write nothing."""
import pytest
import torch

from vllm_ascend_b200 import _native
from vllm_ascend_b200.ops import linear_attn as la

pytestmark = pytest.mark.gpu
DEV = "cuda"


@pytest.mark.parametrize("silent", [40, 50, 63])
@pytest.mark.parametrize("DV", [64, 128])
def test_growing_writes(silent, DV):
    """All keys are one with k . k = 8 and beta is one, so each token multiplies the state by -7 before it adds its value.  The first
    ``silent`` of 64 tokens have none, and the state stays below 7^25; (I + A)^-1 of the chunk has entries up to 7^62, which is no fp32 number."""
    T, H = 64, 2
    gen = torch.Generator(device=DEV).manual_seed(silent + DV)
    k = torch.full((T, H, 128), 0.25, device=DEV).bfloat16()
    q = torch.rand(T, H, 128, device=DEV, generator=gen).bfloat16()
    v = torch.rand(T, H, DV, device=DEV, generator=gen).bfloat16()
    v[:silent] = 0
    g, beta = torch.zeros(T, H, device=DEV), torch.ones(T, H, device=DEV)
    S, cu = torch.zeros(1, H, 128, DV, device=DEV), torch.tensor([0, T], dtype=torch.int32, device=DEV)
    out = la.gated_delta_rule(q, k, v, g, beta, S, cu, cu[:1], cu[:1], 1.0, l2norm=False, cu_cpu=[0, T])
    _native.check_status(torch.device(DEV))
    state = torch.zeros(H, 128, DV, dtype=torch.float64, device=DEV)
    for t in range(T):
        u = v[t].double() - torch.einsum("hkv,hk->hv", state, k[t].double())
        state += torch.einsum("hk,hv->hkv", k[t].double(), u)
        want = torch.einsum("hkv,hk->hv", state, q[t].double())
        # fp32 sums of up to 64 terms at most 8 / 7 + 8 / 49 + ... times the result, one after the other: 64 x 4 units of 2^-24; bf16
        assert bool(((out[t].double() - want).abs() <= want.abs() * (2.0 ** -8 + 2.0 ** -14) + 1e-6).all()), t
    assert bool(((S[0].double() - state).abs() <= state.abs() * 2.0 ** -14 + 1e-6).all())
