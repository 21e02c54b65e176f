"""The grouped product at the edges of its tiles and of its group table: groups without rows, around a tile, tables around a warp."""
import pytest
import torch

from vllm_ascend_b200 import _native
from vllm_ascend_b200.ops import moe_native

pytestmark = pytest.mark.gpu
DEV = "cuda"


@pytest.mark.parametrize("E,N,swiglu", [(1, 264, False), (32, 640, False), (33, 128, True), (70, 384, True)])
def test_grouped_product_of_ragged_groups(E, N, swiglu):
    g = torch.Generator().manual_seed(E)
    sizes = [(0, 1, 127, 128, 129, 0, 300, 3)[e % 8] for e in range(E)]
    sizes[0] = 257
    K, rows = 192, sum(sizes)
    offsets = torch.tensor([0] + sizes).cumsum(0).int()
    a = torch.randn(rows, K, generator=g).bfloat16()
    w = (torch.randn(E, N * (2 if swiglu else 1), K, generator=g) * K ** -0.5).bfloat16()
    got = moe_native.grouped_gemm(a.to(DEV), w.to(DEV), offsets.to(DEV), swiglu)
    torch.cuda.synchronize()
    _native.check_status(torch.device(DEV))
    for e in range(E):
        part = a[offsets[e]:offsets[e + 1]].double()
        want = part @ w[e].double().T
        # fp32 sums of K exact products, then one rounding to bf16 (through SwiGLU: of a product whose factors are such sums)
        slack = (part.abs() @ w[e].double().abs().T) * K * 2.0 ** -24
        if swiglu:
            gate, up = want[:, :N], want[:, N:]
            want = torch.nn.functional.silu(gate) * up
            slack = 1.1 * slack[:, :N] * up.abs() + slack[:, N:] * gate.abs() + 2.0 ** -18 * want.abs()
        err = (got[offsets[e]:offsets[e + 1]].double().cpu() - want).abs()
        assert (err <= want.abs() * 2.0 ** -8 + slack + 1e-6).all(), e
