"""Shapes that the products and the norm refuse, without a GPU: rows without columns."""
import pytest
import torch

from vllm_ascend_b200 import ops


@pytest.mark.parametrize("call", [
    lambda x: ops.linear(x, torch.empty(8, 0, dtype=torch.bfloat16)), lambda x: ops.linear_swiglu(x, torch.empty(16, 0, dtype=torch.bfloat16)),
    lambda x: ops.rms_norm(x, torch.empty(0, dtype=torch.bfloat16), 1e-6)], ids=["linear", "swiglu", "norm"])
@pytest.mark.parametrize("shape", [(4, 0), (2, 2, 0)])
def test_no_columns(monkeypatch, call, shape):
    monkeypatch.setattr(ops, "_use_native", lambda x: True)      # as on a GPU; nothing is launched
    with pytest.raises(RuntimeError, match="reshape"):
        call(torch.empty(shape, dtype=torch.bfloat16))
