"""Output tensors that a caller gives: those of another size than the result are refused."""
import pytest
import torch

from vllm_ascend_b200 import ops

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("call,cols", [
    (lambda x, out: ops.linear(x, x.new_zeros(64, 128), out=out), 64), (lambda x, out: ops.linear_swiglu(x, x.new_zeros(128, 128), out=out), 64),
    (lambda x, out: ops.rms_norm(x, x.new_ones(128), 1e-6, out=out), 128)], ids=["linear", "swiglu", "norm"])
@pytest.mark.parametrize("rows", [(12,), (3, 4)])
def test_wider_outputs(call, cols, rows):
    x = torch.randn(*rows, 128, device="cuda").bfloat16()
    call(x, x.new_empty(12, cols))
    with pytest.raises(RuntimeError, match="view|shape"):
        call(x, x.new_empty(12, cols + 8))
