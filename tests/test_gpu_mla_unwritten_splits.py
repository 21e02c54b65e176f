"""The batches of test_gpu_mla_ragged_splits over scratch that is large enough for them and filled with NaN: a split without keys leaves its
sums unwritten, and the merge must not read them."""
import pytest
import torch

import test_gpu_mla_ragged_splits as ragged
from vllm_ascend_b200.attention import mla
from vllm_ascend_b200.ops.scratch import Scratch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("batch,H,per_seq,window,splits", [
    ("one long", 32, 1, 0, 0), ("even", 128, 1, 0, 0), ("ragged", 16, 1, 0, 0), ("ragged", 32, 1, 300, 7), ("few slots", 64, 1, 0, 3),
    ("one long", 16, 2, 0, 0), ("ragged", 8, 3, 500, 5), ("few slots", 16, 2, 0, 2), ("one long", 32, 1, 0, 31)])
def test_over_nan(monkeypatch, batch, H, per_seq, window, splits):
    dev = torch.device("cuda", torch.cuda.current_device())
    monkeypatch.setattr(mla, "_scratch", Scratch(torch.float32))
    buf = mla._split_scratch(dev, len(ragged.BATCHES[batch]) * per_seq * H * max(splits, mla._MAX_SPLITS) * (512 + 1))
    ragged.test_common_tiles(batch, H, per_seq, window, splits)            # fills the shared tensor with NaN before its call
    assert mla._split_scratch(dev, 1).data_ptr() == buf.data_ptr() and bool(buf.isnan().any())
