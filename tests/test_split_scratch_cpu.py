"""Shared scratch of the split-KV kernels: what a captured graph holds the address of is never replaced."""
import pytest
import torch

from vllm_ascend_b200 import ops
from vllm_ascend_b200.attention import mla


@pytest.mark.parametrize("get", [lambda n: ops._get_scratch(torch.device("cpu"), n), lambda n: mla._split_scratch(torch.device("cpu"), n)],
                         ids=["attention", "latent"])
def test_a_captured_buffer_stays(monkeypatch, get):
    monkeypatch.setattr(torch.cuda, "is_initialized", lambda: True)      # as on a GPU, whose streams can be captured
    monkeypatch.setattr(torch.cuda, "is_current_stream_capturing", lambda: False)
    get(1)
    grown = get(3 << 20)
    assert grown.numel() >= 3 << 20 and get(1).data_ptr() == grown.data_ptr()      # shared, and grown while no graph has it
    monkeypatch.setattr(torch.cuda, "is_current_stream_capturing", lambda: True)
    held = get(1).data_ptr()                        # a graph's launch
    larger = get(4 << 20)                           # another graph's, from its own pool
    assert larger.numel() >= 4 << 20 and larger.data_ptr() != held
    monkeypatch.setattr(torch.cuda, "is_current_stream_capturing", lambda: False)
    assert get(1).data_ptr() == held
    more = get(5 << 20)                             # a later eager step
    assert more.numel() >= 5 << 20 and more.data_ptr() != held
    assert get(1).data_ptr() == held and get(3 << 20).data_ptr() == held


@pytest.mark.parametrize("get", [lambda n: ops._get_scratch(torch.device("cpu"), n), lambda n: mla._split_scratch(torch.device("cpu"), n)],
                         ids=["attention", "latent"])
def test_a_buffer_of_inference_mode_serves_others(get):
    with torch.inference_mode():
        assert not get(6 << 20).is_inference()
