"""Latent attention captured in a graph, beside an eager step that needs more scratch for its splits than the graph's launches share."""
import torch
import pytest

from vllm_ascend_b200 import _native
from vllm_ascend_b200.attention import mla
from vllm_ascend_b200.ops.scratch import Scratch

pytestmark = pytest.mark.gpu


def _call(dev, rows, keys, seed, uniform):
    """``rows`` query rows of 16 heads: one per sequence, or all of one sequence, whose rows share blocks."""
    g = torch.Generator(device=dev).manual_seed(seed)
    B, H, dc, dr, page = (rows if uniform else 1), 16, 512, 64, 64
    width = keys // page
    lat, pe = ((torch.randn(B * width, page, d, device=dev, generator=g) * 0.5).bfloat16() for d in (dc, dr))
    q = torch.randn(rows, H, dc + dr, device=dev, generator=g).bfloat16()
    i32 = dict(dtype=torch.int32, device=dev)
    bt = torch.arange(B * width, **i32).view(B, width)
    cu = torch.arange(0, rows + 1, **i32) if uniform else torch.tensor([0, rows], **i32)
    lens = torch.full((B,), keys, **i32)
    return lambda: mla.latent_attention_tc(q[..., :dc], q[..., dc:], lat, pe, bt, 0.04, cu=cu, seq_lens=lens, uniform=uniform, max_kv_len=keys)


def test_a_graph_keeps_its_scratch(monkeypatch):
    dev = torch.device("cuda", torch.cuda.current_device())
    monkeypatch.setattr(mla, "_scratch", Scratch(torch.float32))
    small, large = _call(dev, 8, 1024, 1, True), _call(dev, 17, 4096, 2, False)
    want, want_large = small(), large()
    monkeypatch.setattr(mla, "_scratch", Scratch(torch.float32))
    stream = torch.cuda.Stream()
    with torch.cuda.stream(stream):
        small()
        torch.cuda.synchronize()
        held = mla._split_scratch(dev, 1).data_ptr()
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph, stream=stream):
            got = small()
        got_large = large()
        assert mla._split_scratch(dev, 1).data_ptr() == held
        others = [torch.full((17 * 16 * 32 * 513,), 7.0, device=dev), torch.full((1 << 20,), 7.0, device=dev)]
        graph.replay()
        torch.cuda.synchronize()
    assert torch.equal(got, want) and torch.equal(got_large, want_large)
    assert all(bool((t == 7).all()) for t in others)
    _native.check_status(dev)
