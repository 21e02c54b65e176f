"""Modes that fix the order of sums: where the keys of a sequence are cut into splits does not depend on its neighbours."""
import types

import pytest
import torch

from vllm_ascend_b200 import _native, batch_invariant, ops
from vllm_ascend_b200.attention import mla

pytestmark = pytest.mark.gpu
DEV = "cuda"


@pytest.fixture(params=["batch-invariant", "training-consistent"])
def mode(request, monkeypatch):
    if request.param == "batch-invariant":
        monkeypatch.setenv("VLLM_B200_BATCH_INVARIANT", "1")
    else:
        monkeypatch.setattr(batch_invariant, "_training_consistent", True)


def _latent(lens, with_lse, splits=0):
    """Bits of the first sequence beside the others of ``lens``: the same page numbers hold its keys in every batch."""
    g = torch.Generator(device=DEV).manual_seed(5)
    H, dc, dr, page = 16, 512, 64, 64
    pages = 256
    lat, pe = ((torch.randn(pages, page, d, device=DEV, generator=g) * 0.5).bfloat16() for d in (dc, dr))
    q = torch.randn(len(lens), H, dc + dr, device=DEV, generator=g).bfloat16()
    q[0] = torch.randn(H, dc + dr, device=DEV, generator=torch.Generator(device=DEV).manual_seed(6)).bfloat16()
    i32 = dict(dtype=torch.int32, device=DEV)
    width = -(-max(lens) // page)
    bt = torch.arange(len(lens) * width, **i32).view(len(lens), width) % pages
    bt[0] = torch.arange(width, **i32) % pages
    lse = torch.empty(len(lens), H, device=DEV) if with_lse else None
    out = mla.mla_decode_native(q, lat, pe, torch.arange(len(lens), **i32), torch.tensor(lens, **i32), bt, 0.04, num_splits=splits,
                                max_kv_len=max(lens), lse_out=lse)
    _native.check_status(torch.device(DEV, 0))
    return out[0].clone(), None if lse is None else lse[0].clone()


@pytest.mark.parametrize("with_lse,splits", [(True, 0), (False, 0), (True, 5), (False, 3)])
@pytest.mark.parametrize("others", [[5100], [1] * 7, [200, 3000, 1, 900] * 8])
def test_latent_attention(mode, with_lse, splits, others):
    alone, beside = _latent([1200], with_lse, splits), _latent([1200] + others, with_lse, splits)
    assert torch.equal(alone[0], beside[0])
    assert not with_lse or torch.equal(alone[1], beside[1])


@pytest.mark.parametrize("splits", [2, 5])
def test_grouped_attention(mode, splits):
    """A split count that the caller names."""
    def first(others):
        lens = [2000] + others
        g = torch.Generator(device=DEV).manual_seed(7)
        B, page, Hq, Hkv, D, pages = len(lens), 128, 16, 4, 128, 128
        kc, vc = (ops.alloc_kv_cache(pages, page, Hkv, D, torch.bfloat16, torch.device(DEV, 0)) for _ in range(2))
        for c in (kc, vc):
            c.copy_(torch.randn(c.shape, device=DEV, generator=g))
        q = torch.randn(B, Hq, D, device=DEV, generator=g).bfloat16()
        q[0] = torch.randn(Hq, D, device=DEV, generator=torch.Generator(device=DEV).manual_seed(8)).bfloat16()
        i32 = dict(dtype=torch.int32, device=DEV)
        width = -(-max(lens) // page)
        bt = torch.arange(B * width, **i32).view(B, width) % pages
        meta = types.SimpleNamespace(query_start_loc=torch.arange(B + 1, **i32), seq_lens=torch.tensor(lens, **i32), block_table=bt,
                                     num_reqs=B, max_query_len=1, max_seq_len=max(lens))
        out = torch.empty_like(q)
        ops.paged_attention_decode_tc(q, kc, vc, meta, D ** -0.5, out, num_splits=splits, max_q_len=1)
        _native.check_status(torch.device(DEV, 0))
        return out[0].clone()
    assert torch.equal(first([2000] * 9), first([9000, 1, 300, 128, 129, 17, 640, 33, 2]))


def test_split_counts(mode):
    from vllm_ascend_b200.attention.variant import AttnOptions, decode_splits
    dev = torch.device(DEV, 0)
    assert ops.choose_num_splits(4, 8, 8192) == decode_splits(4, 2, AttnOptions(scale=1.0), 8192, dev) == mla._num_splits(dev, 4, 8192) == 1
