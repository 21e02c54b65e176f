"""Routing kernels at their edges: expert counts around the unrolled widths, equal scores, pairs around the one-block permutation."""
import pytest
import torch

from vllm_ascend_b200.ops import moe_native

pytestmark = pytest.mark.gpu
DEV = "cuda"


@pytest.mark.parametrize("E,k,bias", [(1, 1, False), (31, 5, True), (128, 8, False), (129, 8, True), (256, 32, False), (257, 3, True),
                                      (512, 10, False)])
def test_equal_scores_go_to_the_lowest_expert(E, k, bias):
    g = torch.Generator().manual_seed(E)
    logits = torch.randint(-2, 3, (53, E), generator=g).float()              # many ties
    b = torch.randint(-1, 2, (E,), generator=g).float() if bias else None    # choices below zero too
    w, ids = moe_native.gating_topk(logits.to(DEV), k, "sigmoid", False, 1, 1, None if b is None else b.to(DEV), 1.0)
    score = torch.sigmoid(logits.double())
    choice = logits if b is None else (score + b)       # without a bias the order of the logits, whose ties are exact
    want = torch.sort(choice, dim=-1, descending=True, stable=True).indices[:, :k]
    assert torch.equal(ids.cpu().long(), want)
    assert torch.allclose(w.cpu().double(), score.gather(1, want), rtol=1e-6)      # expf and a division: a few ulp


@pytest.mark.parametrize("T,k,E", [(1, 1, 1), (48, 8, 128), (1024, 8, 33), (2731, 3, 1024), (8193, 1, 64), (700, 6, 512)])
def test_permutation_is_expert_major(T, k, E):
    g = torch.Generator().manual_seed(T)
    ids = torch.randint(-1, E + 1, (T, k), generator=g, dtype=torch.int32)         # -1 and E: experts of other ranks
    p = moe_native.Permutation(ids.to(DEV), None, E)
    flat = ids.flatten().long()
    here = (flat >= 0) & (flat < E)
    counts = torch.bincount(flat[here], minlength=E)
    offsets = torch.cat([torch.zeros(1, dtype=torch.int64), counts.cumsum(0)])
    assert torch.equal(p.counts.cpu().long(), counts) and torch.equal(p.cursor.cpu().long(), counts)
    assert torch.equal(p.offsets.cpu().long(), offsets)
    pos, src = p.pos.cpu().long(), p.src_token.cpu().long()
    assert (pos[~here] == -1).all()
    assert torch.equal(pos[here].sort().values, torch.arange(int(here.sum())))
    assert torch.equal(torch.searchsorted(offsets, pos[here], right=True) - 1, flat[here])
    assert torch.equal(src[pos[here]], (torch.arange(T * k) // k)[here])
