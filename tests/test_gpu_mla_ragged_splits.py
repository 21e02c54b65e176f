"""KV splits of the latent attention kernel that take the same number of tiles for every sequence: batches of one long sequence and
many short ones (empty splits, a split count that only the longest one uses), even ones, rows without keys, several rows a sequence
and a window, against the same sums in 64 bits."""
import pytest
import torch

from vllm_ascend_b200 import _native
from vllm_ascend_b200.attention import mla

pytestmark = pytest.mark.gpu

BATCHES = {"one long": [9000] + [1, 128, 129, 300, 17, 0, 640], "even": [1500] * 9, "ragged": [130 * i + 1 for i in range(30)],
           "few slots": [4000, 3900, 5, 1]}


@pytest.mark.parametrize("batch,H,per_seq,window,splits", [
    ("one long", 32, 1, 0, 0), ("even", 128, 1, 0, 0), ("ragged", 16, 1, 0, 0), ("ragged", 32, 1, 300, 7), ("few slots", 64, 1, 0, 3),
    ("one long", 16, 2, 0, 0), ("ragged", 8, 3, 500, 5), ("few slots", 16, 2, 0, 2)])
def test_common_tiles(batch, H, per_seq, window, splits):
    lens = [n if per_seq == 1 else max(n, per_seq) for n in BATCHES[batch]]
    g = torch.Generator().manual_seed(H + len(lens))
    dc, dr, page, B = 512, 64, 64, len(lens)
    width = -(-max(lens) // page)
    bt = torch.randperm(B * width, generator=g).view(B, width).int()
    lat, pe = ((torch.randn(B * width, page, d, generator=g) * 0.5).bfloat16() for d in (dc, dr))
    R = B * per_seq
    q = torch.randn(R, H, dc + dr, generator=g).bfloat16()
    scale, dev = (dc + dr) ** -0.5, torch.device("cuda")
    i32 = dict(dtype=torch.int32, device=dev)
    lse = torch.empty(R, H, device=dev)
    mla._split_scratch(dev, 1).fill_(float("nan"))             # what a split leaves unwritten is not read
    got = mla.latent_attention_tc(q[..., :dc].to(dev), q[..., dc:].to(dev), lat.to(dev), pe.to(dev), bt.to(dev), scale,
                                  cu=torch.arange(0, R + 1, per_seq, **i32), seq_lens=torch.tensor(lens, **i32), uniform=per_seq == 1,
                                  window=window, num_splits=splits, max_kv_len=max(lens), lse_out=lse)
    torch.cuda.synchronize()
    _native.check_status(dev)
    for r in range(R):
        b, n = r // per_seq, lens[r // per_seq] - (per_seq - 1 - r % per_seq)
        if n == 0:
            assert not got[r].any() and bool((lse[r] == -float("inf")).all())
            continue
        L, P = (x[bt[b].long()].reshape(-1, x.shape[-1])[max(0, n - window) if window else 0:n].to(dev).double() for x in (lat, pe))
        qr = q[r].to(dev).double()
        s = (qr[:, :dc] @ L.T + qr[:, dc:] @ P.T) * scale
        p = torch.softmax(s, -1)
        # a probability is rounded to bf16 (eight bits: 2^-8; fp32 sums and ex2 stay below 2^-12 of the terms), and so is the result
        before = (p @ L.abs()) * (2.0 ** -8 + 2.0 ** -12)
        bound = before + ((p @ L).abs() + before) * 2.0 ** -8 + 1e-6
        excess = ((got[r].double() - p @ L).abs() - bound).max().item()
        assert excess <= 0, (r, n, excess)
        assert (lse[r].double() - torch.logsumexp(s, -1)).abs().max().item() < 2.0 ** -12 * (1 + s.abs().max().item())
