"""Decode attention with KV splits: stretches of the batch's tiles from eight sequences on, even parts below.  One long sequence among short ones, even batches, sequences without
keys or query rows, several query rows, a window, and split counts from two up to more than a sequence has tiles, against 64 bits."""
import types

import pytest
import torch

from vllm_ascend_b200 import _native, ops

pytestmark = pytest.mark.gpu

BATCHES = {"one long": [9000, 1, 128, 129, 300, 17, 640, 33, 2], "even": [1500] * 9, "ragged": [130 * i + 1 for i in range(40)],
           "holes": [0, 257, None, 1, None, None, 3000, 0, 128, None], "alone": [5000]}


@pytest.mark.parametrize("batch,Hq,Hkv,rows,window,splits", [
    ("one long", 32, 8, 1, 0, 2), ("one long", 32, 4, 1, 0, 32), ("even", 16, 2, 1, 0, 5), ("ragged", 64, 8, 1, 0, 2), ("ragged", 8, 8, 1, 300, 3),
    ("holes", 32, 8, 1, 0, 7), ("alone", 32, 8, 1, 0, 32), ("ragged", 16, 4, 4, 0, 3), ("alone", 4, 1, 2, 1000, 4), ("one long", 128, 8, 1, 0, 33)])
def test_against_fp64(batch, Hq, Hkv, rows, window, splits):
    lens = BATCHES[batch]                                     # None: a sequence without query rows
    lens = [n if n is None or rows == 1 else max(n, rows) for n in lens]
    g = torch.Generator().manual_seed(Hq + len(lens) + splits)
    D, page, B, dev = 128, 128, len(lens), torch.device("cuda")
    width = max(-(-(n or 1) // page) for n in lens)
    bt = torch.randperm(B * width, generator=g).view(B, width).int()
    k, v = ((torch.randn(B * width, page, Hkv, D, generator=g)).bfloat16() for _ in range(2))
    starts = [0]
    for n in lens:
        starts.append(starts[-1] + (0 if n is None else rows))
    T, scale, G = starts[-1], D ** -0.5, Hq // Hkv
    q = torch.randn(T, Hq, D, generator=g).bfloat16()
    i32 = dict(dtype=torch.int32, device=dev)
    meta = types.SimpleNamespace(query_start_loc=torch.tensor(starts, **i32), seq_lens=torch.tensor([n or 0 for n in lens], **i32),
                                 block_table=bt.to(dev), num_reqs=B, max_query_len=rows, max_seq_len=max(n or 0 for n in lens))
    kc, vc = (ops.alloc_kv_cache(B * width, page, Hkv, D, torch.bfloat16, dev) for _ in range(2))
    kc.copy_(k)
    vc.copy_(v)
    nbytes = T * Hq * splits * (D + 1) * 4
    ops._get_scratch(dev, nbytes).view(torch.float32).fill_(float("nan"))      # what a split leaves unwritten is not read
    out = torch.empty(T, Hq, D, dtype=torch.bfloat16, device=dev)
    ops.paged_attention_decode_tc(q.to(dev), kc, vc, meta, scale, out, window, num_splits=splits, max_q_len=rows)
    torch.cuda.synchronize()
    _native.check_status(dev)
    for b, n in enumerate(lens):
        if n is None:
            continue
        K, V = (x[bt[b].long()].reshape(-1, Hkv, D).to(dev).double() for x in (k, v))
        for r in range(rows):
            t, end = starts[b] + r, n - rows + r + 1
            if n == 0:
                assert not out[t].any()
                continue
            lo = max(0, end - window) if window else 0
            qr = q[t].to(dev).double().view(Hkv, G, D)
            s = torch.einsum("hgd,nhd->hgn", qr, K[lo:end]) * scale
            p = torch.softmax(s, -1)
            want = torch.einsum("hgn,nhd->hgd", p, V[lo:end])
            # a probability is rounded to bf16 (eight bits: 2^-8; fp32 sums and ex2 stay below 2^-12 of the terms), and so is the result
            before = torch.einsum("hgn,nhd->hgd", p, V[lo:end].abs()) * (2.0 ** -8 + 2.0 ** -12)
            bound = before + (want.abs() + before) * 2.0 ** -8 + 1e-6
            excess = ((out[t].double().view(Hkv, G, D) - want).abs() - bound).max().item()
            assert excess <= 0, (b, r, n, excess)
