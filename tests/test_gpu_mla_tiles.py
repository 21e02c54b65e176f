"""Latent attention kernel at the edges of its tiles and of its two softmax paths (whole tiles, masked ones): lengths around 128 keys,
odd slab counts, windows, sinks, head counts below and above a block's columns, and scores whose maximum moves late."""
import pytest
import torch

from vllm_ascend_b200 import _native
from vllm_ascend_b200.attention.mla import latent_attention_tc

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("H,dc,dr,block_size,splits,window,sink", [
    (32, 512, 64, 128, 1, 0, False), (32, 512, 64, 16, 2, 0, False), (16, 512, 64, 64, 1, 0, True), (7, 192, 32, 32, 1, 0, False),
    (40, 72, 8, 8, 3, 0, False), (16, 320, 64, 128, 1, 70, True), (32, 512, 64, 256, 2, 1, False)])
def test_tile_edges(H, dc, dr, block_size, splits, window, sink):
    g = torch.Generator().manual_seed(H + dc + window)
    lens = [1, 63, 64, 65, 127, 128, 129, 191, 192, 193, 257, 1030]
    R, nblk = len(lens), -(-max(lens) // block_size)
    bt = torch.randperm(R * nblk, generator=g).view(R, nblk).int()
    lat = (torch.randn(R * nblk, block_size, dc, generator=g) * 0.5).bfloat16()
    pe = (torch.randn(R * nblk, block_size, dr, generator=g) * 0.5).bfloat16()
    lat[bt[-1, -1].item()] *= 4            # the last tile of the longest row raises the maximum: sums and O are scaled again
    q = (torch.randn(R, H, dc + dr, generator=g)).bfloat16()
    sinks = torch.randn(H, generator=g) if sink else None
    scale = (dc + dr) ** -0.5
    dev = torch.device("cuda")
    got = latent_attention_tc(q[..., :dc].to(dev), q[..., dc:].to(dev), lat.to(dev), pe.to(dev), bt.to(dev), scale,
                              row_seq=torch.arange(R, dtype=torch.int32, device=dev),
                              row_kv_len=torch.tensor(lens, dtype=torch.int32, device=dev), window=window,
                              sink=None if sinks is None else sinks.to(dev), num_splits=splits, max_kv_len=max(lens))
    torch.cuda.synchronize()
    _native.check_status(dev)
    for r, n in enumerate(lens):
        L, P = (x[bt[r].long()].reshape(-1, x.shape[-1])[max(0, n - window) if window else 0:n].double() for x in (lat, pe))
        s = (q[r, :, :dc].double() @ L.T + q[r, :, dc:].double() @ P.T) * scale
        if sinks is not None:
            s = torch.cat([s, sinks.double()[:, None]], 1)
            L = torch.cat([L, torch.zeros(1, dc, dtype=torch.float64)])
        p = torch.softmax(s, -1)
        # a probability is rounded to bf16 (2^-9; fp32 sums and ex2 stay below 2^-12 of the terms), and so is the result that they give
        before = (p @ L.abs()) * (2.0 ** -9 + 2.0 ** -12)
        bound = before + ((p @ L).abs() + before) * 2.0 ** -9 + 1e-6
        excess = ((got[r].double().cpu() - p @ L).abs() - bound).max().item()
        assert excess <= 0, (r, n, excess)
