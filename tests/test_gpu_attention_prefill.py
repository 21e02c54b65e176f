"""Prompt attention kernel (both forms) against fp64 attention over the same keys: edges of the 128-row tiles and of the pair
of tiles a block owns, group sizes, page sizes, cache layouts, windows, contexts, decodes in front of prompts.

Bound: probabilities are rounded to bf16 (2^-9 relative each, random signs) before they weight values of unit size, the
result is rounded to bf16; scores carry fp32 sums of D products.  3 x 2^-8 of the values' size holds with room."""
import numpy as np
import pytest
import torch

from vllm_ascend_b200 import _native, ops
from vllm_ascend_b200.attention import mla
from vllm_ascend_b200.attention.metadata import metadata_from_tensors

pytestmark = pytest.mark.gpu
DEV = "cuda"


def _want(q, k, v, old, scale, window=0, causal=True):
    n, H = q.shape[:2]
    kp, qp = torch.arange(k.shape[0], device=DEV)[None], old + torch.arange(n, device=DEV)[:, None]
    off = (kp > qp) & causal
    if window:
        off |= kp <= qp - window
    out = []
    for h in range(H):
        s = (q[:, h].double() @ k[:, h * k.shape[1] // H].double().t() * scale).masked_fill(off, float("-inf"))
        out.append(torch.softmax(s, -1) @ v[:, h * v.shape[1] // H].double())
    return torch.stack(out, 1)


def _batch(new, old, page, g):
    pages = [-(-(n + o) // page) for n, o in zip(new, old)]
    order = torch.randperm(sum(pages), generator=g) + 1
    table = torch.zeros((len(new), max(pages) + 1), dtype=torch.int32)
    at = 0
    for b, n in enumerate(pages):
        table[b, :n] = order[at:at + n]
        at += n
    cu = torch.tensor([0] + list(np.cumsum(new)), dtype=torch.int32)
    lens = torch.tensor([n + o for n, o in zip(new, old)], dtype=torch.int32)
    return table.to(DEV), cu.to(DEV), lens.to(DEV), sum(pages) + 1


def _rows(cache, table, n, page):
    p = torch.arange(n, device=DEV)
    return cache[table.long()[p // page], p % page]


@pytest.mark.parametrize("G,page,layout,window", [(1, 128, "HND", 0), (4, 128, "HND", 0), (4, 16, "NHD", 0), (8, 256, "HND", 100), (16, 64, "NHD", 0),
                                                  (2, 128, "HND", 1)])
def test_paged_prompts(G, page, layout, window):
    g = torch.Generator().manual_seed(G * page)
    tile = 128 // G
    new = [1, tile - 1, tile, tile + 1, 2 * tile, 2 * tile + 1, 300, 3]
    old = [0, 5, 0, 200, 129, 0, 77, 640]
    Hkv, D = 2, 128
    table, cu, lens, blocks = _batch(new, old, page, g)
    k = ops.alloc_kv_cache(blocks, page, Hkv, D, torch.bfloat16, DEV, layout)
    v = ops.alloc_kv_cache(blocks, page, Hkv, D, torch.bfloat16, DEV, layout)
    k.copy_(torch.randn(k.shape, generator=g).to(DEV))
    v.copy_(torch.randn(v.shape, generator=g).to(DEV))
    T = sum(new)
    wide = torch.randn((T, Hkv * G * D + 64), generator=g).to(DEV).bfloat16()
    q = wide[:, :Hkv * G * D].view(T, Hkv * G, D)
    meta = metadata_from_tensors(cu, lens, table, max(new), int(lens.max()), Hkv * G, Hkv, D, decode_kernel=False)
    out = torch.full((T, Hkv * G, D), float("nan"), device=DEV, dtype=torch.bfloat16)
    ops.paged_prefill_attention(q, k, v, meta, D ** -0.5, out, True, window)
    _native.check_status(torch.device(DEV))
    at = 0
    for b, (n, o) in enumerate(zip(new, old)):
        want = _want(q[at:at + n], _rows(k, table[b], n + o, page), _rows(v, table[b], n + o, page), o, D ** -0.5, window)
        assert ((out[at:at + n].double() - want).abs() <= 3 * 2.0 ** -8 * (1 + want.abs())).all(), (b, n, o)
        at += n


@pytest.mark.parametrize("causal", [True, False])
def test_sequences_without_keys_leave_their_rows_alone(causal):
    """Query rows of sequences that have no keys (padding, an encoder without output) between ones that have; and fewer keys than
    queries, where causal rows in front of the first key see none."""
    g = torch.Generator().manual_seed(9)
    Hkv, G, D, page = 8, 4, 128, 128
    new, keys = [300, 700, 40, 1500], [0, 650, 0, 1500]
    table, cu, lens, blocks = _batch([1] * 4, [max(n - 1, 0) for n in keys], page, g)
    cu, lens = (torch.tensor(x, dtype=torch.int32, device=DEV) for x in ([0] + list(np.cumsum(new)), keys))
    k, v = (ops.alloc_kv_cache(blocks, page, Hkv, D, torch.bfloat16, DEV) for _ in range(2))
    for c in (k, v):
        c.copy_(torch.randn(c.shape, generator=g).to(DEV))
    q = torch.randn((sum(new), Hkv * G, D), generator=g).to(DEV).bfloat16()
    meta = metadata_from_tensors(cu, lens, table, max(new), max(keys), Hkv * G, Hkv, D, decode_kernel=False)
    out = torch.full(q.shape, 7.0, device=DEV, dtype=torch.bfloat16)
    ops.paged_prefill_attention(q, k, v, meta, D ** -0.5, out, causal)
    _native.check_status(torch.device(DEV))
    at = 0
    for b, (n, m) in enumerate(zip(new, keys)):
        got = out[at:at + n]
        if m == 0:
            assert (got == 7.0).all(), b
        else:
            first = max(n - m, 0) if causal else 0             # rows that see a key
            want = _want(q[at:at + n], _rows(k, table[b], m, page), _rows(v, table[b], m, page), m - n, D ** -0.5, causal=causal)[first:]
            assert ((got[first:].double() - want).abs() <= 3 * 2.0 ** -8 * (1 + want.abs())).all(), b
        at += n


def test_mixed_step_gives_decodes_and_prompts_their_rows():
    g = torch.Generator().manual_seed(5)
    new, old = [1, 1, 1, 7300, 130], [300, 5, 129, 0, 64]         # enough tiles for the kernel of pairs
    Hkv, G, D, page = 2, 4, 128, 128
    table, cu, lens, blocks = _batch(new, old, page, g)
    k, v = (ops.alloc_kv_cache(blocks, page, Hkv, D, torch.bfloat16, DEV) for _ in range(2))
    k.copy_(torch.randn(k.shape, generator=g).to(DEV))
    v.copy_(torch.randn(v.shape, generator=g).to(DEV))
    q = torch.randn((sum(new), Hkv * G, D), generator=g).to(DEV).bfloat16()
    meta = metadata_from_tensors(cu, lens, table, max(new), int(lens.max()), Hkv * G, Hkv, D)
    assert ops._prefill_pairs(q, Hkv, 3, meta, 3) == (torch.cuda.get_device_properties(0).multi_processor_count <= 150)
    out = ops.paged_attention(q, k, v, meta, D ** -0.5)
    at = 0
    for b, (n, o) in enumerate(zip(new, old)):
        want = _want(q[at:at + n], _rows(k, table[b], n + o, page), _rows(v, table[b], n + o, page), o, D ** -0.5)
        assert ((out[at:at + n].double() - want).abs() <= 3 * 2.0 ** -8 * (1 + want.abs())).all(), (b, n, o)
        at += n


@pytest.mark.parametrize("H,dc,dr,dv,page", [(3, 512, 64, 128, 128), (1, 64, 16, 72, 16), (4, 128, 64, 64, 64)])
def test_latent_prompts(H, dc, dr, dv, page):
    g = torch.Generator().manual_seed(H + dc)
    dn, new, old = 128, [127, 128, 129, 256, 257, 40], [0, 130, 0, 7, 0, 300]
    first = 2                                                    # one-token sequences in front: not this function's rows
    table, cu, lens, blocks = _batch([1] * first + new, [9, 300] + old, page, g)
    lat = torch.randn((blocks, page, 1, dc), generator=g).to(DEV).bfloat16()
    pe = torch.randn((blocks, page, 1, dr), generator=g).to(DEV).bfloat16()
    kv_b = (torch.randn((H * (dn + dv), dc), generator=g) * dc ** -0.5).to(DEV).bfloat16()
    q = torch.randn((first + sum(new), H, dn + dr), generator=g).to(DEV).bfloat16()
    meta = metadata_from_tensors(cu, lens, table, max(new), int(lens.max()), H, H, 128, decode_kernel=False)
    plan = mla.expanded_prompts(meta, H, dn, dr, dv, q, lat, pe)
    assert plan == (first, sum(new) + sum(old))
    out = torch.full((q.shape[0], H, dv), float("nan"), device=DEV, dtype=torch.bfloat16)
    scale = (dn + dr) ** -0.5
    mla.prompt_attention_expanded(q, kv_b, lat, pe, meta, scale, dv, *plan, out)
    _native.check_status(torch.device(DEV))
    assert out[:first].isnan().all()
    at = first
    for b, (n, o) in enumerate(zip(new, old)):
        t = table[first + b]
        kv = (_rows(lat, t, n + o, page)[:, 0].double() @ kv_b.double().t()).view(n + o, H, dn + dv)
        # keys and values are rounded to bf16 once: another 2^-9 of values of unit size, and of scores of unit size
        k = torch.cat([kv[..., :dn].bfloat16().double(), _rows(pe, t, n + o, page).double().expand(-1, H, -1)], -1)
        want = _want(q[at:at + n], k, kv[..., dn:].bfloat16(), o, scale)
        assert ((out[at:at + n].double() - want).abs() <= 3 * 2.0 ** -8 * (1 + want.abs())).all(), (b, n, o)
        at += n


def test_rule_keeps_decodes_and_long_contexts_in_the_latent_space():
    def plan(new, old, **kw):
        table, cu, lens, blocks = _batch(new, old, 128, torch.Generator().manual_seed(0))
        meta = metadata_from_tensors(cu, lens, table, max(new), int(lens.max()), 2, 2, 128, decode_kernel=False)
        q = torch.zeros((sum(new), 2, kw.get("dn", 128) + 64), device=DEV, dtype=kw.get("dtype", torch.bfloat16))
        lat, pe = (torch.zeros((blocks, 128, 1, d), device=DEV, dtype=q.dtype) for d in (512, 64))
        return mla.expanded_prompts(meta, kw.get("heads", 2), kw.get("dn", 128), 64, 128, q, lat, pe)
    assert plan([1, 1], [40, 50]) is None
    assert plan([8], [4000]) is None                              # 8 pairs per key
    assert plan([64], [4000]) == (0, 4064)
    assert plan([64], [0], dn=64) is None
    assert plan([64], [0], dtype=torch.float32) is None
    assert plan([1000], [0], heads=1 << 12) is None              # 2 GB of projected rows


@pytest.mark.parametrize("H", [1, 16])
def test_workspace_stays_within_its_limit(monkeypatch, H):
    """What a step allocates beside its output is what the plan was allowed: projected rows, dense latents and rotary keys together."""
    dn, dr, dv, dc, n = 128, 64, 128, 512, 20000
    monkeypatch.setattr(mla, "_EXPAND_BYTES", n * 2 * (H * (dn + dv) + dc + dr))
    for keys in (n, n + 1):
        table, cu, lens, blocks = _batch([keys], [0], 128, torch.Generator().manual_seed(0))
        meta = metadata_from_tensors(cu, lens, table, keys, keys, H, H, 128, decode_kernel=False)
        q = torch.zeros((keys, H, dn + dr), device=DEV, dtype=torch.bfloat16)
        lat, pe = (torch.zeros((blocks, 128, 1, d), device=DEV, dtype=q.dtype) for d in (dc, dr))
        plan = mla.expanded_prompts(meta, H, dn, dr, dv, q, lat, pe)
        assert plan == ((0, n) if keys == n else None)
        if plan is None:
            continue
        kv_b = torch.zeros((H * (dn + dv), dc), device=DEV, dtype=q.dtype)
        out = torch.empty((keys, H, dv), device=DEV, dtype=q.dtype)
        torch.cuda.synchronize()
        torch.cuda.reset_peak_memory_stats()
        before = torch.cuda.memory_allocated()
        mla.prompt_attention_expanded(q, kv_b, lat, pe, meta, 0.1, dv, *plan, out)
        _native.check_status(torch.device(DEV))
        assert torch.cuda.max_memory_allocated() - before <= mla._EXPAND_BYTES + (4 << 20)     # allocations are rounded up


def test_many_sequences_start_where_the_ones_before_end():
    n = 2500
    lens = torch.randint(1, 4, (n,), generator=torch.Generator().manual_seed(1), dtype=torch.int32)
    keys = int(lens.sum())
    lat, pe = torch.randn(n, 4, 8).to(DEV).bfloat16(), torch.randn(n, 4, 8).to(DEV).bfloat16()
    table = torch.randperm(n, dtype=torch.int32).view(n, 1).to(DEV)
    starts = torch.empty(n + 1, dtype=torch.int32, device=DEV)
    a, b = (torch.empty((keys, 8), dtype=torch.bfloat16, device=DEV) for _ in range(2))
    dl = lens.to(DEV)
    _native.check(_native.lib().b200_gather_latents(
        lat.data_ptr(), pe.data_ptr(), 8, 8, 4, n, dl.data_ptr(), table.data_ptr(), 1, n, keys, starts.data_ptr(), a.data_ptr(),
        b.data_ptr(), _native.status_word(torch.device(DEV)).data_ptr(), _native.stream_ptr()), "gather_latents")
    assert starts.tolist() == [0] + lens.cumsum(0).tolist()
    seq = torch.repeat_interleave(torch.arange(n), lens.long()).to(DEV)
    pos = torch.arange(keys, device=DEV) - starts[:-1].long()[seq]
    assert torch.equal(a, lat[table[seq, 0].long(), pos]) and torch.equal(b, pe[table[seq, 0].long(), pos])
    _native.check_status(torch.device(DEV))


@pytest.mark.parametrize("new,old,Hkv,G,pairs", [([2048], 0, 8, 4, True), ([137], 0, 8, 4, False), ([16] * 100, 4000, 8, 4, False), ([33] * 256, 0, 8, 8, True),
                                                 ([100] * 20 + [3000], 100, 1, 8, False), ([700] * 8, 0, 1, 8, False), ([700] * 8, 0, 8, 4, True)])
def test_rule_counts_waves_and_empty_halves(monkeypatch, new, old, Hkv, G, pairs):
    """What runs in pairs, and the same rows from either kernel: probabilities and results are rounded to bf16 in both."""
    g = torch.Generator().manual_seed(len(new))
    D, page = 128, 128
    table, cu, lens, blocks = _batch(new, [old] * len(new), page, g)
    k, v = (ops.alloc_kv_cache(blocks, page, Hkv, D, torch.bfloat16, DEV) for _ in range(2))
    for c in (k, v):
        c.copy_(torch.randn(c.shape, dtype=torch.bfloat16, generator=g).to(DEV))
    q = torch.randn((sum(new), Hkv * G, D), generator=g).to(DEV).bfloat16()
    meta = metadata_from_tensors(cu, lens, table, max(new), int(lens.max()), Hkv * G, Hkv, D)
    if torch.cuda.get_device_properties(0).multi_processor_count == 148:
        assert ops._prefill_pairs(q, Hkv, 0, meta) == pairs
    rows = []
    for choice in (True, False):
        monkeypatch.setattr(ops, "_prefill_pairs", lambda *a: choice)
        rows.append(ops.paged_attention(q, k, v, meta, D ** -0.5).double())
    assert ((rows[0] - rows[1]).abs() <= 6 * 2.0 ** -8 * (1 + rows[1].abs())).all()
    _native.check_status(torch.device(DEV))
