"""Chunked gated delta rule against its definition in fp64, and against the token-serial kernel's distance from it.

State and sums are 32-bit in both kernels: what the state is off by is a few 2^-24 of its largest terms per chunk or token.  The
test allows 4e-6 of the state's norm, and no more than one and a half times the token-serial kernel's error where that is
larger; read-outs are rounded to bf16 (2^-9)."""
import numpy as np
import pytest
import torch

from vllm_ascend_b200 import _native
from vllm_ascend_b200.ops import linear_attn as la

pytestmark = pytest.mark.gpu
DEV = "cuda"


def _exact(q, k, v, g, beta, state, cu, slots, init, scale, l2norm):
    q, k, v, g, beta, out = *(t.double() for t in (q, k, v, g, beta)), torch.zeros(v.shape, dtype=torch.float64, device=DEV)
    S = state.double()
    if l2norm:
        q, k = (x * torch.rsqrt((x * x).sum(-1, keepdim=True) + 1e-6) for x in (q, k))
    rep = v.shape[1] // q.shape[1]
    q, k = q.repeat_interleave(rep, 1) * scale, k.repeat_interleave(rep, 1)
    for b in range(len(slots)):
        if cu[b + 1] == cu[b]:
            continue
        s = S[slots[b]] if init[b] else torch.zeros_like(S[0])
        for t in range(cu[b], cu[b + 1]):
            s = s * g[t].exp()[:, None, None]
            u = (v[t] - torch.einsum("hkv,hk->hv", s, k[t])) * beta[t][:, None]
            s = s + k[t][..., None] * u[:, None]
            out[t] = torch.einsum("hkv,hk->hv", s, q[t])
        S[slots[b]] = s
    return out, S


def _err(a, b):
    return float((a.double() - b).norm() / b.norm())


@pytest.mark.parametrize("Hk,Hv,DV,lens,decay,l2norm", [
    (1, 2, 128, [64], 0.3, True), (2, 4, 128, [1, 31, 32, 63, 65, 128, 0, 200], 0.3, True), (1, 1, 64, [127, 40], 2.0, True),
    (2, 2, 192, [129, 3], 20.0, True), (1, 2, 256, [66], 0.01, False), (16, 32, 128, [150, 90, 33], 0.9, True)])
def test_chunks_against_the_definition(monkeypatch, Hk, Hv, DV, lens, decay, l2norm):
    gen = torch.Generator(device=DEV).manual_seed(sum(lens) + DV)
    T, B = sum(lens), len(lens)
    cu_h = [sum(lens[:i]) for i in range(B + 1)]

    def rnd(*s):
        return torch.randn(*s, device=DEV, generator=gen)
    rows = rnd(T, (2 * Hk) * 128 + Hv * DV + 16).bfloat16() * (1.0 if l2norm else 0.08)        # q | k | v in one row, as layers have them
    q, k = rows[:, :Hk * 128].view(T, Hk, 128), rows[:, Hk * 128:2 * Hk * 128].view(T, Hk, 128)
    v = rows[:, 2 * Hk * 128:2 * Hk * 128 + Hv * DV].view(T, Hv, DV)
    g = -torch.rand(T, Hv, device=DEV, generator=gen) * decay
    g[T // 2] = -300.0                                           # a token that forgets everything before it
    beta = torch.rand(T, Hv, device=DEV, generator=gen)
    S0 = rnd(B + 2, Hv, 128, DV) * 0.1
    slots_h, init_h = [B - i for i in range(B)], [i % 2 for i in range(B)]
    cu, slots, init = (torch.tensor(x, dtype=torch.int32, device=DEV) for x in (cu_h, slots_h, init_h))
    want, S_want = _exact(q, k, v, g, beta, S0, cu_h, slots_h, init_h, 128 ** -0.5, l2norm)
    errors = {}
    for way in ("chunks", "tokens"):
        if way == "tokens":
            monkeypatch.setenv("VLLM_B200_GDN_CHUNK_MIN", "0")
        S = S0.clone()
        launches = _native.launch_counter[0]
        out = la.gated_delta_rule(q, k, v, g, beta, S, cu, slots, init, 128 ** -0.5, l2norm, cu_cpu=cu_h)
        assert _native.launch_counter[0] - launches == 1 + (way == "chunks" and any(0 < n < 32 for n in lens) and max(lens) >= 32)
        _native.check_status(torch.device(DEV))
        untouched = [i for i in range(B + 2) if i not in slots_h or lens[slots_h.index(i)] == 0]
        assert torch.equal(S[untouched], S0[untouched])
        errors[way] = (_err(out, want), _err(S, S_want))
    assert errors["chunks"][0] < 2.0 ** -8
    assert errors["chunks"][1] < max(4e-6, 1.5 * errors["tokens"][1]), errors


def test_prompt_in_two_portions_continues_its_state():
    gen = torch.Generator(device=DEV).manual_seed(1)
    T, H = 190, 2
    q, k, v = (torch.randn(T, H, 128, device=DEV, generator=gen).bfloat16() for _ in range(3))
    g, beta = -torch.rand(T, H, device=DEV, generator=gen), torch.rand(T, H, device=DEV, generator=gen)
    slot = torch.zeros(1, dtype=torch.int32, device=DEV)
    whole, parts = torch.zeros(1, H, 128, 128, device=DEV), torch.ones(1, H, 128, 128, device=DEV)

    def run(a, b, S, init):
        cu = torch.tensor([0, b - a], dtype=torch.int32, device=DEV)
        return la.gated_delta_rule(q[a:b], k[a:b], v[a:b], g[a:b], beta[a:b], S, cu, slot, slot + init, 128 ** -0.5, cu_cpu=[0, b - a])
    o = run(0, T, whole, 0)
    o2 = torch.cat([run(0, 70, parts, 0), run(70, 80, parts, 1), run(80, T, parts, 1)])
    assert _err(parts, whole.double()) < 4e-6
    assert _err(o2, o.double()) < 2.0 ** -8


@pytest.mark.parametrize("form", ["fp32", "DK64", "odd rows", "unaligned"])
def test_other_forms_stay_token_by_token(form):
    T, H, DK = 70, 1, 64 if form == "DK64" else 128
    dt = torch.float32 if form == "fp32" else torch.bfloat16
    gen = torch.Generator(device=DEV).manual_seed(2)
    extra = 3 if form == "odd rows" else 8
    wide = torch.randn(T, 3 * H * DK + extra, device=DEV, generator=gen).to(dt)
    at = 4 if form == "unaligned" else 0
    q, k, v = (wide[:, at + i * DK:at + (i + 1) * DK].view(T, H, DK) for i in range(3))
    g, beta = -torch.rand(T, H, device=DEV, generator=gen), torch.rand(T, H, device=DEV, generator=gen)
    S0 = torch.randn(1, H, DK, DK, device=DEV, generator=gen)
    cu, slot = torch.tensor([0, T], dtype=torch.int32, device=DEV), torch.zeros(1, dtype=torch.int32, device=DEV)
    S = S0.clone()
    out = la.gated_delta_rule(q, k, v, g, beta, S, cu, slot, slot + 1, DK ** -0.5, cu_cpu=[0, T])
    want, S_want = _exact(q, k, v, g, beta, S0, [0, T], [0], [1], DK ** -0.5, True)
    assert _err(S, S_want) < 4e-6 and _err(out, want) < 2.0 ** -8


def test_many_short_portions_share_out_between_the_kernels():
    """A step whose portions of 32 and more tokens run in chunks and shorter ones in the other kernel, and one whose 65-token portions
    go token by token: the states and read-outs of both kernels side by side, each its own sequences."""
    gen = torch.Generator(device=DEV).manual_seed(5)
    for lens in ([39, 40, 64, 3] * 4, [65] * 12 + [200] * 3):
        Hk, Hv, DV, T, B = 32, 32, 128, sum(lens), len(lens)
        cu_h = [sum(lens[:i]) for i in range(B + 1)]
        q, k, v = (torch.randn(T, h, 128, device=DEV, generator=gen).bfloat16() for h in (Hk, Hk, Hv))
        g, beta = -torch.rand(T, Hv, device=DEV, generator=gen), torch.rand(T, Hv, device=DEV, generator=gen)
        S0 = torch.randn(B, Hv, 128, DV, device=DEV, generator=gen) * 0.1
        slots_h, init_h = list(range(B)), [1] * B
        cu, slots, init = (torch.tensor(x, dtype=torch.int32, device=DEV) for x in (cu_h, slots_h, init_h))
        want, S_want = _exact(q, k, v, g, beta, S0, cu_h, slots_h, init_h, 128 ** -0.5, True)
        S = S0.clone()
        launches = _native.launch_counter[0]
        out = la.gated_delta_rule(q, k, v, g, beta, S, cu, slots, init, 128 ** -0.5, True, cu_cpu=cu_h)
        assert _native.launch_counter[0] - launches == 2
        _native.check_status(torch.device(DEV))
        assert _err(out, want) < 2.0 ** -8 and _err(S, S_want) < 4e-6


@pytest.mark.parametrize("at", [0, 5, 63, 70])
def test_a_nan_reaches_no_earlier_token(at):
    """Causality holds for values that no product with zero removes: rows before a NaN are what they are without it, bit for bit."""
    gen = torch.Generator(device=DEV).manual_seed(at)
    T, H = 100, 2
    q, k, v = (torch.randn(T, H, 128, device=DEV, generator=gen).bfloat16() for _ in range(3))
    g, beta = -torch.rand(T, H, device=DEV, generator=gen), torch.rand(T, H, device=DEV, generator=gen)
    cu, slot = torch.tensor([0, T], dtype=torch.int32, device=DEV), torch.zeros(1, dtype=torch.int32, device=DEV)

    def run(v):
        S = torch.zeros(1, H, 128, 128, device=DEV)
        return la.gated_delta_rule(q, k, v, g, beta, S, cu, slot, slot, 128 ** -0.5, cu_cpu=[0, T]).view(T, H, 128), S
    assert la._portions(np.asarray([0, T], np.int32).tobytes(), H, 128, _native.sm_count(torch.device(DEV)))[0] > 0
    clean, _ = run(v)
    v = v.clone()
    v[at, 0, 3] = float("nan")
    out, S = run(v)
    assert torch.equal(out[:at], clean[:at]) and torch.equal(out[:, 1], clean[:, 1])
    assert out[at:, 0, 3].isnan().all() and S[0, 0, :, 3].isnan().all()
    others = [c for c in range(128) if c != 3]
    assert torch.equal(out[:, 0, others], clean[:, 0, others])
