"""The chunked delta rule's workspace in slices, and values that no product with zero removes."""
import pytest
import torch

from vllm_ascend_b200 import _native
from vllm_ascend_b200.ops import linear_attn as la

pytestmark = pytest.mark.gpu
DEV = "cuda"


def _inputs(lens, Hk, Hv, DV, seed):
    gen = torch.Generator(device=DEV).manual_seed(seed)
    T, B = sum(lens), len(lens)
    cu_h = [sum(lens[:i]) for i in range(B + 1)]
    q, k, v = (torch.randn(T, h, d, device=DEV, generator=gen).bfloat16() for h, d in ((Hk, 128), (Hk, 128), (Hv, DV)))
    g, beta = -torch.rand(T, Hv, device=DEV, generator=gen), torch.rand(T, Hv, device=DEV, generator=gen)
    S = torch.randn(B, Hv, 128, DV, device=DEV, generator=gen) * 0.1
    return q, k, v, g, beta, S, cu_h


def _run(q, k, v, g, beta, S, cu_h, init=None):
    B = len(cu_h) - 1
    cu, slots = torch.tensor(cu_h, dtype=torch.int32, device=DEV), torch.arange(B, dtype=torch.int32, device=DEV)
    init = torch.tensor([i % 2 for i in range(B)] if init is None else init, dtype=torch.int32, device=DEV)
    S = S.clone()
    out = la.gated_delta_rule(q, k, v, g, beta, S, cu, slots, init, 128 ** -0.5, cu_cpu=cu_h)
    _native.check_status(torch.device(DEV))
    return out, S


@pytest.mark.parametrize("lens", [[640], [64, 63, 1, 129, 128, 65, 200], [75, 1000]])
@pytest.mark.parametrize("DV", [64, 192])
@pytest.mark.parametrize("chunks", [1, 2, 5])
def test_slices_give_the_same_bits(monkeypatch, lens, DV, chunks):
    x = _inputs(lens, 1, 2, DV, sum(lens))
    whole = _run(*x)
    monkeypatch.setattr(la, "_CHUNK_WORKSPACE", chunks * len(lens) * 2 * la._CHUNK_PLACE)
    parts = _run(*x)
    assert torch.equal(whole[0], parts[0]) and torch.equal(whole[1], parts[1])


@pytest.mark.parametrize("what", ["v", "k", "q", "g", "beta", "state"])
@pytest.mark.parametrize("bad", [float("nan"), float("inf")])
def test_bad_values_stay_with_their_tokens(what, bad):
    """A NaN or infinity at token 70 leaves earlier tokens' bits and other heads alone, and the next sequence too (whose tokens
    follow its last, partial chunk)."""
    lens, at = [100, 90], 70
    q, k, v, g, beta, S, cu = _inputs(lens, 2, 2, 128, 3)
    clean, S_clean = _run(q, k, v, g, beta, S, cu, [1, 1])
    t = dict(q=q, k=k, v=v, g=g, beta=beta, state=S)[what].clone()
    if what == "state":
        t[0, 0, 5, 9] = bad
    elif what in ("g", "beta"):
        t[at, 0] = bad
    else:
        t[at, 0, 3] = bad
    args = dict(q=q, k=k, v=v, g=g, beta=beta, S=S, **{})
    args["S" if what == "state" else what] = t
    out, S_out = _run(*args.values(), cu, [1, 1])
    first = 0 if what == "state" else at
    assert torch.equal(out[:first], clean[:first]) and torch.equal(out[:, 1], clean[:, 1])
    assert torch.equal(out[100:], clean[100:]) and torch.equal(S_out[1], S_clean[1])
    if what == "q":
        assert torch.equal(out[at + 1:], clean[at + 1:]) and torch.equal(S_out, S_clean)
    elif not (what == "g" and bad > 0):
        assert not out[at:100, 0].isfinite().all()


def test_a_full_gpu_repeats_its_bits():
    """192 blocks of 35 to 47 chunks, two on an SM: what a thread ahead of others overwrites shows as bits that differ from run to run, or
    as read-outs that are off by more than the other kernel's rounding."""
    x = _inputs([2300, 1700, 3000], 4, 32, 128, 9)
    first = _run(*x)
    for _ in range(12):
        again = _run(*x)
        assert torch.equal(first[0], again[0]) and torch.equal(first[1], again[1])
    q, k, v, g, beta, S, cu = x
    slots, init = torch.arange(3, dtype=torch.int32, device=DEV), torch.tensor([0, 1, 0], dtype=torch.int32, device=DEV)
    want = la.gated_delta_rule(q, k, v, g, beta, S.clone(), torch.tensor(cu, dtype=torch.int32, device=DEV), slots, init, 128 ** -0.5)
    # two roundings to bf16 of sums that differ by a few 2^-24 of their terms
    assert bool(((first[0].float() - want.float()).abs() <= 2.0 ** -7 * want.float().abs() + 2.0 ** -16).all())
