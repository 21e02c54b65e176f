"""Sampling kernel against its definition in numpy: kept set by sorting in fp64, random numbers by Philox4x32-10, race of
p / Exp(1).  Rows of every storage form (in the cluster's shared memory, too long for it, unaligned) and of every shape
that chooses another cut (peaked, flat, masked, fewer large elements than top-k)."""
import numpy as np
import pytest
import torch

from vllm_ascend_b200 import _native, ops

pytestmark = pytest.mark.gpu


def _philox(ctr, key):
    M0, M1, W0, W1 = (np.uint64(v) for v in (0xD2511F53, 0xCD9E8D57, 0x9E3779B9, 0xBB67AE85))
    m = np.uint64(0xFFFFFFFF)
    x, y, z, w = (np.asarray(c, dtype=np.uint64) for c in ctr)
    k0, k1 = np.uint64(key & 0xFFFFFFFF), np.uint64(key >> 32)
    for _ in range(10):
        a, b = M0 * x, M1 * z
        x, y, z, w = (b >> np.uint64(32)) ^ y ^ k0, b & m, (a >> np.uint64(32)) ^ w ^ k1, a & m
        k0, k1 = (k0 + W0) & m, (k1 + W1) & m
    return np.stack([x, y, z, w], -1)


#: largest error of the fast logarithm between 0.5 and 2, as CUDA documents it: where u is near 1, -log u has no more digits
LOG_ERROR = 2.0 ** -21


#: by how much the kernel's fp32 exponentials and sums may move a cut (relative)
CUT_ERROR = 1e-5


def _expected(row, T, k, p, min_p, seed, offset):
    """Tokens that the race may give: winners over what any cut within CUT_ERROR of the asked one keeps.  NaN logits are never
    chosen, rank above all others, and leave no mass to take a share of."""
    x = row.astype(np.float64)
    nans = np.isnan(x)
    if T < 1e-5:
        return [int(np.nanargmax(x))]
    e = np.where(nans, 0, np.exp((x - x[~nans].max()) / T))
    order = np.argsort(-e, kind="stable")
    surely, maybe = ~nans, ~nans                # kept by every cut in question, by some
    if 0 < k < len(x):
        last = e[order[max(k - nans.sum(), 1) - 1]] if k > nans.sum() else np.inf
        surely, maybe = surely & (e >= last * (1 + 1e-6)), maybe & (e >= last * (1 - 1e-6))
    if p < 1 and not nans.any():
        ks = order[(maybe & (e >= (last if 0 < k < len(x) else 0)))[order]]
        cum = np.cumsum(e[ks])
        lo, hi = (e[ks[min(int(np.searchsorted(cum, p * f * cum[-1])), len(ks) - 1)]] for f in (1 - CUT_ERROR, 1 + CUT_ERROR))
        surely, maybe = surely & (e >= lo * (1 + 1e-6)), maybe & (e >= hi * (1 - 1e-6))
    if min_p > 0:
        surely, maybe = surely & (e >= min_p * (1 + CUT_ERROR)), maybe & (e >= min_p * (1 - CUT_ERROR))
    V = len(x)
    g = np.arange(0, V, 4)
    r = _philox((g, np.full_like(g, offset & 0xFFFFFFFF), np.full_like(g, offset >> 32), np.zeros_like(g)), seed).reshape(-1)[:V]
    ex = -np.log(((r >> np.uint64(8)).astype(np.float64) + 1) / 16777216)
    low = np.where(surely & (e > 0), e / (ex + LOG_ERROR) * (1 - 1e-5), -1)
    high = np.where(maybe & (e > 0), e / np.maximum(ex - LOG_ERROR, 1e-20) * (1 + 1e-5), -1)
    return np.nonzero((high >= low.max()) & (high > 0))[0].tolist() or [int(np.nanargmax(x))]


def _rows(kind, B, V, rng):
    x = rng.standard_normal((B, V)).astype(np.float32)
    if kind == "peaked":
        x *= 4
    elif kind == "flat":
        x *= 1e-2
    elif kind == "masked":
        x = np.where(rng.random((B, V)) < 0.98, -np.inf, x * 3).astype(np.float32)
        x[:, V // 2] = 1.0
    elif kind == "spikes":                       # three large elements, the rest below every cut
        x -= 60
        x[:, [0, V // 3, V - 1]] += 60
    return x


def _check(wide, V, T, k, p, mp, rng):
    B = wide.shape[0]
    logits = wide.cuda()[:, :V]
    seeds = rng.integers(0, 1 << 62, B)
    offsets = rng.integers(0, 1 << 34, B)
    host = logits.cpu().numpy()
    got = ops.sample(logits, torch.tensor(T).cuda(), torch.tensor(k, dtype=torch.int32).cuda(), torch.tensor(p).cuda(),
                     torch.tensor(mp).cuda(), torch.from_numpy(seeds).cuda(), torch.from_numpy(offsets).cuda()).cpu().tolist()
    _native.check_status(torch.device("cuda"))
    for b in range(B):
        want = _expected(host[b], T[b], k[b], p[b], mp[b], int(seeds[b]), int(offsets[b]))
        assert got[b] in want, (b, got[b], want)


@pytest.mark.parametrize("V,pad", [(5, 3), (31, 1), (4096, 0), (32000, 0), (50257, 3), (151936, 0), (409601, 1), (420004, 4)])
@pytest.mark.parametrize("kind", ["peaked", "flat", "masked", "spikes"])
def test_sample_is_the_race_over_the_kept_set(V, pad, kind):
    rng = np.random.default_rng(V)
    B = 6
    wide = torch.zeros((B, V + pad))
    wide[:, :V] = torch.from_numpy(_rows(kind, B, V, rng))
    T = [0.0, 0.7, 1.0, 1.3, 0.9, 1.0]
    k = [5, 3, min(50, V), 0, 0, V]
    p = [0.9, 1.0, 0.9, 0.8, 0.97, 1.0]
    mp = [0.0, 0.0, 0.0, 0.0, 0.013, 0.0]
    _check(wide, V, T, k, p, mp, rng)


@pytest.mark.parametrize("B,V,pad", [(38, 4099, 2), (75, 22000, 0), (80, 70, 0), (149, 3, 5), (150, 5003, 1), (150, 23000, 0)])
def test_more_rows_take_fewer_blocks_each(B, V, pad):
    """Row counts from which a row has four, two and one block, with all shapes of rows and of requests mixed."""
    rng = np.random.default_rng(B + V)
    wide = torch.zeros((B, V + pad))
    for i, kind in enumerate(("peaked", "flat", "masked", "spikes")):
        wide[i::4, :V] = torch.from_numpy(_rows(kind, len(range(i, B, 4)), V, rng))
    pick = [(0.0, 5, 0.9, 0.0), (0.7, 3, 1.0, 0.0), (1.0, min(50, V), 0.9, 0.0), (1.3, 0, 0.8, 0.0), (0.9, 0, 0.97, 0.013), (1.0, V, 1.0, 0.0),
            (1.0, max(V * 2 // 3, 1), 0.999, 0.0)]
    T, k, p, mp = (list(c) for c in zip(*(pick[(b // 4) % len(pick)] for b in range(B))))
    _check(wide, V, T, k, p, mp, rng)


@pytest.mark.parametrize("B,V", [(6, 70), (6, 151936), (160, 5000)])
def test_nan_and_infinite_logits(B, V):
    """NaN is never chosen, an infinite logit always; what else a row asks for still ends, and other rows are not touched."""
    rng = np.random.default_rng(V)
    x = _rows("peaked", B, V, rng)
    x[0::6, rng.integers(0, V, 3)] = np.nan
    x[1::6, V // 2] = np.inf
    x[2::6, : V // 2] = -np.inf
    T, k, p = [(0.0, 1.0, 0.8, 1.0, 1.0)[b % 5] for b in range(B)], [(0, 0, 20, 0, 20)[b % 5] for b in range(B)], [(1.0, 1.0, 1.0, 0.9, 0.9)[b % 5] for b in range(B)]
    finite = [b for b in range(B) if b % 6 != 1]
    logits = torch.from_numpy(x).cuda()
    seeds, offsets = torch.arange(B).cuda(), torch.zeros(B, dtype=torch.int64).cuda()
    got = ops.sample(logits.clone(), torch.tensor(T).cuda(), torch.tensor(k, dtype=torch.int32).cuda(), torch.tensor(p).cuda(),
                     torch.zeros(B).cuda(), seeds, offsets).cpu().tolist()
    _native.check_status(torch.device("cuda"))
    assert [got[b] for b in range(1, B, 6)] == [V // 2] * len(range(1, B, 6))
    for b in finite:
        want = _expected(x[b], T[b], k[b], p[b], 0.0, b, 0)
        assert got[b] in want, (b, got[b], want)


@pytest.mark.parametrize("B,V,pad", [(65535, 8, 0), (65536, 3, 5), (131073, 9, 7), (3, 16385, 7), (4, 0, 0)])
def test_logits_become_fp32_row_by_row(B, V, pad):
    """More rows than a grid has in y, no columns, columns around a block's share."""
    x = torch.randn(B, V + pad, generator=torch.Generator().manual_seed(B)).bfloat16().cuda()[:, :V]
    assert torch.equal(ops.to_float_logits(x), x.float())


def test_threads_may_sample_rows_of_different_lengths():
    """Each thread on a stream of its own; how much shared memory the kernel may use does not depend on who asks first."""
    from concurrent.futures import ThreadPoolExecutor
    rows = [torch.randn(3, V, generator=torch.Generator().manual_seed(V)).cuda() for V in (700, 409601, 30000, 151936, 64, 262144) * 4]

    def sample(x):
        with torch.cuda.stream(torch.cuda.Stream()):
            n = x.shape[0]
            out = ops.sample(x.clone(), torch.ones(n).cuda(), torch.full((n,), 40, dtype=torch.int32).cuda(), torch.full((n,), 0.9).cuda(),
                             torch.zeros(n).cuda(), torch.arange(n).cuda(), torch.zeros(n, dtype=torch.int64).cuda())
            return out.cpu().tolist()
    torch.cuda.synchronize()
    with ThreadPoolExecutor(8) as pool:
        together = list(pool.map(sample, rows))
    assert together == [sample(x) for x in rows]
