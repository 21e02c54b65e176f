"""Small top-k, which looks at what reaches a bound from the threads' maxima: at the edges of k, of slices and of what a block can
list, with equal logits, and with the values that send a row the other way."""
import numpy as np
import pytest
import torch

from test_gpu_sampler_rows import _check, _rows

pytestmark = pytest.mark.gpu


# rows and columns: eight, four, two blocks a row and one; 16-byte rows and odd ones (last slices that end inside a group of four, or are empty)
@pytest.mark.parametrize("B,V", [(3, 151936), (2, 1003), (160, 60003), (150, 32000), (300, 8001)])
@pytest.mark.parametrize("k", [1, 2, 50, 128, 129, 256, 257])
def test_edges_of_k(B, V, k):
    rng = np.random.default_rng(V + k)
    x = rng.standard_normal((B, V)).astype(np.float32) * 3
    _check(torch.from_numpy(x), V, np.float32([0.8] * B), np.int32([k] * B), np.float32(rng.choice([0.9, 1.0], B)), np.zeros(B, np.float32), rng)


@pytest.mark.parametrize("kind", ["ties", "level", "two levels", "masked", "spikes", "nan", "many nans", "inf", "minus inf", "zeros"])
@pytest.mark.parametrize("B,V", [(4, 40000), (300, 4096)])
def test_rows_that_offer_too_much_or_the_wrong_thing(kind, B, V):
    rng = np.random.default_rng(len(kind) + V)
    x = _rows(kind, B, V, rng)
    if kind == "ties":
        x = np.round(x * 4) / 4                              # hundreds of elements level with the k-th
    elif kind == "level":
        x[:] = 1.5
    elif kind == "two levels":
        x[:] = -1.0
        x[:, ::97] = 2.0                                     # more than k and more than a block lists, and nothing between
    elif kind == "nan":
        x[:, [5, V // 2]] = np.nan
    elif kind == "many nans":
        x[:, ::50] = np.nan
    elif kind == "minus inf":
        x[:, 7:] = -np.inf
    elif kind == "zeros":
        x = np.where(x > 0, 0.0, -0.0).astype(np.float32)
        x[:, 11] = 1e-30
    k = 20
    if kind == "inf":                                        # no probabilities: any token of the row, as before
        from vllm_ascend_b200 import ops
        x[:, 3] = np.inf
        out = ops.sample(torch.from_numpy(x).cuda(), torch.full((B,), 0.8, device="cuda"), torch.full((B,), k, dtype=torch.int32, device="cuda"),
                         torch.ones(B, device="cuda"), None, torch.arange(B, device="cuda"), torch.arange(B, device="cuda"))
        assert bool(((out >= 0) & (out < V)).all())
        return
    _check(torch.from_numpy(x), V, np.float32([0.7] * B), np.int32([k] * B), np.float32([0.9, 1.0] * (B // 2)), np.zeros(B, np.float32), rng)
