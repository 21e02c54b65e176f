"""Batch invariance on the GPU: the value computed for a row must not depend on how many other rows
share the launch.  The GEMM kernels pick tile shapes (1-CTA / paired-CTA, tile width) from the problem
size; every shape accumulates an output element over K in one order, which is what these tests pin."""
import numpy as np
import pytest
import torch

from vllm_ascend_b200 import _native, ops

pytestmark = pytest.mark.gpu
DEV = "cuda"
SIZES = (1, 8, 100, 128, 255, 256, 300, 768, 1000, 2048, 4096)


@pytest.mark.parametrize("N,K", [(4096, 4096), (6144, 4096), (4096, 12288), (1536, 512)])
def test_gemm_rows_do_not_depend_on_the_row_count(N, K):
    g = torch.Generator(device="cpu").manual_seed(0)
    x = (torch.randn(4096, K, generator=g) * 0.5).bfloat16().to(DEV)
    w = (torch.randn(N, K, generator=g) * 0.05).bfloat16().to(DEV)
    bias = torch.randn(N, generator=g).bfloat16().to(DEV)
    full = ops.linear(x, w, bias)
    for m in SIZES:
        part = ops.linear(x[:m], w, bias)
        assert torch.equal(part, full[:m]), f"rows differ at M={m}"
    # rows taken from the middle of the batch as a batch of their own
    assert torch.equal(ops.linear(x[1000:1003].contiguous(), w, bias), full[1000:1003])
    torch.cuda.synchronize()
    _native.check_status(torch.device(DEV))


def test_swiglu_gemm_norm_and_activation_rows_do_not_depend_on_the_row_count():
    g = torch.Generator(device="cpu").manual_seed(1)
    K, I = 2048, 3072
    x = (torch.randn(2048, K, generator=g) * 0.5).bfloat16().to(DEV)
    w = (torch.randn(2 * I, K, generator=g) * 0.05).bfloat16().to(DEV)
    nw = torch.rand(K, generator=g).bfloat16().to(DEV)
    res = torch.randn(2048, K, generator=g).bfloat16().to(DEV)
    full = ops.linear_swiglu(x, w)
    fn, fr = ops.rms_norm(x, nw, 1e-6, residual=res.clone())
    for m in (1, 8, 128, 256, 300, 768, 2048):
        assert torch.equal(ops.linear_swiglu(x[:m], w), full[:m]), m
        pn, pr = ops.rms_norm(x[:m], nw, 1e-6, residual=res[:m].clone())
        assert torch.equal(pn, fn[:m]) and torch.equal(pr, fr[:m]), m
    torch.cuda.synchronize()
    _native.check_status(torch.device(DEV))


def test_engine_in_batch_invariant_mode_gives_a_request_the_same_tokens_alone_and_in_a_batch(monkeypatch):
    from test_gpu_engine import _cfg
    from vllm_ascend_b200 import batch_invariant
    from vllm_ascend_b200.engine.llm import LLM
    from vllm_ascend_b200.engine.request import SamplingParams
    monkeypatch.setenv("VLLM_B200_BATCH_INVARIANT", "1")
    try:
        rng = np.random.default_rng(7)
        prompts = [rng.integers(0, 2048, size=n).tolist() for n in (150, 40, 333, 129, 64, 90)]
        sp = SamplingParams(temperature=0.0, max_tokens=12, ignore_eos=True, logprobs=3)
        llm = LLM(_cfg("bfloat16"), device="cuda", max_model_len=512, max_num_seqs=8, max_num_batched_tokens=1024,
                  num_gpu_blocks_override=64, enforce_eager=True, enable_prefix_caching=False)
        assert batch_invariant.is_batch_invariant()
        assert not getattr(llm.engine.runner.model, "norm_folded", False)
        together = llm.generate(prompts, sp)
        for i in (0, 2, 5):
            alone = llm.generate([prompts[i]], sp)[0]
            assert alone.outputs[0].token_ids == together[i].outputs[0].token_ids
            assert alone.outputs[0].logprobs == together[i].outputs[0].logprobs
    finally:
        batch_invariant.disable_batch_invariant_mode()


@pytest.mark.parametrize("Hkv,G,decodes", [(8, 4, 0), (8, 4, 3), (4, 8, 0)])
def test_prompt_attention_rows_do_not_depend_on_the_rows_beside_them(monkeypatch, Hkv, G, decodes):
    """A prompt alone, below the row count from which steps may take the kernel of two query tiles per block, and beside others far above it."""
    from vllm_ascend_b200.attention.metadata import metadata_from_tensors
    monkeypatch.setenv("VLLM_B200_BATCH_INVARIANT", "1")
    g = torch.Generator(device="cpu").manual_seed(3)
    D, page = 128, 128
    new, old = [1] * decodes + [300, 2600, 77], [50] * decodes + [40, 0, 513]
    pages = [-(-(n + o) // page) for n, o in zip(new, old)]
    k, v = (ops.alloc_kv_cache(sum(pages), page, Hkv, D, torch.bfloat16, DEV) for _ in range(2))
    for c in (k, v):
        c.copy_(torch.randn(c.shape, generator=g).to(DEV))
    q = torch.randn(sum(new), Hkv * G, D, generator=g).bfloat16().to(DEV)
    table = torch.zeros(len(new), max(pages), dtype=torch.int32)
    at = 0
    for b, n in enumerate(pages):
        table[b, :n] = torch.arange(at, at + n)
        at += n
    starts = np.cumsum([0] + new)

    def run(seqs):
        rows = torch.cat([torch.arange(starts[b], starts[b + 1]) for b in seqs]).to(DEV)
        cu = torch.tensor(np.cumsum([0] + [new[b] for b in seqs]), dtype=torch.int32, device=DEV)
        lens = torch.tensor([new[b] + old[b] for b in seqs], dtype=torch.int32, device=DEV)
        meta = metadata_from_tensors(cu, lens, table[seqs].to(DEV), max(new[b] for b in seqs), int(lens.max()), Hkv * G, Hkv, D)
        return rows, ops.paged_attention(q[rows], k, v, meta, D ** -0.5)
    _, together = run(list(range(len(new))))
    for b in range(len(new)):
        rows, alone = run([b])
        assert torch.equal(alone, together[rows]), b
    _native.check_status(torch.device(DEV))


def _logprobs_alone_and_together(cfg, **kw):
    """Greedy log-probabilities of requests whose steps hold 2048 rows together, and of each by itself."""
    from vllm_ascend_b200.engine.llm import LLM
    from vllm_ascend_b200.engine.request import SamplingParams
    rng = np.random.default_rng(8)
    prompts = [rng.integers(0, 2048, size=n).tolist() for n in (300, 900, 130, 700, 20)]
    sp = SamplingParams(temperature=0.0, max_tokens=4, ignore_eos=True, logprobs=3)
    llm = LLM(cfg, device="cuda", max_model_len=1024, max_num_seqs=8, max_num_batched_tokens=2048, num_gpu_blocks_override=64,
              enforce_eager=True, enable_prefix_caching=False, **kw)
    together = llm.generate(prompts, sp)
    return [(llm.generate([p], sp)[0].outputs[0].logprobs, t.outputs[0].logprobs) for p, t in zip(prompts, together)]


def _wide_cfg():
    """Heads that fill the GPU with prompt tiles, products with enough columns of K to be split."""
    from vllm_ascend_b200.config import ModelConfig
    return ModelConfig(name="t", architecture="Qwen3ForCausalLM", vocab_size=2048, hidden_size=2048, intermediate_size=4096,
                       num_hidden_layers=2, num_attention_heads=32, num_key_value_heads=8, head_dim=128, qk_norm=True,
                       rope_theta=1e6, dtype="bfloat16", init_std=0.05)


def test_engine_in_batch_invariant_mode_with_prompts_that_fill_the_gpu(monkeypatch):
    from vllm_ascend_b200 import batch_invariant
    monkeypatch.setenv("VLLM_B200_BATCH_INVARIANT", "1")
    try:
        for alone, together in _logprobs_alone_and_together(_wide_cfg()):
            assert alone == together
    finally:
        batch_invariant.disable_batch_invariant_mode()


def test_training_consistent_products_do_not_depend_on_the_row_count():
    """The switch by itself, without batch-invariant mode: products of a decode step and of the full sequence agree."""
    from vllm_ascend_b200.attention.backend import set_training_consistent_attention
    from vllm_ascend_b200.ops import linear_attn
    from vllm_ascend_b200.quantization import schemes
    g = torch.Generator(device="cpu").manual_seed(2)
    K, N = 4096, 2048
    x = (torch.randn(600, K, generator=g) * 0.5).bfloat16().to(DEV)
    w = (torch.randn(N, K, generator=g) * 0.05).bfloat16().to(DEV)
    w8 = torch.randn(N, K, generator=g).to(DEV).to(torch.float8_e4m3fn)
    ws = torch.rand(N // 128, K // 128, generator=g).to(DEV)
    cu, H = [0, 100, 140], 2
    rows = torch.randn(140, 3 * H * 128, generator=g).bfloat16().to(DEV)
    q, k, v = (r.view(140, H, 128) for r in rows.split(H * 128, 1))
    decay, beta = (torch.rand(140, H, generator=g).to(DEV) for _ in range(2))

    def delta(parts):
        out, state = [], torch.zeros(1, H, 128, 128, device=DEV)
        for i, (a, b) in enumerate(zip(parts, parts[1:])):
            t, has = torch.tensor([0, b - a], dtype=torch.int32, device=DEV), torch.tensor([i > 0], dtype=torch.int32, device=DEV)
            out.append(linear_attn.gated_delta_rule(q[a:b], k[a:b], v[a:b], -decay[a:b], beta[a:b], state, t, torch.zeros_like(has), has,
                                                    128 ** -0.5, True, cu_cpu=np.array([0, b - a])))
        return torch.cat(out), state
    set_training_consistent_attention(True)
    try:
        for step in (lambda x: ops.linear_step(x, w), lambda x: ops.linear_swiglu_step(x, w),
                     lambda x: schemes.fp8_block_linear(x, w8, ws)):
            full = step(x)
            for m in (1, 128, 256, 300):
                assert torch.equal(step(x[:m]), full[:m]), m
        whole, parts = delta([0, 140]), delta([0, 70, 71, 140])
        assert torch.equal(whole[0], parts[0]) and torch.equal(whole[1], parts[1])
    finally:
        set_training_consistent_attention(False)
    _native.check_status(torch.device(DEV))


def test_engine_with_training_consistency_alone():
    import os
    from vllm_ascend_b200.attention.backend import set_training_consistent_attention
    from vllm_ascend_b200.batch_invariant import is_batch_invariant
    from vllm_ascend_b200.platform_config import clear_b200_config
    saved = dict(os.environ)
    try:
        pairs = _logprobs_alone_and_together(_wide_cfg(), additional_config={"rl_config": {"enabled": True, "enable_training_consistency": True}})
        assert not is_batch_invariant()
        for alone, together in pairs:
            assert alone == together
    finally:
        set_training_consistent_attention(False)
        clear_b200_config()
        os.environ.clear()
        os.environ.update(saved)
