"""Batch-invariant (run-to-run and batch-size independent) execution mode.

What changes a result with the batch composition here is the reduction order.  The places that
choose it from the batch, and what the mode does there:

* the split-KV factor of decode attention (grouped, latent, variants): 1.  Where a context-parallel rank needs the log-sum-exp
  of latent attention, which two splits give, or a caller names a factor, the splits are even parts of each sequence by itself
  (latent attention cuts by the lengths of all sequences of the step in other modes);
* the collective algorithm: a fixed one;
* products of few rows, which split K over the blocks of a cluster (bf16 and block-scaled fp8): not
  taken.  The other GEMM kernels accumulate every output element over K in one fixed order whatever
  the tile shape;
* prompt attention with two query tiles per block, and latent prompts over up-projected keys and
  values: not taken;
* gated delta rule in chunks of 64 tokens: token by token;
* norms folded into the GEMMs around them: not folded.

The norm / activation / sampling kernels reduce per row.  The reference reaches the same goal by
swapping aten matmul/softmax/mean/rmsnorm for batch-invariant kernels and setting deterministic
collective variables (vllm_ascend/batch_invariant.py:76-162).
"""
from __future__ import annotations

import os

from . import envs

_flag = envs.raw("VLLM_B200_BATCH_INVARIANT")
_enabled = False
_training_consistent = False


def fixed_sums() -> bool:
    """Whether a row's sums have one order whatever shares its step: batch-invariant mode, or training-consistent attention
    (``attention.backend``), whose decode steps have to agree with the trainer's full-sequence pass in every kernel."""
    return _training_consistent or is_batch_invariant()


def set_training_consistent(on: bool) -> None:
    global _training_consistent
    _training_consistent = bool(on)


def is_training_consistent() -> bool:
    return _training_consistent


def is_batch_invariant() -> bool:
    return _enabled or _flag() == b"1"


def enable_batch_invariant_mode() -> None:
    global _enabled
    _enabled = True
    os.environ["VLLM_B200_BATCH_INVARIANT"] = "1"
    # fixed NCCL algorithm/protocol: reduction order no longer depends on message size heuristics
    os.environ.setdefault("NCCL_ALGO", "Ring")
    os.environ.setdefault("NCCL_PROTO", "Simple")
    os.environ.setdefault("NCCL_NVLS_ENABLE", "0")
    os.environ.setdefault("CUBLAS_WORKSPACE_CONFIG", ":4096:8")
    try:
        import torch
        torch.backends.cuda.matmul.allow_tf32 = False
        torch.backends.cudnn.deterministic = True
    except Exception:
        pass


def disable_batch_invariant_mode() -> None:
    global _enabled
    _enabled = False
    os.environ["VLLM_B200_BATCH_INVARIANT"] = "0"
