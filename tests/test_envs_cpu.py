"""Variables as the readers of envs and batch_invariant see them, whatever mapping is in the place of os.environ."""
import os

import pytest

from vllm_ascend_b200 import batch_invariant, envs


class _Other(dict):
    """A mapping of its own with a private dictionary of the name that the standard one uses."""
    def __init__(self, *a):
        super().__init__(*a)
        self._data = {k: "other" for k in self}


@pytest.mark.parametrize("kind", [dict, _Other])
def test_a_mapping_in_place_of_environ(monkeypatch, kind):
    monkeypatch.setattr(os, "environ", kind({"VLLM_B200_GEMM": "cublas", "VLLM_B200_GEMM_2CTA_MIN_M": "77", "VLLM_B200_CUDA_GRAPH": "0",
                                             "VLLM_B200_BATCH_INVARIANT": "1"}))
    assert envs.VLLM_B200_GEMM == "cublas" and envs.VLLM_B200_GEMM_2CTA_MIN_M == 77 and not envs.VLLM_B200_CUDA_GRAPH
    assert batch_invariant.is_batch_invariant()
    monkeypatch.setattr(os, "environ", kind())
    assert envs.VLLM_B200_GEMM != "cublas" and not batch_invariant.is_batch_invariant()


def test_numbers_and_switches_as_text(monkeypatch):
    """What int and str.strip take of text."""
    monkeypatch.setenv("VLLM_B200_GEMM_2CTA_MIN_M", " 7_0 ")
    assert envs.VLLM_B200_GEMM_2CTA_MIN_M == 70
    monkeypatch.setenv("VLLM_B200_GEMM_2CTA_MIN_M", "٣٢")
    assert envs.VLLM_B200_GEMM_2CTA_MIN_M == 32
    monkeypatch.setenv("VLLM_B200_CUDA_GRAPH", " ON ")
    assert envs.VLLM_B200_CUDA_GRAPH
    monkeypatch.setenv("VLLM_B200_GEMM_2CTA_MIN_M", "x")
    with pytest.raises(ValueError):
        envs.VLLM_B200_GEMM_2CTA_MIN_M
