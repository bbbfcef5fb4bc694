"""Batched decode steps of a context that finds no room on the device for what it has to allocate after loading.

Tolerance: that of test_gpu_few_rows.py for rows of fp16 activations, 1e-3 of the largest logit."""
import numpy as np
import pytest
import torch

import synth
from synth import rel_err

pytestmark = pytest.mark.gpu
TOL = 1e-3
synth.TINY["room"] = dict(synth.TINY["llama-tiny"], hidden=2048, n_layers=2, n_heads=16, n_kv_heads=4, ffn=4096, vocab=5000)
ROWS = 256       # their logits are 5.1 MB


def model():
    return synth.synth_model("room", "Q4_K_M", 272, max_batch=ROWS)


def tokens(n, k):
    return np.random.default_rng([n, k]).integers(0, 5000, n).astype(np.uint32)


def fill(leave):
    torch.cuda.empty_cache()
    return torch.empty(torch.cuda.mem_get_info()[0] - leave, dtype=torch.uint8, device="cuda")


def test_a_step_that_failed_leaves_a_context_that_works(b200, monkeypatch):
    """256 rows find no room for their logits: the call fails, and the steps after it give what they give without it."""
    monkeypatch.setenv("B200_FEW_GEMM", "0")          # (no buffers to give back)
    arch, desc, tensors = model()
    out = []
    for full in (False, True):
        gpu = b200.GpuOnlyInference(desc, tensors)
        try:
            got = [gpu.decode_batch(list(range(8)), tokens(8, 0))]
            if full:
                block = fill(3 << 20)
                with pytest.raises(b200.AllocationFailed):
                    gpu.decode_batch(list(range(ROWS)), tokens(ROWS, 1))
                del block
                torch.cuda.empty_cache()
            got += [gpu.decode_batch(list(range(8)), tokens(8, k)) for k in (2, 3, 4)]
            out.append(got)
        finally:
            gpu.close()
    for a, b in zip(*out):
        assert np.array_equal(a, b)
