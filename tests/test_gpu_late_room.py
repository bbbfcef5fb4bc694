"""Batched decode steps of a context that finds no room on the device for what it has to allocate after loading.

Tolerance: that of test_gpu_few_rows.py for rows of fp16 activations, 1e-3 of the largest logit."""
import ctypes as C

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


class Full:
    """All device memory but less than 4 MB in one piece, taken straight from the driver (the caching allocator rounds, and what free memory there is may be in pieces)."""

    def __init__(self):
        torch.cuda.empty_cache()
        self.rt, self.at = C.CDLL("libcudart.so.12"), []
        for size in [(1 << 30) * 16, 1 << 30, 1 << 26, 1 << 24, 1 << 22]:
            p = C.c_void_p()
            while self.rt.cudaMalloc(C.byref(p), C.c_size_t(size)) == 0:
                self.at.append(p)
                p = C.c_void_p()
            self.rt.cudaGetLastError()

    def free(self):
        for p in self.at:
            assert self.rt.cudaFree(p) == 0


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
                block = Full()
                try:
                    with pytest.raises(b200.AllocationFailed):
                        gpu.decode_batch(list(range(ROWS)), tokens(ROWS, 1))
                finally:
                    block.free()
            got += [gpu.decode_batch(list(range(8)), tokens(8, k)) for k in (2, 3, 4)]
            out.append(got)
        finally:
            gpu.close()
    for a, b in zip(*out):
        assert np.array_equal(a, b)


def test_buffers_of_few_rows_are_given_back(b200, monkeypatch):
    """Captured steps of eight rows; then 256 rows whose logits fit only where the images and pieces of the products of few rows were, eight rows on the full device, and
    eight with room again.  The steps captured before name buffers that are gone, and the one captured meanwhile does without them: none of them may be replayed.  The buffers
    are not asked for at every step: after the one that finds no room, the next does not ask."""
    arch, desc, tensors = model()
    calls = [(8, 0), (8, 1), (8, 2), (ROWS, 3), (8, 4), (8, 5), (8, 6), (8, 7)]
    out, launches = {}, {}
    for few in ("0", "1"):      # (the first also loads the kernels that the full device needs)
        monkeypatch.setenv("B200_FEW_GEMM", few)
        gpu = b200.GpuOnlyInference(desc, tensors)
        blocks = []
        try:
            out[few], launches[few] = [], []
            for k, (n, seed) in enumerate(calls):
                if few == "1" and k in (3, 4):        # (at 4: what was given back is taken as well)
                    blocks.append(Full())
                if few == "1" and k == 5:
                    while blocks:
                        blocks.pop().free()
                before = gpu.stats()["kernel_launches"]
                out[few].append(gpu.decode_batch(list(range(n)), tokens(n, seed)))
                launches[few].append(gpu.stats()["kernel_launches"] - before)
        finally:
            for b in blocks:
                b.free()
            gpu.close()
    few_path = 8 * desc["n_layers"] + 6
    assert [x == few_path for x in launches["1"]] == [True] * 3 + [False] * 3 + [True] * 2, launches
    assert few_path not in launches["0"]
    for a, b in zip(out["1"], out["0"]):
        assert max(rel_err(x, y) for x, y in zip(a, b)) < TOL
