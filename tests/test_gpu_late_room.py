"""Batched decode steps of a context that finds no room on the device for what it has to allocate after loading.

Tolerance: that of test_gpu_few_rows.py for rows of fp16 activations, 1e-3 of the largest logit; rows in f32 (csrc/exact_rows.cuh) against token by token that of
test_gpu_exact_rows.py, 1e-5, and without room for their buffers the bits of token by token."""
import ctypes as C

import numpy as np
import pytest
import torch

import lazilorn_synth
import synth
from synth import rel_err

pytestmark = pytest.mark.gpu
TOL = 1e-3
synth.TINY["room"] = dict(synth.TINY["llama-tiny"], hidden=2048, n_layers=2, n_heads=16, n_kv_heads=4, ffn=4096, vocab=5000)
ROWS = 256       # their logits are 5.1 MB
# rows in f32 up to 32 sequences (no fp16 products of these blocks): the logits of 32 are 5.1 MB
synth.TINY["room-f32"] = dict(synth.TINY["llama-tiny"], hidden=256, n_layers=2, n_heads=4, n_kv_heads=2, head_dim=64, ffn=352, vocab=40000)
EXACT_TOL = 1e-5


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


def exact_calls(b200, monkeypatch, desc, tensors, calls, fill=None):
    """The calls with and without rows in f32; fill(k, blocks): before call k of the run with them."""
    out, launches = {}, {}
    for exact in ("0", "1"):
        monkeypatch.setenv("B200_EXACT_ROWS", exact)
        gpu = b200.GpuOnlyInference(desc, tensors)
        blocks = []
        try:
            out[exact], launches[exact] = [], []
            for k, call in enumerate(calls):
                if exact == "1" and fill:
                    fill(k, blocks)
                before = gpu.stats()["kernel_launches"]
                out[exact].append(call(gpu))
                launches[exact].append(gpu.stats()["kernel_launches"] - before)
        finally:
            while blocks:
                blocks.pop().free()
            gpu.close()
    return out, [a != b for a, b in zip(launches["1"], launches["0"])]      # (which calls took the rows)


def step(n, k, vocab=5000, greedy=False):
    t = np.random.default_rng([n, k]).integers(0, vocab, n).astype(np.uint32)
    return lambda gpu: (gpu.decode_batch_greedy if greedy else gpu.decode_batch)(list(range(n)), t)


def test_rows_in_f32_on_a_full_device(b200, monkeypatch):
    """The first steps and prompts of several rows find no room: none for their logits.  They go sequence by sequence and token by token, with those bits; the rows come
    when there is room."""
    arch, desc, tensors = synth.synth_model("room-f32", "Q4_0", 96, max_batch=32)
    prompt = lambda gpu: gpu.prefill(synth.prompt_tokens(9, desc["vocab"]), 31)  # noqa: E731

    def alone(gpu):      # (graphs of single tokens, one per slot and kind, are made while there is room)
        for s in range(32):
            gpu.prefill_token(1, s)
            gpu.decode_greedy(2, 1, s)
        return np.array([gpu.forward(3, s) for s in range(32)])
    calls = [alone, step(32, 0, 40000), step(32, 1, 40000, True), step(3, 2, 40000), prompt] + [step(32, 3 + k, 40000) for k in range(8)]

    def fill(k, blocks):
        if k == 1:
            blocks.append(Full())
        if k == 6:
            blocks.pop().free()
    out, rows = exact_calls(b200, monkeypatch, desc, tensors, calls, fill)
    assert not any(rows[:3]) and all(rows[-4:]), rows      # (three rows may fit what is left)
    for k, (a, b) in enumerate(zip(out["1"], out["0"])):
        if not any(rows[:k + 1]):
            assert np.array_equal(a, b)
        assert max(rel_err(x, y) for x, y in zip(np.atleast_2d(a), np.atleast_2d(b))) < EXACT_TOL


def test_rows_in_f32_beside_calls_that_need_all_room(b200, monkeypatch):
    """Captured steps of seven sequences and a long prompt in f32; then, on a full device, 256 rows whose logits fit only where the long prompt's buffers were.  The steps keep theirs and
    replay; the next long prompt goes token by token until there is room."""
    monkeypatch.setenv("B200_FEW_GEMM", "0")          # (nothing else to give back)
    monkeypatch.setenv("B200_PREFILL_GEMM_MIN", "1000")
    arch, desc, tensors = model()
    prompt = lambda n: lambda gpu: gpu.prefill(synth.prompt_tokens(n, desc["vocab"]), 250)  # noqa: E731
    alone = lambda gpu: (gpu.prefill_token(1, 250), gpu.forward(2, 250))[1]  # noqa: E731
    calls = [alone, step(8, 0)] + [step(7, k) for k in (1, 2, 3)] + [prompt(50), step(ROWS, 4), step(7, 5), prompt(40), step(7, 6), prompt(9), prompt(36), prompt(35), prompt(34)]

    def fill(k, blocks):
        if k in (6, 7):
            blocks.append(Full())
        if k == 10:
            while blocks:
                blocks.pop().free()
    out, rows = exact_calls(b200, monkeypatch, desc, tensors, calls, fill)
    assert rows[2:6] == [True] * 4 and rows[7:11] == [True, False, True, True] and rows[-1], rows
    for k, (a, b) in enumerate(zip(out["1"], out["0"])):
        assert max(rel_err(x, y) for x, y in zip(np.atleast_2d(a), np.atleast_2d(b))) < (EXACT_TOL if k < 6 and k != 1 else TOL)      # (from 6 on they read cache rows of fp16 activations)


def test_short_calls_keep_their_rows_when_a_long_prompt_finds_no_room(b200, monkeypatch):
    arch, desc, tensors = synth.synth_model("room-f32", "Q4_0", 160, max_batch=32)
    prompt = lambda n: lambda gpu: gpu.prefill(synth.prompt_tokens(n, desc["vocab"]), 30)  # noqa: E731
    alone = lambda gpu: (gpu.prefill_token(1, 30), gpu.forward(2, 30))[1]  # noqa: E731
    calls = [alone, step(3, 0, 40000), prompt(5), prompt(100), step(3, 1, 40000), prompt(7), step(3, 2, 40000), step(3, 3, 40000)]

    def fill(k, blocks):
        if k == 3:
            blocks.append(Full())
    out, rows = exact_calls(b200, monkeypatch, desc, tensors, calls, fill)
    assert rows == [False, True, True, False, True, True, True, True]
    for a, b in zip(out["1"], out["0"]):
        assert max(rel_err(x, y) for x, y in zip(np.atleast_2d(a), np.atleast_2d(b))) < EXACT_TOL


def test_a_layer_program_after_a_step_that_found_no_room(b200):
    """300 rows' logits (24 MB) find no room: the step fails, and smaller ones after it, on the full device and with room again, give what they give without it."""
    cfg = lazilorn_synth.config([lazilorn_synth.parallel_layer(), lazilorn_synth.delta_layer(ff=80)], vocab=20000)
    w = lazilorn_synth.random_weights(cfg, 1)
    toks = [int(t) for t in np.random.default_rng(1).integers(0, cfg["vocab"], 310)]
    out = []
    for full in (False, True):
        gpu = lazilorn_synth.gpu_model(cfg, w, "float32", max_seq_len=320)
        try:
            got = [gpu.step([(0, toks[:300])], [299]), gpu.step([(0, [toks[300]])], [0])]
            if full:
                gpu.step([(1, toks[:3])], [2])
                block = Full()
                try:
                    with pytest.raises(b200.AllocationFailed):
                        gpu.step([(1, toks[:300])], list(range(300)))
                    got.append(gpu.step([(0, [toks[301]])], [0]))
                finally:
                    block.free()
            else:
                got.append(gpu.step([(0, [toks[301]])], [0]))
            got += [gpu.step([(0, toks[302:306])], [0, 1, 2, 3]), gpu.step([(0, [toks[306]])], [0])]
            out.append(got)
        finally:
            gpu.close()
    for a, b in zip(*out):
        assert np.array_equal(a, b)
