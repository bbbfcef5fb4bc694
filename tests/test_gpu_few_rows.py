"""Products of few token rows straight from the blocks (csrc/gemm_few.cuh, few_rows.cuh) against the token-by-token kernels, which keep f32 accuracy:
prompts and batched decode steps, every block type, row counts at the edges of the token tiles (16, 32, 64) and of the path (256), tiles cut between blocks.

Tolerance: activations are rounded to fp16 at four places per layer; with weights rounded to fp16 too such roundings measure 0.9e-4 .. 5.3e-4 of the largest
logit, within the bound of 1e-3 that every path of rows holds.  Here Q4_K and Q5_K weights are exact, Q6_K ones rounded where an integer is above 2048 (2^-12 of
itself), Q8_0 ones once, as before.  A wrong row, block or piece is off by the size of the logits."""
import numpy as np
import pytest
import torch

import synth
from synth import rel_err

pytestmark = pytest.mark.gpu
TOL = 1e-3
synth.TINY["few-128"] = dict(synth.TINY["llama-tiny"], hidden=2048, n_layers=2, n_heads=16, n_kv_heads=4, ffn=4096, vocab=700)
# heads of 64, NeoX rope, biases; in K-quants the heads' sums of 32 activations meet a minimum term
synth.TINY["few-64"] = dict(synth.TINY["qwen-tiny"], hidden=1024, n_layers=2, n_heads=16, n_kv_heads=2, ffn=2048, vocab=1000)
# hidden above ffn: the sums that the residual stream still lacks are wider than the gate rows in whose place they lie
synth.TINY["few-wide"] = dict(synth.TINY["llama-tiny"], hidden=2048, n_layers=2, n_heads=2, n_kv_heads=1, ffn=256, vocab=300)
MODELS = [("few-wide", "Q4_K"), ("few-128", "Q4_K_M"), ("few-128", "Q5_K_M"), ("few-128", "Q6_K"), ("few-64", "Q8_0"), ("few-64", "Q4_K"), ("few-64", "Q5_K")]


def launches(gpu, call):
    before = gpu.stats()["kernel_launches"]
    out = call()
    return out, gpu.stats()["kernel_launches"] - before


@pytest.mark.parametrize("preset,mix", MODELS)
@pytest.mark.parametrize("n", [32, 33, 64, 65, 150, 256])
def test_prompts(b200, monkeypatch, preset, mix, n):
    arch, desc, tensors = synth.synth_model(preset, mix, n + 8)
    prompt = synth.prompt_tokens(n, desc["vocab"])
    got, want = {}, {}
    for env, out in ((("B200_FEW_GEMM", "1"), got), (("B200_PREFILL_GEMM", "0"), want)):
        monkeypatch.setenv(*env)
        gpu = b200.GpuOnlyInference(desc, tensors)
        try:
            out["prompt"], out["n"] = launches(gpu, lambda: gpu.prefill(prompt))
            out["next"] = gpu.forward(3)      # reads the caches that the prompt has written
        finally:
            gpu.close()
    assert rel_err(got["prompt"], want["prompt"]) < TOL and rel_err(got["next"], want["next"]) < TOL
    assert got["n"] == 2 + 11 * desc["n_layers"] + 1, got["n"]      # the path that is meant: 11 kernels a layer


@pytest.mark.parametrize("preset,mix", MODELS)
@pytest.mark.parametrize("n", [8, 16, 17, 33, 64, 70])
def test_batched_decode(b200, monkeypatch, preset, mix, n):
    """Rows of slots at different positions; three steps (eager, captured, replayed)."""
    arch, desc, tensors = synth.synth_model(preset, mix, 96, max_batch=n)      # (a step has at most as many rows as the context has positions)
    rng = np.random.default_rng(n)
    steps = [rng.integers(0, desc["vocab"], n).astype(np.uint32) for _ in range(3)]
    out, count = {}, {}
    for way, least in (("rows", "8"), ("single", "1000")):
        monkeypatch.setenv("B200_BATCH_GEMM_MIN", least)
        gpu = b200.GpuOnlyInference(desc, tensors)
        try:
            for s in range(0, n, 3):
                gpu.forward(int(s % desc["vocab"]), seq=s) if s % 2 else [gpu.forward(int(t), seq=s) for t in range(40)]
            out[way], count[way] = zip(*[launches(gpu, lambda: gpu.decode_batch(list(range(n)), t)) for t in steps])
        finally:
            gpu.close()
    assert set(count["rows"]) == {8 * desc["n_layers"] + 6}, count      # the path that is meant: 8 kernels a layer, eager, captured and replayed
    for a, b in zip(out["rows"], out["single"]):
        assert max(rel_err(x, y) for x, y in zip(a, b)) < TOL


def test_switched_off(b200, monkeypatch):
    """Models the path does not take (and B200_FEW_GEMM=0) keep the products they had."""
    arch, desc, tensors = synth.synth_model("few-128", "Q4_K_M", 64)
    prompt = synth.prompt_tokens(40, desc["vocab"])
    n = []
    for on in ("1", "0"):
        monkeypatch.setenv("B200_FEW_GEMM", on)
        gpu = b200.GpuOnlyInference(desc, tensors)
        try:
            n.append(launches(gpu, lambda: gpu.prefill(prompt))[1])
        finally:
            gpu.close()
    assert n[0] != n[1]


def test_no_fp16_rows_for_prompts_that_need_none(b200):
    """The fp16 weight rows of the two-pass products are allocated by the first prompt that uses them, not by one of up to 256 tokens."""
    arch, desc, tensors = synth.synth_model("few-128", "Q4_K_M", 320)
    gpu = b200.GpuOnlyInference(desc, tensors)
    try:
        gpu.prefill(synth.prompt_tokens(256, desc["vocab"]))
        before = torch.cuda.mem_get_info()[0]
        gpu.reset()
        gpu.prefill(synth.prompt_tokens(300, desc["vocab"]))
        rows = 2 * 2 * desc["ffn"] * desc["hidden"]      # gate and up in fp16
        assert before - torch.cuda.mem_get_info()[0] >= rows
    finally:
        gpu.close()
