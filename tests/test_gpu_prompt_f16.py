"""The two-pass products of prompts (csrc/prompt_f16.cuh: blocks -> fp16 rows, plain tcgen05 products) against the fused dequant-GEMM on the same
prompts: every block type, rows that are no multiple of a weight tile, biases, token counts around the token tiles of 64, 128 and 256, matrices
that need several portions of the scratch rows.

Tolerance: both round the same f32 block values to fp16 and add in f32, in another order; from there an activation near a tie rounds to the other
fp16 neighbour (2^-11), at three places per layer.  Against the oracle such roundings measure 0.9e-4 .. 5.3e-4 of the largest logit
(tests/test_gpu_prefill.py); two independent sets of them are at most sqrt(2) times as far apart, 7.5e-4, within the 1e-3 that either path
holds.  A wrong row, block or portion is off by the size of the logits."""
import pytest

import synth
from synth import rel_err

pytestmark = pytest.mark.gpu
TOL = 1e-3


def logits(b200, monkeypatch, desc, tensors, prompt, **env):
    for k, v in env.items():
        monkeypatch.setenv(k, v)
    gpu = b200.GpuOnlyInference(desc, tensors)
    try:
        return gpu.prefill(prompt)
    finally:
        gpu.close()


@pytest.mark.parametrize("preset,mix", [("llama-tiny", "Q4_K_M"), ("llama-tiny", "Q5_K_M"), ("llama-tiny", "Q6_K"), ("tinyllama-tiny", "Q8_0"), ("qwen-tiny", "Q8_0")])
@pytest.mark.parametrize("n", [32, 65, 129, 300])
def test_two_passes_against_the_fused_product(b200, monkeypatch, preset, mix, n):
    arch, desc, tensors = synth.synth_model(preset, mix, n + 8)
    prompt = synth.prompt_tokens(n, desc["vocab"])
    fused = logits(b200, monkeypatch, desc, tensors, prompt, B200_PROMPT_F16_MIN="100000")
    two = logits(b200, monkeypatch, desc, tensors, prompt, B200_PROMPT_F16_MIN="1")
    assert rel_err(two, fused) < TOL
    few = logits(b200, monkeypatch, desc, tensors, prompt, B200_PROMPT_F16_MIN="1", B200_PROMPT_F16_KROWS="1")     # portions of the least size
    assert rel_err(few, two) < TOL


@pytest.mark.parametrize("preset,mix", [("llama-tiny", "Q4_K_M"), ("qwen-tiny", "Q8_0")])
def test_a_refused_tensor_map_takes_the_fused_products(b200, monkeypatch, preset, mix):
    """Bit for bit what the fused kernels give; the refusal is the host's (B200_PROMPT_F16_MAPS=0)."""
    arch, desc, tensors = synth.synth_model(preset, mix, 160)
    prompt = synth.prompt_tokens(129, desc["vocab"])
    fused = logits(b200, monkeypatch, desc, tensors, prompt, B200_PROMPT_F16_MIN="100000")
    refused = logits(b200, monkeypatch, desc, tensors, prompt, B200_PROMPT_F16_MIN="1", B200_PROMPT_F16_MAPS="0")
    assert (refused == fused).all()


@pytest.mark.parametrize("first,second", [("Q4_K_M", "Q6_K"), ("Q6_K", "Q4_K_M")])
def test_each_layer_goes_by_its_own_types(b200, monkeypatch, first, second):
    """40 tokens through two layers, one of Q4_K (fused products up to 64 tokens) and one of Q6_K (two passes from 32 on), in either order: another number of
    kernels than with either way for both layers."""
    arch, desc, a = synth.synth_model("llama-tiny", first, 48, n_layers=2)
    _, _, b = synth.synth_model("llama-tiny", second, 48, n_layers=2)
    tensors = dict(a, **{k: v for k, v in b.items() if k.startswith("blk.1.")})
    prompt = synth.prompt_tokens(40, desc["vocab"])
    count = {}
    for rule in ("0", "1", "100000"):
        monkeypatch.setenv("B200_PROMPT_F16_MIN", rule)
        gpu = b200.GpuOnlyInference(desc, tensors)
        try:
            gpu.prefill(prompt)
            before = gpu.stats()["kernel_launches"]
            gpu.reset()
            gpu.prefill(prompt)
            count[rule] = gpu.stats()["kernel_launches"] - before
        finally:
            gpu.close()
    assert count["0"] not in (count["1"], count["100000"]), count


@pytest.mark.parametrize("mix,ffn,n,two_pass", [("Q8_0", 16384, 40, True), ("Q8_0", 49152, 40, False), ("Q8_0", 49152, 50, True), ("Q8_0", 73728, 50, False),
                                                ("Q8_0", 73728, 65, True), ("Q6_K", 73728, 40, True), ("Q4_K", 16384, 64, False)])
def test_short_prompts_go_by_the_size_of_the_layer(b200, monkeypatch, mix, ffn, n, two_pass):
    """Up to 64 tokens the two passes are taken while gate and up as fp16 rows fit in L2 (512 wide: 16384 units 34 MB, 49152 101 MB, 73728 151 MB); the number of
    kernels shows which way a prompt went."""
    monkeypatch.setitem(synth.TINY, "wide", dict(synth.TINY["tinyllama-tiny"], n_layers=1, ffn=ffn))
    arch, desc, tensors = synth.synth_model("wide", mix, 80)
    prompt = synth.prompt_tokens(n, desc["vocab"])
    count = {}
    for rule in ("0", "1", "100000"):
        monkeypatch.setenv("B200_PROMPT_F16_MIN", rule)
        gpu = b200.GpuOnlyInference(desc, tensors)
        try:
            gpu.prefill(prompt)
            before = gpu.stats()["kernel_launches"]
            gpu.reset()
            gpu.prefill(prompt)
            count[rule] = gpu.stats()["kernel_launches"] - before
        finally:
            gpu.close()
    assert count["1"] != count["100000"] and count["0"] == count["1" if two_pass else "100000"], count
