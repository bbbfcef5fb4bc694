"""Unpacking of prompts' weights (csrc/prompt_f16.cuh) in runs of eight units per warp, which matrices of 4.9 M elements and more take (the smaller ones of
test_gpu_prompt_f16.py go in runs of two): the two-pass products against the fused ones, every block type, a last run that is cut.

Tolerance: as test_gpu_prompt_f16.py, two sets of fp16 roundings of the same operands: 7.5e-4 of the largest logit, within 1e-3."""
import pytest

import synth
from synth import rel_err

pytestmark = pytest.mark.gpu
synth.TINY["unpack"] = dict(synth.TINY["tinyllama-tiny"], n_layers=1, ffn=9728)          # 512 x 9728 = 19456 units: 2432 runs of eight, 304 blocks
synth.TINY["unpack-cut"] = dict(synth.TINY["qwen-tiny"], n_layers=1, ffn=11008)          # 448 x 11008 = 19264 units of 256, rows of 1.75 units


@pytest.mark.parametrize("preset,mix", [("unpack", "Q4_K_M"), ("unpack", "Q5_K_M"), ("unpack", "Q6_K"), ("unpack", "Q8_0"), ("unpack-cut", "Q8_0")])
def test_runs_of_eight(b200, monkeypatch, preset, mix):
    arch, desc, tensors = synth.synth_model(preset, mix, 96)
    prompt = synth.prompt_tokens(80, desc["vocab"])
    out = {}
    for rule in ("1", "100000"):
        monkeypatch.setenv("B200_PROMPT_F16_MIN", rule)
        gpu = b200.GpuOnlyInference(desc, tensors)
        try:
            out[rule] = gpu.prefill(prompt)
        finally:
            gpu.close()
    assert rel_err(out["1"], out["100000"]) < 1e-3
