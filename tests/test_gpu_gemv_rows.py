"""Rows per warp of the CUDA-core dequant-GEMV (csrc/gemv.cuh: 4, 2 or 1 by the number of rows) and the line below which K-quant products take it: one token after
the other through small models whose products fall on either side, against the oracle.

Tolerance: the GEMV keeps f32 throughout, as the oracle does in another order; the bound is the one every per-token path holds (1e-3 of the largest logit)."""
import pytest

import synth
from synth import rel_err

pytestmark = pytest.mark.gpu
# rows of a product: 448 and 64 (one row per warp), 2368 x 2 of gate and up and 5001 of the head (two), 9600 (four); K-quants below the line (2 to 7 MB) and above it (9.4);
# ragged row counts
synth.TINY["rows-1"] = dict(synth.TINY["qwen-tiny"], n_layers=1, ffn=768)
synth.TINY["rows-2"] = dict(synth.TINY["qwen-tiny"], n_layers=1, ffn=2368, vocab=5001)
synth.TINY["rows-4"] = dict(synth.TINY["qwen-tiny"], n_layers=1, ffn=9600, vocab=9601)
synth.TINY["line"] = dict(synth.TINY["tinyllama-tiny"], n_layers=1, ffn=8192)
synth.TINY["line-above"] = dict(synth.TINY["tinyllama-tiny"], n_layers=1, ffn=16384)


@pytest.mark.parametrize("preset,mix", [("rows-1", "Q4_K_M"), ("rows-1", "Q8_0"), ("rows-2", "Q4_K_M"), ("rows-4", "Q8_0"), ("rows-4", "Q4_K_M"), ("line", "Q4_K_M"),
                                        ("line", "Q6_K"), ("line-above", "Q4_K_M")])
def test_tokens(b200, oracle, monkeypatch, preset, mix):
    monkeypatch.setenv("B200_MEGA", "0")
    arch, desc, tensors = synth.synth_model(preset, mix, 16)
    prompt = synth.prompt_tokens(5, desc["vocab"])
    gpu = b200.GpuOnlyInference(desc, tensors)
    ref = oracle.OracleModel(desc, tensors)
    try:
        for i, t in enumerate(prompt):
            got, want = gpu.forward(int(t)), ref.forward([int(t)])
            assert rel_err(got, want) < 1e-3, i
    finally:
        gpu.close()
