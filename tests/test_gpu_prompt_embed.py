"""Embedding rows of prompts (prefill_embed_kernel): eight elements per thread, up to 256 rows split between four blocks of 128 threads each, which rows wider
than 4096 go through twice; the last part of a row is cut.  Prompts of both launch shapes against the oracle, every kind of block.

Tolerance: that of test_gpu_prefill.py for these products, 1e-3 of the largest logit; a wrong element of a row is an error of the order of 1."""
import numpy as np
import pytest

import synth
from synth import rel_err

pytestmark = pytest.mark.gpu
synth.TINY["embed-wide"] = dict(synth.TINY["llama-tiny"], n_layers=1, hidden=4608, n_heads=36, n_kv_heads=9, ffn=512, vocab=300)
synth.TINY["embed-narrow"] = dict(synth.TINY["qwen-tiny"], n_layers=1)


@pytest.mark.parametrize("preset,mix,table,n", [("embed-wide", "Q4_K", "Q4_K", 34), ("embed-wide", "Q5_K", "Q5_K", 33), ("embed-wide", "Q6_K", "Q6_K", 33), ("embed-wide", "Q4_K", "Q4_K", 260),
                                                ("embed-narrow", "Q8_0", "Q8_0", 33), ("embed-narrow", "Q8_0", "Q5_0", 257), ("embed-narrow", "Q8_0", "Q4_0", 33)])
def test_rows_of_the_table(b200, oracle, preset, mix, table, n):
    arch, desc, tensors = synth.synth_model(preset, mix, 272)
    if table != mix:      # matrices of a type that a pass of rows takes, another for the table
        ne = tensors["token_embd.weight"][1]
        values = np.random.default_rng(5).standard_normal(int(np.prod(ne))).astype(np.float32) * 0.08
        tensors["token_embd.weight"] = (getattr(b200, table), ne, oracle.quantize(getattr(b200, table), values))
    prompt = synth.prompt_tokens(n, desc["vocab"])
    ref = oracle.OracleModel(desc, tensors)
    gpu = b200.GpuOnlyInference(desc, tensors)
    try:
        before = gpu.stats()["kernel_launches"]
        assert rel_err(gpu.prefill(prompt), ref.forward(prompt)) < 1e-3
        assert gpu.stats()["kernel_launches"] - before < n      # one pass, not token by token
    finally:
        gpu.close()
