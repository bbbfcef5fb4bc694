"""Products by pairs of CTAs (csrc/gemm_tc.cuh, PAIR) against single CTAs (B200_TC_PAIR=0): the same products of 16 added in the same order, so the same bits.  Token rows
around one and two tiles of 256 and their halves, an odd number of weight tiles (the second CTA of the last pair has none), weight rows and widths that are no multiple
of a tile or a slab, gated units, experts, heads."""
import numpy as np
import pytest

import gefovik_synth as S
import synth

pytestmark = pytest.mark.gpu
synth.TINY["pair-128"] = dict(synth.TINY["llama-tiny"], hidden=1152, n_layers=2, n_heads=9, n_kv_heads=3, ffn=1472, vocab=300)


@pytest.mark.parametrize("rows", [257, 300, 385, 512, 700])
def test_gguf_prompts(b200, monkeypatch, rows):
    monkeypatch.setenv("B200_FEW_GEMM", "0")
    arch, desc, tensors = synth.synth_model("pair-128", "Q8_0", rows + 4)
    out = {}
    for pair in ("2", "0"):
        monkeypatch.setenv("B200_TC_PAIR", pair)
        gpu = b200.GpuOnlyInference(desc, tensors)
        try:
            out[pair] = [gpu.prefill(synth.prompt_tokens(rows, desc["vocab"])), gpu.forward(3)]
            assert gpu.watchdog() == [0] * 8
        finally:
            gpu.close()
    # (single CTAs may cut K over clusters here: f32 sums in another order behind fp16 operands)
    assert max(synth.rel_err(a, b) for a, b in zip(out["2"], out["0"])) < 1e-3


@pytest.mark.parametrize("width,ff", [(200, 336), (1024, 2048)])
@pytest.mark.parametrize("rows", [129, 257, 300, 385, 512, 700])
def test_the_same_bits_in_programs_with_experts(b200, monkeypatch, rows, width, ff):
    cfg = S.config([S.attn(heads=4, kv_heads=2, dim=16, mlp=S.dense(ff)), S.latent(heads=3, dim=16, vdim=24, kv_rank=32, mlp=S.moe(experts=3, identity=1, ff=width // 8 * 8))],
                   width=width, vocab=264)
    w = S.random_weights(cfg, 7)
    toks = [int(t) for t in np.random.default_rng(rows).integers(0, cfg["vocab"], rows)]
    out = {}
    for pair in ("2", "0"):
        monkeypatch.setenv("B200_TC_PAIR", pair)
        gpu = S.gpu_model(cfg, w, "bfloat16", max_seq_len=rows + 8)
        try:
            out[pair] = gpu.step([(0, toks)], list(range(rows)))
        finally:
            gpu.close()
    assert (out["2"] == out["0"]).all()


def test_the_switch_is_read_when_the_context_is_made(b200, monkeypatch):
    """Products whose K is cut without pairs show by their bits which of the two ran."""
    monkeypatch.setenv("B200_FEW_GEMM", "0")
    arch, desc, tensors = synth.synth_model("pair-128", "Q8_0", 304)
    out = []
    for made, called in (("0", "0"), ("0", "2"), ("2", "2"), ("2", "0")):
        monkeypatch.setenv("B200_TC_PAIR", made)
        gpu = b200.GpuOnlyInference(desc, tensors)
        try:
            monkeypatch.setenv("B200_TC_PAIR", called)
            out.append(gpu.prefill(synth.prompt_tokens(300, desc["vocab"])))
        finally:
            gpu.close()
    assert (out[0] == out[1]).all() and (out[2] == out[3]).all() and (out[0] != out[2]).any()
