"""The tensor-core products of the layer-program engine (csrc/gemm_tc.cuh) at the edges of their tiles: row counts around the token tiles
of 64, 128 and 256, widths that are no multiple of a slab of 64 or of a weight tile of 128, K steps cut over 1 to 8 CTAs, gated units, experts,
heads.  Same operands through the CUDA-core product (B200_LP_TC=0): f32 sums in another order, so a bf16 activation may round to its
neighbour, 2^-8 of its value; a few in a hundred do, so a row differs by less than 2^-8 per rounding it passes through (under 10 of them: 4e-2 at the very
most, measured 5e-3).  The bound is on the LARGEST row: the last token tile of 65, 129 or 257 rows is one row, and a wrong row is off by its size.
The mixtures' choices are decided (gefovik_synth.decided_weights), so that no row may turn."""
import numpy as np
import pytest

import gefovik_synth as S

pytestmark = pytest.mark.gpu

LAYERS = {
    "dense_and_heads": lambda width, ff: [S.attn(heads=4, kv_heads=2, dim=16, mlp=S.dense(ff)), S.latent(heads=3, dim=16, vdim=24, kv_rank=32, mlp=S.dense(ff // 2))],
    "experts": lambda width, ff: [S.attn(heads=4, kv_heads=2, dim=16, mlp=S.moe(experts=5, identity=1, ff=width // 8 * 8))],
}


@pytest.mark.parametrize("width,ff", [(72, 144), (200, 336), (1024, 2048)])
@pytest.mark.parametrize("rows", [17, 63, 64, 65, 128, 129, 257, 700])
@pytest.mark.parametrize("kind", list(LAYERS))
def test_products_at_tile_edges(b200, monkeypatch, kind, rows, width, ff):
    cfg = S.config(LAYERS[kind](width, ff), width=width, vocab=264)
    w = S.decided_weights(cfg, 7)
    toks = [int(t) for t in np.random.default_rng(rows).integers(0, cfg["vocab"], rows)]
    out = {}
    for tc in ("1", "0"):
        monkeypatch.setenv("B200_LP_TC", tc)
        gpu = S.gpu_model(cfg, w, "bfloat16", max_seq_len=rows + 8)
        try:
            out[tc] = gpu.step([(0, toks)], list(range(rows)))
        finally:
            gpu.close()
    assert S.rel_err(out["1"], out["0"]) < 4e-2


def test_refused_tensor_maps_take_the_cuda_core_products(b200, monkeypatch):
    """Gated layers and experts included, whose units the tensor-core products make in their epilogues.  The refusal is the host's (B200_LP_TC_MAPS=0)."""
    cfg = S.config([S.attn(heads=4, kv_heads=2, dim=16, mlp=S.dense(136)), S.latent(heads=3, dim=16, vdim=24, kv_rank=32, mlp=S.moe(ff=72))], width=72, vocab=264)
    w = S.random_weights(cfg, 7)
    toks = [int(t) for t in np.random.default_rng(1).integers(0, cfg["vocab"], 90)]
    out = {}
    for env in ("B200_LP_TC", "B200_LP_TC_MAPS"):
        monkeypatch.setenv(env, "0")
        gpu = S.gpu_model(cfg, w, "bfloat16", max_seq_len=96)
        try:
            out[env] = gpu.step([(0, toks)], list(range(90)))
        finally:
            gpu.close()
            monkeypatch.delenv(env)
    assert (out["B200_LP_TC"] == out["B200_LP_TC_MAPS"]).all()


@pytest.mark.parametrize("kind", list(LAYERS))
def test_programs_with_experts_add_in_the_order_of_k(b200, monkeypatch, kind):
    """32 rows at a width where K would be cut over clusters (B200_LP_ANY_ORDER=1): not in a program with experts, whose choices another order of the sums would turn in
    close calls."""
    cfg = S.config(LAYERS[kind](1024, 2048), width=1024, vocab=264)
    w = S.random_weights(cfg, 7)
    toks = [int(t) for t in np.random.default_rng(1).integers(0, cfg["vocab"], 32)]
    out = {}
    for split in ("", "0", "1"):
        monkeypatch.setenv("B200_LP_ANY_ORDER", split)
        gpu = S.gpu_model(cfg, w, "bfloat16", max_seq_len=40)
        try:
            out[split] = gpu.step([(0, toks)], list(range(32)))
        finally:
            gpu.close()
    as_told = "0" if kind == "experts" else "1"
    assert (out[""] == out[as_told]).all() and (out["0"] != out["1"]).any()


def test_a_batch_of_sequences_row_by_row(b200):
    """32 prompts in one step, then steps of all 32, at the width where K is cut over clusters: every row of logits against the library's own f32 mode, which shares no
    product or prompt-attention kernel with it and is held to the float64 oracle in the models' tests.  bf16 through two layers: 4e-3 of a row."""
    cfg = S.config([S.attn(heads=16, kv_heads=4, dim=128, scale=128 ** -0.5, softcap=50.0, mlp=S.dense(8192)),
                    S.latent(heads=16, dim=96, vdim=128, kv_rank=128, mlp=S.moe(experts=8, identity=2, ff=2048))], width=2048, vocab=512, scale=1.0)
    w = S.decided_weights(cfg, 11)
    rng = np.random.default_rng(2)
    runs = [(i, [int(t) for t in rng.integers(0, cfg["vocab"], 48)]) for i in range(32)]
    steps = [[(i, [int(rng.integers(0, cfg["vocab"]))]) for i in range(32)] for _ in range(3)]
    out = {}
    for compute in ("bfloat16", "float32"):
        gpu = S.gpu_model(cfg, w, compute, max_seq_len=64, max_batch=32)
        try:
            out[compute] = np.concatenate([gpu.step(runs, [48 * i + 47 for i in range(32)])] + [gpu.step(s, list(range(32))) for s in steps])
        finally:
            gpu.close()
    assert S.rel_err(out["bfloat16"], out["float32"]) < 1.6e-2
