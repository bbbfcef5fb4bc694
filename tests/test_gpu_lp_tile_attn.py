"""The tcgen05 attention of prompt rows (csrc/lp_tile_attn.cuh), and the mma.sync kernels that stand in for it where the bf16 copies find no room
(B200_LP_KEYS16_MB=0), against the warp kernel (B200_LP_ATTN_TILE=0), which scores in f32: kept first
tokens that fill, end inside and pass their tiles of 64, windows that leave tiles out between them and the first visible key, blocks of 128
(token, head) pairs that end inside a token, portions that continue a cache, scores large enough that the running maximum jumps and
the sums are rescaled.  Tolerance: bf16 queries, keys and probabilities (2^-8 each) against f32, as in the models' own tests; a wrong key or factor
is off by the size of the result."""
import numpy as np
import pytest

import gefovik_synth as GS
import lazilorn_synth as S
import marosun_synth as MA
import mefurax_synth as ME

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("heads,kv_heads,dim,vdim", [(4, 2, 128, 128), (3, 1, 64, 64), (5, 1, 48, 72), (2, 2, 80, 8)])
@pytest.mark.parametrize("window,keep,scale", [(200, 130, 1.0), (40, 64, 1.0), (100, 3, 12.0), (1000, 0, 4.0), (1, 5, 1.0)])
def test_against_the_warp_kernel(b200, monkeypatch, heads, kv_heads, dim, vdim, window, keep, scale):
    cfg = S.config([S.parallel_layer(heads=heads, kv_heads=kv_heads, dim=dim, vdim=vdim, window=window, keep_first=keep, scale=scale * dim ** -0.5, left_scale=1.0,
                                     right_scale=0.0, ff=0)], width=64, vocab=80)
    w = S.random_weights(cfg, 5)
    rng = np.random.default_rng(window + keep)
    a, b, more = ([int(t) for t in rng.integers(0, cfg["vocab"], n)] for n in (450, 131, 97))
    outs = {}
    for tile, mb in (("1", "1024"), ("0", "1024"), ("mma", "0")):
        monkeypatch.setenv("B200_LP_ATTN_TILE", "0" if tile == "0" else "1")
        monkeypatch.setenv("B200_LP_KEYS16_MB", mb)
        gpu = S.gpu_model(cfg, w, "bfloat16", max_seq_len=640)
        try:
            first = gpu.step([(0, a), (1, b)], list(range(len(a) + len(b))))
            second = gpu.step([(1, more[:1]), (0, more)], list(range(1 + len(more))))
            outs[tile] = np.concatenate([first, second])
        finally:
            gpu.close()
    tol = 2e-2 if scale < 8 else 6e-2      # (scores of tens: a bf16 score error is 2^-8 of them)
    assert S.rel_err(outs["1"], outs["0"]) < tol and S.rel_err(outs["mma"], outs["0"]) < tol


@pytest.mark.parametrize("layer", [GS.attn(heads=4, kv_heads=2, dim=128, scale=1.0, softcap=50.0), GS.attn(heads=3, kv_heads=1, dim=64, scale=1.0, softcap=1000.0),
                                   GS.latent(heads=3, dim=16, vdim=24, kv_rank=128, scale=1.0), GS.latent(heads=4, dim=48, vdim=64, kv_rank=64, scale=1.0)])
@pytest.mark.parametrize("n", [65, 130, 300])
def test_rounds_what_the_mma_kernels_round(b200, monkeypatch, layer, n):
    """Queries, keys as they are stored and probabilities are rounded to bf16, and nothing else: a key row's factor meets the f32 score.  The mma.sync kernels
    (B200_LP_KEYS16_MB=0) round the same numbers, probabilities against another maximum: each is 2^-8 of itself apart at most, a row 4e-3 where one of them is nearly
    all of it (measured 2.3e-3).  A product of key and factor that is rounded moves scores of some tens (scale 1) by 2^-9 of themselves, the row by 7e-3 to 1.4e-2."""
    cfg = GS.config([layer], width=256, vocab=80)
    w = GS.random_weights(cfg, 5)
    toks = [int(t) for t in np.random.default_rng(n).integers(0, cfg["vocab"], n)]
    outs = {}
    for mb in ("1024", "0"):
        monkeypatch.setenv("B200_LP_KEYS16_MB", mb)
        gpu = GS.gpu_model(cfg, w, "bfloat16", max_seq_len=320)
        try:
            outs[mb] = gpu.step([(0, toks), (1, toks[: n // 2 + 8])], list(range(n + n // 2 + 8)))
        finally:
            gpu.close()
    assert GS.rel_err(outs["1024"], outs["0"]) < 4e-3


@pytest.mark.parametrize("lens,mlp,same", [((48, 64, 17), "moe", True), ((48, 64, 17), "dense", False), ((48, 65, 17), "moe", False)])
def test_one_tile_of_keys_per_run_in_programs_with_experts(b200, monkeypatch, lens, mlp, same):
    """Steps of programs with experts whose runs see one tile of keys each: bit for bit the mma.sync kernels (B200_LP_KEYS16_MB=0).  Without experts, or with one run of
    65 keys, the other kernel takes the step."""
    cfg = GS.config([GS.attn(heads=4, kv_heads=2, dim=128, softcap=50.0), GS.latent(heads=3, dim=16, vdim=24, kv_rank=128, mlp=GS.moe() if mlp == "moe" else GS.dense())],
                    width=256, vocab=80)
    w = GS.random_weights(cfg, 5)
    rng = np.random.default_rng(1)
    runs = [(i, [int(t) for t in rng.integers(0, cfg["vocab"], n)]) for i, n in enumerate(lens)]
    outs = {}
    for mb in ("1024", "0"):
        monkeypatch.setenv("B200_LP_KEYS16_MB", mb)
        gpu = GS.gpu_model(cfg, w, "bfloat16", max_seq_len=128)
        try:
            outs[mb] = gpu.step(runs, list(range(sum(lens))))
        finally:
            gpu.close()
    assert (outs["1024"] == outs["0"]).all() == same


FORMS = {   # (synth module, layer, added to the learned extra terms of the denominator)
    "slope_window": (ME, ME.layer_a(heads=4, kv_heads=2, dim=64, vdim=72, window=200, scale=0.125), 0.0),
    "softcap_chunks_head_gate": (ME, ME.layer_b(heads=4, kv_heads=2, dim=64, vdim=64, chunk=100, softcap=5.0, scale=0.125), 0.0),
    "softcap_bites": (ME, ME.layer_b(heads=4, kv_heads=1, dim=128, vdim=128, chunk=300, softcap=1.5, scale=0.2), 0.0),
    "turned_values_sink": (MA, MA.layer_a(heads=4, kv_heads=2, dim=64, vdim=64), 0.0),
    "sink_above_all": (MA, MA.layer_a(heads=4, kv_heads=2, dim=64, vdim=64), 25.0),
    "sink_below_all": (MA, MA.layer_a(heads=3, kv_heads=1, dim=48, vdim=80), -60.0),
    "channel_gate_chunks_sink": (MA, MA.layer_p(heads=4, kv_heads=2, dim=64, vdim=40, chunk=100, right_scale=0.0), 0.0),
    "one_in_the_denominator": (MA, MA.layer_q(heads=4, kv_heads=2, dim=32, vdim=64), 0.0),
    "values_from_unit_keys": (GS, GS.attn(heads=6, kv_heads=2, dim=128, scale=0.25, softcap=50.0), 0.0),
    "values_from_unit_keys_capped": (GS, GS.attn(heads=4, kv_heads=4, dim=64, scale=0.25, softcap=2.0), 0.0),
    "latent_sink_above": (GS, GS.latent(heads=3, dim=16, vdim=24, kv_rank=128), 20.0),
    "latent_sink_below": (GS, GS.latent(heads=5, dim=48, vdim=64, kv_rank=64), -60.0),
}


@pytest.mark.parametrize("form", list(FORMS))
def test_every_form_against_the_warp_kernel(b200, monkeypatch, form):
    """What a score goes through besides the products, over several tiles of keys and a portion that continues them: row by row, the bound of bf16 queries, keys and
    probabilities (scores of a few units: 2^-8 of them in a probability, halved by the average over the keys; four times that)."""
    M, layer, shift = FORMS[form]
    cfg = M.config([layer], width=64, vocab=80)
    w = M.random_weights(cfg, 5)
    for k in w:
        if k.endswith("sink"):
            w[k] = (w[k] + shift).astype(np.float32)
    rng = np.random.default_rng(3)
    a, b, more = ([int(t) for t in rng.integers(0, cfg["vocab"], n)] for n in (300, 131, 97))
    outs = {}
    for tile in ("1", "0"):
        monkeypatch.setenv("B200_LP_ATTN_TILE", tile)
        gpu = M.gpu_model(cfg, w, "bfloat16", max_seq_len=512)
        try:
            outs[tile] = np.concatenate([gpu.step([(0, a), (1, b)], list(range(len(a) + len(b)))), gpu.step([(1, more[:1]), (0, more)], list(range(1 + len(more))))])
        finally:
            gpu.close()
    assert GS.rel_err(outs["1"], outs["0"]) < 2e-2
