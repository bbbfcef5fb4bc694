"""The tensor-core products of the layer-program engine (csrc/gemm_tc.cuh) at the edges of their tiles: row counts around the token tiles
of 64, 128 and 256, widths that are no multiple of a slab of 64 or of a weight tile of 128, K steps cut over 1 to 8 CTAs, gated units, experts,
heads.  Same operands through the CUDA-core product (B200_LP_TC=0): f32 sums in another order, so a bf16 activation may round to its
neighbour (2^-8 of its value) and a close call of a router may turn; a wrong tile is off by the size of the result."""
import numpy as np
import pytest

import gefovik_synth as S

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("width,ff", [(72, 136), (200, 328), (1024, 2048)])
@pytest.mark.parametrize("rows", [17, 63, 64, 65, 128, 129, 257, 700])
def test_products_at_tile_edges(b200, monkeypatch, rows, width, ff):
    cfg = S.config([S.attn(heads=4, kv_heads=2, dim=16, mlp=S.dense(ff)), S.latent(heads=3, dim=16, vdim=24, kv_rank=32, mlp=S.moe(ff=width // 8 * 8))],
                   width=width, vocab=264)
    w = S.random_weights(cfg, 7)
    toks = [int(t) for t in np.random.default_rng(rows).integers(0, cfg["vocab"], rows)]
    out = {}
    for tc in ("1", "0"):
        monkeypatch.setenv("B200_LP_TC", tc)
        gpu = S.gpu_model(cfg, w, "bfloat16", max_seq_len=rows + 8)
        try:
            out[tc] = gpu.step([(0, toks)], list(range(rows)))
        finally:
            gpu.close()
    d = np.array([S.rel_err(a, b) for a, b in zip(out["1"], out["0"])])
    assert np.median(d) < 1e-2 and (d < 4e-2).mean() > 0.9, (np.median(d), d.max())
