"""Products of a step's 17 to 128 rows with the rows as M (csrc/gemm_tc.cuh, lp_gemm_tc_rows_kernel) against the tiles of 128 weight rows (B200_LP_TC_ROWS=0): the same
products of 16 added in the same order, so the same bits.  Row counts at the edges of M = 64 and 128 and of a row group of 8, widths that are no multiple of a slab of 64,
of four slabs or of a weight tile, more slabs than the ring holds."""
import numpy as np
import pytest

import gefovik_synth as S

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("width,ff", [(72, 144), (200, 336), (1024, 4096)])
@pytest.mark.parametrize("rows", [17, 24, 33, 63, 64, 65, 127, 128])
def test_the_same_bits(b200, monkeypatch, rows, width, ff):
    cfg = S.config([S.attn(heads=4, kv_heads=2, dim=16, mlp=S.dense(ff)), S.latent(heads=3, dim=16, vdim=24, kv_rank=32, mlp=S.moe(experts=5, identity=1, ff=width // 8 * 8))],
                   width=width, vocab=264)
    w = S.random_weights(cfg, 7)
    toks = [int(t) for t in np.random.default_rng(rows).integers(0, cfg["vocab"], rows)]
    out = {}
    for on in ("1", "0"):
        monkeypatch.setenv("B200_LP_TC_ROWS", on)
        gpu = S.gpu_model(cfg, w, "bfloat16", max_seq_len=rows + 8)
        try:
            out[on] = gpu.step([(0, toks)], list(range(rows)))
        finally:
            gpu.close()
    assert (out["1"] == out["0"]).all()
