"""Single rows of windowed attention whose keys and values come through a ring in shared memory (layerprog.cu, lp_window_attn_kernel): row after row of a prompt in f32,
which runs every position through it, against the float64 oracle.  Fewer than one block of 32 keys, more blocks than warps (the ring has room for three chunks of
each then), kept first tokens, ragged last blocks, sizes up to 128 that are no multiple of 32.  The bound is the models' (f32 sums in another order)."""
import numpy as np
import pytest

import lazilorn_oracle as O
import lazilorn_synth as S

pytestmark = pytest.mark.gpu
F32_TOL = 2e-5


@pytest.mark.parametrize("dim,vdim,window,keep_first,n", [(128, 128, 1024, 0, 650), (128, 64, 300, 5, 380), (64, 128, 40, 3, 100), (36, 20, 70, 33, 130)])
def test_rows_against_the_oracle(b200, dim, vdim, window, keep_first, n):
    cfg = S.config([S.parallel_layer(heads=4, kv_heads=2, dim=dim, vdim=vdim, window=window, keep_first=keep_first)])
    w = S.random_weights(cfg, 3)
    toks = [int(t) for t in np.random.default_rng(n).integers(0, cfg["vocab"], n)]
    want = O.Model(cfg, w).forward(toks)
    gpu = S.gpu_model(cfg, w, max_seq_len=n + 4)
    try:
        got = gpu.step([(0, toks)], list(range(n)))
    finally:
        gpu.close()
    assert S.rel_err(got, want) < F32_TOL
