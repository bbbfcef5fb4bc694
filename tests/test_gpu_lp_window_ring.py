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


@pytest.mark.parametrize("compute,tol", [("float32", F32_TOL), ("bfloat16", 6e-2)])
@pytest.mark.parametrize("rows,start", [(1, 30), (40, 3), (9, 75)])
def test_steps_read_the_row_that_they_write(b200, rows, start, compute, tol):
    """Decoding norms and stores the position's key and value in the attention kernel itself; the ring must hold that row and not what the cache held before.  Slots are used twice,
    so that the row before is another sequence's; a step done again gives the same bits."""
    cfg = S.config([S.parallel_layer(heads=8, kv_heads=2, dim=128, vdim=128, window=64, keep_first=4), S.parallel_layer(heads=8, kv_heads=2, dim=64, vdim=128, window=64, keep_first=0)], width=256)
    w = S.random_weights(cfg, 3)
    rng = np.random.default_rng(rows)
    toks = rng.integers(0, cfg["vocab"], (2, rows, start + 6))
    gpu = S.gpu_model(cfg, w, compute, max_seq_len=start + 8, max_batch=rows)
    try:
        out = []
        for k in (1, 0, 1, 0):
            for r in range(rows):
                gpu.reset(r)
            gpu.step([(r, [int(t) for t in toks[k, r, :start]]) for r in range(rows)], [])
            out.append([np.array(gpu.step([(r, [int(t)]) for r, t in enumerate(col)], list(range(rows)))) for col in toks[k, :, start:].T])
    finally:
        gpu.close()
    for a, b in ((0, 2), (1, 3)):
        assert all(np.array_equal(x, y) for x, y in zip(out[a], out[b]))
    for r in (0, rows - 1):
        want = O.Model(cfg, w).forward([int(t) for t in toks[0, r]])[start:]
        assert max(S.rel_err(out[1][t][r], want[t]) for t in range(6)) < tol
