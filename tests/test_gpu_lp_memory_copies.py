"""Steps of many sequences through the matrix memory (layerprog.cu, lp_matrix_memory_kernel): the column blocks of a head share n and m, and a block that is placed after another has
finished must read them as they were before the step.  The same steps again and again give the same bits; prompts (tokens one after the other and in chunks), steps
and prompts behind steps against the float64 oracle."""
import numpy as np
import pytest

import lazilorn_oracle as O
import lazilorn_synth as S

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("compute,rows,times", [("bfloat16", 27, 12), ("bfloat16", 33, 8), ("float32", 200, 4)])
def test_a_step_done_again(b200, compute, rows, times):
    cfg = S.config([S.parallel_layer(heads=8, kv_heads=2, dim=128, vdim=128, window=1024, keep_first=4, mheads=4, mdim=64, mvdim=128, ff=4096)], width=1024)
    w = S.random_weights(cfg, 2)
    toks = np.random.default_rng(rows).integers(0, cfg["vocab"], (rows, 36))
    gpu = S.gpu_model(cfg, w, compute, max_seq_len=40, max_batch=rows)
    try:
        first = None
        for _ in range(times):
            for r in range(rows):
                gpu.reset(r)
            gpu.step([(r, [int(t) for t in toks[r, :32]]) for r in range(rows)], [])
            got = [np.array(gpu.step([(r, [int(t)]) for r, t in enumerate(col)], list(range(rows)))) for col in toks[:, 32:].T]
            first = first or got
            assert all(np.array_equal(a, b) for a, b in zip(first, got))
    finally:
        gpu.close()


@pytest.mark.parametrize("chunks", ["1", "0"])
def test_prompts_and_steps_in_turn(b200, monkeypatch, chunks):
    """Two slots take steps of unequal numbers: each reads the copy that its own last step wrote.  A slot used again starts from zeros."""
    monkeypatch.setenv("B200_LP_CHUNK_SCAN", chunks)
    cfg = S.config([S.parallel_layer(mheads=3, mdim=20, mvdim=36), S.parallel_layer(mheads=2, mdim=64, mvdim=24)])
    w = S.random_weights(cfg, 5)
    toks = np.random.default_rng(1).integers(0, cfg["vocab"], (3, 140))
    gpu = S.gpu_model(cfg, w, "float32", max_seq_len=140)
    at, want = [0, 0], [O.Model(cfg, w).forward([int(t) for t in row]) for row in toks]

    def go(runs):      # runs: (slot, sequence, tokens)
        got = gpu.step([(s, [int(t) for t in toks[q, at[s]:at[s] + n]]) for s, q, n in runs], list(range(sum(n for *_, n in runs))))
        row = 0
        for s, q, n in runs:
            assert S.rel_err(got[row:row + n], want[q][at[s]:at[s] + n]) < 2e-5
            at[s] += n
            row += n
    try:
        for runs in ([(0, 0, 50)], [(0, 0, 1)], [(0, 0, 1), (1, 1, 60)], [(1, 1, 1)], [(0, 0, 1), (1, 1, 1)], [(0, 0, 49), (1, 1, 2)], [(1, 1, 1)], [(0, 0, 1), (1, 1, 50)]):
            go(runs)
        gpu.reset(1)
        at[1] = 0
        for runs in ([(0, 0, 1), (1, 2, 3)], [(1, 2, 1)], [(0, 0, 1), (1, 2, 70)], [(0, 0, 1), (1, 2, 1)]):
            go(runs)
    finally:
        gpu.close()
