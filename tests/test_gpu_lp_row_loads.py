"""Products of one to four rows whose weight loads come eight to a round (layerprog.cu, gemv_dot: rounds of 8 x 32 x 16 bytes per warp): less than one round, one more
or fewer 16-byte word than a round, two rounds and a rest; one and two rows take the rounds, three and four the plain loop.  Steps of single tokens against the
float64 oracle, sequence by sequence, within the models' bounds (weights and tokens are drawn so that no row magnifies bf16's rounding), and the rounds against the plain
loop bit for bit: both add a lane's products in the order of K."""
import numpy as np
import pytest

import lazilorn_oracle as O
import lazilorn_synth as S

pytestmark = pytest.mark.gpu
TOL = {"float32": 2e-5, "bfloat16": 6e-2}
FF = [24, 1016, 1032, 2040, 2056, 4424]


def model(ff):
    cfg = S.config([S.parallel_layer(ff=ff), S.delta_layer(ff=ff)])
    return cfg, S.random_weights(cfg, ff + 4), np.random.default_rng([4, 4]).integers(0, cfg["vocab"], (4, 5))


def steps(cfg, w, toks, compute):
    gpu = S.gpu_model(cfg, w, compute, max_seq_len=16)
    try:
        return [np.atleast_2d(gpu.step([(r, [int(t)]) for r, t in enumerate(col)], list(range(len(col))))) for col in toks.T]
    finally:
        gpu.close()


@pytest.mark.parametrize("rows", [1, 2, 3, 4])
@pytest.mark.parametrize("ff", FF)
def test_rows_against_the_oracle(b200, ff, rows):
    cfg, w, toks = model(ff)
    want = [O.Model(cfg, w).forward([int(t) for t in row]) for row in toks[:rows]]
    for compute, tol in TOL.items():
        got = steps(cfg, w, toks[:rows], compute)
        assert max(S.rel_err(got[t][r], want[r][t]) for r in range(rows) for t in range(5)) < tol, compute


@pytest.mark.parametrize("compute", ["float32", "bfloat16"])
@pytest.mark.parametrize("ff", FF)
def test_rounds_and_the_plain_loop_give_the_same_bits(b200, monkeypatch, ff, compute):
    monkeypatch.setenv("B200_LP_GEMV_MMA", "0")      # (four bf16 rows on the CUDA cores as well)
    cfg, w, toks = model(ff)
    four = steps(cfg, w, toks, compute)
    for rows in (1, 2):
        for a, b in zip(four, steps(cfg, w, toks[:rows], compute)):
            assert np.array_equal(a[:rows], b)
