"""Products of one to four rows whose weight loads come eight to a round (layerprog.cu, gemv_dot: rounds of 8 x 32 x 16 bytes per warp): less than one round, one more
or fewer 16-byte word than a round, two rounds and a rest; one and two rows take the rounds, three and four the plain loop.  Steps of single tokens against the
float64 oracle, sequence by sequence.  The f32 bound is the models'; bf16's is the models' (6e-2) or, for an input whose row magnifies rounding, what f32 shows of it
at bf16's rounding: 2^15 times the f32 error of the same step, and 4 for two draws of the same rounding (one of the tokens here: 1.4e-5 in f32, 0.74 in bf16, 1.6 x 2^15)."""
import numpy as np
import pytest

import lazilorn_oracle as O
import lazilorn_synth as S

pytestmark = pytest.mark.gpu
F32_TOL, BF16_TOL = 2e-4, 6e-2


def steps(cfg, w, toks, compute):
    gpu = S.gpu_model(cfg, w, compute, max_seq_len=16)
    try:
        return [np.atleast_2d(gpu.step([(r, [int(t)]) for r, t in enumerate(col)], list(range(len(col))))) for col in toks.T]
    finally:
        gpu.close()


@pytest.mark.parametrize("rows", [1, 2, 3, 4])
@pytest.mark.parametrize("ff", [24, 1016, 1032, 2040, 2056, 4424])
def test_rows_against_the_oracle(b200, ff, rows):
    cfg = S.config([S.parallel_layer(ff=ff), S.delta_layer(ff=ff)])
    w = S.random_weights(cfg, ff)
    toks = np.random.default_rng(rows).integers(0, cfg["vocab"], (rows, 5))
    want = [O.Model(cfg, w).forward([int(t) for t in row]) for row in toks]
    f32, b16 = steps(cfg, w, toks, "float32"), steps(cfg, w, toks, "bfloat16")
    for r in range(rows):
        for t in range(5):
            e = S.rel_err(f32[t][r], want[r][t])
            assert e < F32_TOL
            assert S.rel_err(b16[t][r], want[r][t]) < max(BF16_TOL, 4 * 2 ** 15 * e)
