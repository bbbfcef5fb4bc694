"""The scans of prompts in chunks of 32 tokens (csrc/lp_chunk_scan.cuh) against the scans that go token by token (B200_LP_CHUNK_SCAN=0), f32
compute: runs that end inside a chunk, fill it and pass it by one, several unequal runs in a step (a single token among them), portions that continue
a state and decoding from it, key and value sizes inside and at the edges of the kernels' blocks.  Both are f32 sums of the same terms in
another order; the bound is the one the models' f32 tests hold against their float64 oracles (2e-4)."""
import numpy as np
import pytest

import lazilorn_synth as LS
import madudra_synth as MS

pytestmark = pytest.mark.gpu


def both(monkeypatch, S, cfg, lens, more):
    w = S.random_weights(cfg, 3)
    rng = np.random.default_rng(sum(lens))
    runs = [(i, [int(t) for t in rng.integers(0, cfg["vocab"], n)]) for i, n in enumerate(lens)]
    cont = [int(t) for t in rng.integers(0, cfg["vocab"], more)]
    outs, launches = {}, {}
    for on in ("1", "0"):
        monkeypatch.setenv("B200_LP_CHUNK_SCAN", on)
        gpu = S.gpu_model(cfg, w, "float32", max_seq_len=max(lens) + more + 8)
        try:
            first = gpu.step(runs, list(range(sum(lens))))
            second = gpu.step([(0, cont)], list(range(more)))
            last = gpu.step([(0, cont[:1])], [0])
            outs[on] = np.concatenate([first, second, last])
            launches[on] = gpu.stats()["kernel_launches"]
        finally:
            gpu.close()
    assert launches["1"] == launches["0"] + 2, launches        # both prompts went in chunks: two kernels for one, in the only scan of the model
    assert S.rel_err(outs["1"], outs["0"]) < 2e-4


@pytest.mark.parametrize("lens,more", [((48, 1, 33), 65), ((64, 31), 48), ((129, 96, 32), 50), ((300,), 61)])
@pytest.mark.parametrize("layer", [LS.delta_layer(heads=4, kv_heads=2, dim=16, vdim=24, conv=3), LS.delta_layer(heads=2, kv_heads=2, dim=128, vdim=128, conv=4),
                                   LS.delta_layer(heads=2, kv_heads=1, dim=68, vdim=4, conv=1),
                                   LS.parallel_layer(left_scale=0.0, right_scale=1.0, mheads=2, mdim=16, mvdim=24, ff=0),
                                   LS.parallel_layer(left_scale=0.0, right_scale=1.0, mheads=4, mdim=64, mvdim=128, ff=0),
                                   LS.parallel_layer(left_scale=0.0, right_scale=1.0, mheads=4, mdim=100, mvdim=8, cap=2.0, ff=0)])
def test_delta_rule_and_matrix_memory(b200, monkeypatch, layer, lens, more):
    both(monkeypatch, LS, LS.config([layer], width=64, vocab=80), lens, more)


@pytest.mark.parametrize("lens,more", [((129, 1, 96), 160), ((128, 31), 129), ((300,), 133)])
@pytest.mark.parametrize("sizes", [dict(heads=4, vdim=8, state=16, groups=2, conv=4), dict(heads=2, vdim=128, state=128, groups=1, conv=4), dict(heads=4, vdim=20, state=72, groups=1, conv=3)])
def test_state_space(b200, monkeypatch, sizes, lens, more):
    both(monkeypatch, MS, MS.config([MS.scan(**sizes)]), lens, more)
