"""Several rows at once in f32 (csrc/exact_rows.cuh) against the same calls token by token (B200_EXACT_ROWS=0): short prompts, prompts of models whose blocks the
tensor-core products do not take, prompts into an int8 cache, steps of fewer than eight sequences; row counts at the edges of the warp passes (2, 4, 8), of that
kernel's range (32) and of the tiles (32, 64).

Tolerance: both sides sum in f32 (or in integers, to 21 bits of a group's largest activation); one product's sums differ by some 3e-7 of their size, seven
products a layer and three layers give 1e-5 of the largest logit.  A wrong row, block or piece is off by the size of the logits.  Int8 caches: a key or value that
lies within such a difference of the middle between two codes takes the other one, 1/127 of the row's largest element away: 1e-3, the bound of that format."""
import numpy as np
import pytest

import synth
from synth import rel_err

pytestmark = pytest.mark.gpu
TOL = 1e-5
# every weight type; a width that needs K in portions (8 rows of 10240), 16 query heads over 4
synth.TINY["rows-q4_0"] = dict(synth.TINY["llama-tiny"], hidden=256, n_heads=4, n_kv_heads=2, head_dim=64, ffn=352, vocab=300)
synth.TINY["rows-wide"] = dict(synth.TINY["llama-tiny"], hidden=512, n_layers=1, n_heads=4, n_kv_heads=1, ffn=10240, vocab=300)
SHORT = [("qwen-tiny", "Q4_K_M"), ("llama-tiny", "Q4_K_M"), ("llama-tiny", "Q5_K_M"), ("tinyllama-tiny", "Q8_0"), ("rows-wide", "Q6_K"), ("rows-q4_0", "Q4_0"), ("rows-q4_0", "F16")]


def both(b200, monkeypatch, desc, tensors, call, **kw):
    out, count = [], []
    for on in ("1", "0"):
        monkeypatch.setenv("B200_EXACT_ROWS", on)
        gpu = b200.GpuOnlyInference(desc, tensors, **kw)
        before = gpu.stats()["kernel_launches"]
        try:
            out.append(call(gpu))
            count.append(gpu.stats()["kernel_launches"] - before)
        finally:
            gpu.close()
    assert count[0] != count[1], count      # (another path)
    return [max(rel_err(a, b) for a, b in zip(np.atleast_2d(x), np.atleast_2d(y))) for x, y in zip(*out)]


def prompts(lens, vocab):
    """A prompt, a portion behind it, a single token that reads both."""
    def call(gpu):
        t = synth.prompt_tokens(sum(lens), vocab)
        out, at = [], 0
        for n in lens:
            out.append(gpu.prefill(t[at:at + n]))
            at += n
        return out + [gpu.forward(3)]
    return call


@pytest.mark.parametrize("preset,mix", SHORT)
@pytest.mark.parametrize("lens", [(2, 3), (4, 5), (8, 9), (31, 17)])
def test_short_prompts(b200, monkeypatch, preset, mix, lens):
    arch, desc, tensors = synth.synth_model(preset, mix, 64)
    assert max(both(b200, monkeypatch, desc, tensors, prompts(lens, desc["vocab"]))) < TOL


@pytest.mark.parametrize("lens", [(32,), (33, 32), (64,), (65, 40), (200, 100)])
@pytest.mark.parametrize("preset,mix", [("qwen-tiny", "Q4_K_M"), ("rows-q4_0", "Q4_0")])
def test_prompts_in_tiles(b200, monkeypatch, preset, mix, lens):
    arch, desc, tensors = synth.synth_model(preset, mix, 320)
    assert max(both(b200, monkeypatch, desc, tensors, prompts(lens, desc["vocab"]))) < TOL


@pytest.mark.parametrize("preset,mix", [("llama-tiny", "Q4_K_M"), ("llama-tiny", "Q6_K"), ("tinyllama-tiny", "Q8_0")])
def test_tiles_of_the_block_types_of_256(b200, monkeypatch, preset, mix):
    monkeypatch.setenv("B200_PREFILL_GEMM_MIN", "1000")
    arch, desc, tensors = synth.synth_model(preset, mix, 160)
    assert max(both(b200, monkeypatch, desc, tensors, prompts((100, 45), desc["vocab"]))) < TOL


@pytest.mark.parametrize("preset,mix", [("qwen-tiny", "Q4_K_M"), ("llama-tiny", "Q4_K_M")])
@pytest.mark.parametrize("lens", [(2, 3), (5, 9), (31, 16)])
def test_int8_prompts(b200, monkeypatch, preset, mix, lens):
    arch, desc, tensors = synth.synth_model(preset, mix, 64)
    assert max(both(b200, monkeypatch, desc, tensors, prompts(lens, desc["vocab"]), kv_format="int8")) < 1e-3


@pytest.mark.parametrize("preset,mix,n", [("llama-tiny", "Q4_K_M", 2), ("llama-tiny", "Q5_K_M", 7), ("tinyllama-tiny", "Q8_0", 5), ("qwen-tiny", "Q4_K_M", 3), ("qwen-tiny", "Q4_K_M", 19)])
def test_steps_of_sequences(b200, monkeypatch, preset, mix, n):
    """Slots at different positions, one past a split of the keys; eager, captured and replayed, then the pick on the device."""
    arch, desc, tensors = synth.synth_model(preset, mix, 96, max_batch=n)
    rng = np.random.default_rng(n)
    steps = [rng.integers(0, desc["vocab"], n).astype(np.uint32) for _ in range(3)]

    def call(gpu):
        for s in range(n):
            for t in range(1 + 23 * s % 70):
                gpu.prefill_token(int(t % desc["vocab"]), s)
        out = [gpu.decode_batch(list(range(n)), t) for t in steps]
        assert len(gpu.decode_batch_greedy(list(range(n)), steps[0])) == n
        return out
    assert max(both(b200, monkeypatch, desc, tensors, call)) < TOL


@pytest.mark.parametrize("preset,mix,kv", [("qwen-tiny", "Q4_K_M", "int8"), ("llama-tiny", "Q4_K_M", "f32")])
def test_first_short_prompt_allocates_nothing(b200, preset, mix, kv):
    """The buffers of up to 32 rows come with the context."""
    import torch
    arch, desc, tensors = synth.synth_model(preset, mix, 64)
    for _ in range(2):      # (kernels loaded)
        gpu = b200.GpuOnlyInference(desc, tensors, kv_format=kv)
        try:
            before = gpu.stats()["kernel_launches"], torch.cuda.mem_get_info()[0]
            gpu.prefill(synth.prompt_tokens(31, desc["vocab"]))
            launches, free = gpu.stats()["kernel_launches"] - before[0], torch.cuda.mem_get_info()[0]
        finally:
            gpu.close()
    assert launches < 31 * desc["n_layers"]      # (as rows)
    assert free == before[1]


@pytest.mark.parametrize("n", [40, 100])
def test_rows_are_no_further_from_float64_than_token_by_token(b200, monkeypatch, n):
    """Prompts in tiles: root mean square of the distances over eight inputs, which spreads by 3 %."""
    from perf import cases
    case = dict(family="gguf", preset="qwen2.5-0.5b", layers=2, vocab=4096, mix="Q4_K_M", kv="f32", batch=1, prompt=n, decode=0)
    err = {"1": [], "0": []}
    for seed in range(201, 209):
        want = cases.exact(case, seed)[0].cpu().numpy()
        for on in err:
            monkeypatch.setenv("B200_EXACT_ROWS", on)
            state = cases.prepare(case, seed)
            got = np.asarray(cases.run(state)[0], dtype=np.float64)
            state["gpu"].close()
            err[on].append(np.linalg.norm(got - want) / np.linalg.norm(want))
    rows, tokens = (float(np.sqrt(np.mean(np.square(err[on])))) for on in ("1", "0"))
    print(f"{n} tokens: rows {rows:.3e}, token by token {tokens:.3e}")
    assert rows < 1.05 * tokens
