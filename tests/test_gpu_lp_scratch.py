"""Scratch that steps of the layer programs keep (bf16 keys, terms of the chunked scans) against the memory that a step has to have."""
import numpy as np
import pytest
import torch

import lazilorn_synth as S

pytestmark = pytest.mark.gpu


def test_a_slot_takes_the_room_of_kept_scratch(b200):
    """A prompt of 16384 tokens leaves 128 MiB of bf16 keys behind; with 192 MiB free, a second slot of 256 MiB fits only where they were."""
    n = 16384
    cfg = S.config([S.parallel_layer(heads=16, kv_heads=16, dim=128, vdim=128, window=256, keep_first=0, ff=0)], width=64, vocab=80)
    w = S.random_weights(cfg, 5)
    toks = [int(t) for t in np.random.default_rng(0).integers(0, cfg["vocab"], n)]
    gpu = S.gpu_model(cfg, w, "bfloat16", max_seq_len=n + 16, max_batch=2)
    try:
        gpu.step([(0, toks)], [n - 1])
        short = toks[:40]
        torch.cuda.empty_cache()
        free, _ = torch.cuda.mem_get_info()
        block = torch.empty(free - (192 << 20), dtype=torch.uint8, device="cuda")
        tight = gpu.step([(1, short)], [39])
        del block
        torch.cuda.empty_cache()
        gpu.reset(1)
        assert S.rel_err(tight, gpu.step([(1, short)], [39])) < 2e-2       # (bf16 keys and probabilities; either attention kernel)
    finally:
        gpu.close()
