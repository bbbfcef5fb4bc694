"""The selected experts of a token in one launch per product (csrc/gemv_mma.cuh, n_slots) against the CUDA-core products, one expert after the other (B200_GEMV_MMA=0).
Two and three experts (148 CTAs do not split by three), tiles cut between the CTAs of one expert, a ragged last tile.  f32 sums in another order, activations to 21 bits of a
group's largest: 1e-5 of the largest logit."""
import pytest

import synth
from synth import rel_err

pytestmark = pytest.mark.gpu
synth.TINY["experts-wide"] = dict(synth.TINY["mixtral-tiny"], hidden=1024, n_layers=1, n_heads=8, n_kv_heads=2, head_dim=128, ffn=8192, n_experts=3)


@pytest.mark.parametrize("mix,used,ffn", [("Q5_K_M", 2, 8192), ("Q4_K_M", 3, 8192), ("Q8_0", 2, 8224)])
def test_experts_in_one_launch(b200, monkeypatch, mix, used, ffn):
    monkeypatch.setitem(synth.TINY, "experts-wide", dict(synth.TINY["experts-wide"], n_experts_used=used, ffn=ffn))
    arch, desc, tensors = synth.synth_model("experts-wide", mix, 32)
    out, count = {}, {}
    for mma in ("1", "0"):
        monkeypatch.setenv("B200_GEMV_MMA", mma)
        gpu = b200.GpuOnlyInference(desc, tensors)
        try:
            gpu.forward(1)
            before = gpu.stats()["kernel_launches"]
            out[mma] = [gpu.forward(t) for t in (5, 9, 400)]
            count[mma] = gpu.stats()["kernel_launches"] - before
        finally:
            gpu.close()
    assert count["0"] - count["1"] == 3 * (2 * used - 3), count      # two launches and the sum instead of two per expert
    assert max(rel_err(a, b) for a, b in zip(out["1"], out["0"])) < 1e-5
