"""Contexts beside a program that keeps the legacy stream busy (torch's default stream): what a context clears or copies before its own stream reads it must not wait there.
A kernel that sleeps for half a second stands for the program's work; memory that the context gets was filled with ones before.  The same bits as without it."""
import numpy as np
import pytest
import torch

import synth

pytestmark = pytest.mark.gpu


def ones_behind():
    """Free device memory holds ones: a counter that nobody has cleared does not start at zero."""
    torch.cuda.empty_cache()
    free, _ = torch.cuda.mem_get_info()
    for x in [torch.ones(min(free, 8 << 30) // 4, dtype=torch.int32, device="cuda")]:
        torch.cuda.synchronize()
        del x
    torch.cuda.empty_cache()


def busy():
    torch.cuda._sleep(1_000_000_000)


def both(call):
    call()               # (kernels loaded)
    want = call()
    ones_behind()
    torch.cuda.synchronize()
    got = call(busy)
    torch.cuda.synchronize()
    assert len(got) == len(want)
    for a, b in zip(got, want):
        assert np.array_equal(a, b)


@pytest.mark.parametrize("n", [2, 5])
def test_first_step_of_several_sequences(b200, n):
    """Splits of the keys merged by tickets that the first step brings (csrc/engine.cu, exact_rows_room)."""
    arch, desc, tensors = synth.synth_model("llama-tiny", "Q4_K_M", 160, max_batch=n)

    def call(first=lambda: None):
        gpu = b200.GpuOnlyInference(desc, tensors)
        try:
            for s in range(n):
                gpu.debug_set_position(100 + s, s)
            first()
            return [gpu.decode_batch(list(range(n)), [3 + k + s for s in range(n)]) for k in range(3)]
        finally:
            gpu.close()
    both(call)


@pytest.mark.parametrize("preset", ["mixtral-tiny", "llama-tiny"])
def test_loading(b200, preset):
    """Counters of the router and of cut tiles, caches and states, all cleared while the context is made."""
    arch, desc, tensors = synth.synth_model(preset, "Q4_K_M", 96)

    def call(first=lambda: None):
        first()
        gpu = b200.GpuOnlyInference(desc, tensors)
        try:
            return [gpu.forward(t) for t in (5, 9, 4)]
        finally:
            gpu.close()
    both(call)
