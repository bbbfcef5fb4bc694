"""The norm of a prompt's rows before its fp16 products (csrc/prefill.cuh): rows by 16-byte words add their squares in the order of the kernel for rows of any length, so
the same bits.  Lengths at the edges of the instances (1024, 2048, 4096, 8192) and of a block's words, and the first length that no instance takes."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [8, 64, 896, 1020, 1024, 1028, 2048, 2056, 4096, 4100, 8192, 8200])
def test_words_and_elements_give_the_same_bits(b200, n):
    """160 rows: another order of the sum moves 1 / rms by a last place in every third row, and with it about one of 6000 fp16 results."""
    rng = np.random.default_rng(n)
    x = (rng.standard_normal((160, n)) * np.exp(rng.standard_normal((160, 1)))).astype(np.float32)
    w = (1.0 + 0.1 * rng.standard_normal(n)).astype(np.float32)
    got, want = b200.prompt_norm(x, w, 1e-5), b200.prompt_norm(x, w, 1e-5, any_length=True)
    assert np.array_equal(got.view(np.uint16), want.view(np.uint16))
    exact = x.astype(np.float64) / np.sqrt((x.astype(np.float64) ** 2).mean(1, keepdims=True) + 1e-5) * w
    assert np.abs(got - exact).max() < 2 ** -11 * 1.001 * np.abs(exact).max()
