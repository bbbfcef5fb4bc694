"""Which products pairs of CTAs take (csrc/gemm_tc.cuh, tc_plan): only those whose K single CTAs would not cut, so that no sum changes its order for them.  Host logic."""
import pytest

SHAPES = [(4096, 6144, 4096, 14336), (2048, 2560, 2048, 5632), (896, 1152, 896, 4864), (1024, 1536, 1024, 4096), (2048, 3072, 2048, 8192), (8192, 10240, 8192, 28672), (5120, 7168, 5120, 13824)]


@pytest.mark.parametrize("hidden,qkv,heads,ffn", SHAPES)
def test_pairs_do_not_replace_cuts(b200, hidden, qkv, heads, ffn):
    taken = 0
    for rows in list(range(1, 400, 7)) + list(range(401, 4097, 53)) + [128, 129, 256, 257, 512, 640, 641, 700, 768, 1153, 1280, 2048, 4096]:
        for n, k, glu in ((qkv, hidden, False), (hidden, heads, False), (ffn, hidden, True), (hidden, ffn, False)):
            with_pairs, without = b200.tc_plan(rows, n, k, glu), b200.tc_plan(rows, n, k, glu, pairs=0)
            assert not without[3]
            if with_pairs[3]:
                assert without[2] == 1 and with_pairs[2] == 1 and rows > 128
                taken += 1
            else:
                assert with_pairs == without
    assert taken > 20      # (and they are taken)


def test_sums_that_may_not_be_cut_take_pairs_too(b200):
    assert b200.tc_plan(700, 4096, 14336)[2:] == (2, 0)      # cut in two: no pair in its place
    assert b200.tc_plan(700, 4096, 14336, may_cut=False)[2:] == (1, 1)
