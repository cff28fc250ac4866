"""Which products one block an SM walks tile by tile (`_waves_width`, `grouped_waves`): both sides of every line."""
import pytest


@pytest.mark.parametrize("m,n,k,epi,width", [
    # gated pairs (2 x n columns): from 200 tiles of 256 on
    (1100, 2 * 2816, 2048, "SWIGLU_BF16", 0), (1200, 2 * 2816, 2048, "SWIGLU_BF16", 256), (2048, 2 * 2048, 768, "SWIGLU_BF16", 256),
    # bfloat16 results: at 256 columns from two waves on, at 192 from three or at a short K, from four by a long one
    (1100, 8192, 2048, "STORE_BF16", 256), (2048, 5120, 2048, "STORE_BF16", 192), (2048, 3072, 1024, "STORE_BF16", 192),
    (1600, 6144, 4096, "STORE_BF16", 0), (1800, 6144, 4096, "STORE_BF16", 256), (1100, 4608, 2048, "STORE_BF16", 0),
    # float32 results: more than a wave; by a long K 1.4 waves, and not where tall tiles fill their waves with half as many
    (1100, 4096, 128, "STORE_F32", 0), (1300, 4096, 128, "STORE_F32", 192), (1300, 4096, 1024, "STORE_F32", 192),
    (1300, 4096, 2048, "STORE_F32", 0), (1100, 6144, 2048, "STORE_F32", 192), (2048, 4096, 512, "STORE_F32", 256),
    (2048, 4096, 2048, "STORE_F32", 0), (2048, 8192, 2048, "STORE_F32", 0), (3000, 8192, 2048, "STORE_F32", 0),
    (1300, 16384, 2048, "STORE_F32", 256), (2048, 50304, 2048, "STORE_F32", 256), (2048, 50304, 768, "STORE_F32", 256),
    (100, 50304, 2048, "STORE_F32", 192), (64, 4096, 2048, "STORE_F32", 0),
    # sums into rows, rotated rows: never
    (2048, 50304, 768, "ACCUM_F32", 0), (2048, 8192, 2048, "ROPE_APPEND", 0)])
def test_products_in_waves_by_size(m, n, k, epi, width):
    from crucible_b200.ops import tensor_core as tc
    got = tc._waves_width(m, n, k, getattr(tc, epi))
    assert bool(got) == bool(width) and got in (0, 192, 256)
    assert width == 0 or got == width


def test_a_rule_of_sizes_alone():
    from crucible_b200.ops import tensor_core as tc
    for m in (1, 65, 128, 129, 513, 2047, 2048, 9000):
        for n in (64, 768, 4096, 50304):
            for k in (64, 768, 1024, 2048, 4096):
                for epi in range(5):
                    assert tc._waves_width(m, n, k, epi) in (0, 192, 256)
                    assert epi != tc.SWIGLU_BF16 or tc._waves_width(m, n, k, epi) != 192


@pytest.mark.parametrize("pairs,experts,cols,waves", [
    (4096, 8, 2 * 2816, True), (4096, 8, 2048, True), (2048, 8, 2 * 2816, True), (2048, 8, 2048, False), (1024, 8, 2 * 2816, True),
    (500, 8, 2 * 5632, False), (4096, 128, 2 * 2816, False), (8192, 128, 2 * 768, True), (64, 1, 2 * 2816, False)])
def test_grouped_products_in_waves_by_size(pairs, experts, cols, waves):
    from crucible_b200.ops import tensor_core as tc
    assert tc.grouped_waves(pairs, experts, cols) is waves
