"""Which kernel a float32 product takes: both sides of the lines that `pick_form` draws (csrc/gemm_simt.cu)."""
import pytest

ROWS = -1


@pytest.mark.parametrize("m,n,k,heads,form", [
    (5, 1024, 1024, 1, 0), (28, 1024, 1024, 1, 0), (300, 1024, 1024, 1, 1), (700, 768, 768, 1, 3), (2050, 2050, 1024, 1, 3),
    # K up to 16, but few rows of few columns
    (16, 2050, 16, 1, ROWS), (64, 768, 16, 1, ROWS), (2050, 2050, 16, 1, ROWS), (64, 64, 16, 1, 0), (16, 2050, 20, 1, 0),
    # a K in the first half of a stage, with more tiles than SMs
    (700, 2050, 136, 1, ROWS), (700, 2050, 144, 1, ROWS), (700, 2050, 148, 1, 3), (700, 2050, 160, 1, 3), (700, 2050, 520, 1, 3),
    (700, 768, 136, 1, 3), (700, 768, 36, 1, ROWS), (500, 1280, 136, 1, ROWS), (500, 1280, 200, 1, 2), (300, 768, 136, 1, 2),
    # four and a part of the tiles to an SM
    (1300, 2050, 128, 1, ROWS), (1300, 2050, 768, 1, 3), (2050, 2050, 128, 1, 3), (65, 1280, 128, 11, 3), (64, 1280, 128, 33, ROWS),
    # few rows of many columns, short K
    (16, 4592, 64, 1, 1), (16, 4608, 64, 1, ROWS), (8, 9216, 72, 1, ROWS), (16, 4608, 100, 1, 0), (4, 4608, 64, 1, 0), (16, 1280, 72, 1, 1), (16, 768, 72, 1, 0)])
def test_the_form_of_a_float32_product(m, n, k, heads, form):
    from crucible_b200.ops import build
    assert build.load("gemm_simt").cb_gemm_simt_form(m, n, k, heads) == form


@pytest.mark.parametrize("m,tallest", [(16 * 65535, 16), (16 * 65535 + 1, 32), (32 * 65535, 32), (32 * 65535 + 1, 64), (64 * 65535, 64)])
def test_a_grid_has_room_for_every_tile_of_rows(m, tallest):
    """Few columns, for which the smallest tiles are the cheapest: a form whose tiles of rows a grid can hold."""
    from crucible_b200.ops import build
    rows = {0: 16, 1: 32, 2: 64, 3: 64, ROWS: 64}[build.load("gemm_simt").cb_gemm_simt_form(m, 8, 64, 1)]
    assert rows >= tallest and -(-m // rows) <= 65535
