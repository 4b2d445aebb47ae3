"""Rules that size the launches of a bucket's plan (host side only)."""
import math

import pytest

from conef_b200.parallel.engine import decompress_rows, one_wave_extent, split_k


def _block_ctas(shapes):
    return lambda rows: sum(math.ceil(math.ceil(n / rows) * (w // 32) / 8) for n, w in shapes)


@pytest.mark.parametrize("shapes,rows", [([(640, 576)] * 2, 8), ([(30528, 102)], 8), ([(640, 576)], 4), ([(4096, 102)], 4),
                                         ([(1024, 102)], 4), ([(512, 102)], 2), ([(64, 115)] * 4, 1), ([], 1), ([(1, 64)], 1)])
def test_decompress_rows_of_block_layout_matrices(shapes, rows):
    """The measured best (or within 3 % of it) for matrices of the count sketch's block layout: (rows, sketch width)."""
    assert decompress_rows(_block_ctas(shapes), 0, 0) == rows


@pytest.mark.parametrize("off_rows,width,rows", [(3552, 0, 8), (3551, 0, 4), (888, 10, 2), (887, 10, 1), (10_000, 1600, 8),
                                                 (10_000, 1601, 4), (10_000, 12_801, 1), (10_000, 50_000, 1)])
def test_decompress_rows_of_column_order_matrices(off_rows, width, rows):
    """Three row blocks per SM, and one accumulator row of the sketch per matrix row in 50 KB of shared memory."""
    assert decompress_rows(_block_ctas([]), off_rows, width) == rows


@pytest.mark.parametrize("dims", [[(512, 512), (512, 52)], [(640, 5760)] * 2 + [(640, 576)] * 2, [(5760, 640)] * 2 + [(576, 640)] * 2,
                                  [(1024, 30528), (104, 30528)], [(1, 1)], [(16, 27), (129, 33)], [(128 * 296, 64)],
                                  [(1024, 1 << 20)]])
def test_one_wave_extent_fits_and_covers(dims):
    """All CTAs are resident at once, and the CTAs of a product cover its K range in multiples of 32."""
    extent = one_wave_extent(dims)
    assert extent % 32 == 0 and extent >= 128
    total = 0
    for mn, K in dims:
        tiles, klen, splits = split_k(mn, K, extent)
        assert klen % 32 == 0 and (splits - 1) * klen < K <= splits * klen and tiles * 128 >= mn
        total += tiles * splits
    assert total <= 296


def test_one_wave_extent_gives_up_on_too_many_output_tiles():
    assert one_wave_extent([]) is None
    assert one_wave_extent([(128 * 297, 64)]) is None
    assert one_wave_extent([(30528, 1024), (30528, 104)]) is None
