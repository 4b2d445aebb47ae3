"""Rules that size the launches of a bucket's plan (host side only)."""
import math

import pytest

from conef_b200.parallel.engine import decompress_rows


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
