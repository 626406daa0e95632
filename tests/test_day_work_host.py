"""What the batched day's work buffer holds per pixel."""
import pytest


@pytest.mark.parametrize("rows,cols", [(2000, 2000), (517, 389)])
def test_a_day_reserves_no_second_copy_of_the_walk_words(rows, cols):
    """Quads 16, ground view factors 12 and patch sums 16 bytes per pixel and hour,
    the albedo without shadow 4 per pixel; tables, rays and the tiles' samples add
    less than 2 % and 3 MB."""
    from solweig_cuda_b200 import _lib
    got = _lib.lib().solweig_day_batched_work_bytes(rows, cols, 24, 0)
    assert got <= 1.02 * rows * cols * (24 * (16 + 12 + 16) + 4) + 3e6
