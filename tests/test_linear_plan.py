"""Which tiles a 32-bit product takes: the rule and the test hook that overrides it, on the host."""
import pytest

from tinyllama_c_b200 import ops


def test_tiles_that_do_not_exist_cannot_be_asked_for():
    """Shares of a tile's rows that are no whole numbers would leave rows out, more blocks than eight their sums."""
    chosen = ops.linear_f32_plan(310, 2048, 148)
    try:
        for rows, split in ((32, 1), (32, 8), (64, 0), (64, 2), (64, 8)):
            ops.linear_f32_tiles(rows, split)
            assert ops.linear_f32_plan(310, 2048, 148) == (rows, split)
        for rows, split in ((32, 0), (32, 3), (64, 5), (64, 16), (64, -1), (48, 4), (0, 4)):
            with pytest.raises(ops.KernelError, match="no 32-bit tiles"):
                ops.linear_f32_tiles(rows, split)
            ops.library().tlc_linear_f32_tiles(rows, split)          # the library's own entry: as if nothing had been asked for
            assert ops.linear_f32_plan(310, 2048, 148) == chosen
    finally:
        ops.linear_f32_tiles(0)
    assert ops.linear_f32_plan(310, 2048, 148) == chosen
