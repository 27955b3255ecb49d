"""Which kernels a product takes: the rules, and the test hooks that override them, on the host."""
import pytest

from tinyllama_c_b200 import ops


def test_tiles_that_do_not_exist_cannot_be_asked_for():
    """Shares of a tile's rows that are no whole numbers would leave rows out, more blocks than eight their sums."""
    chosen = ops.linear_f32_plan(310, 2048, 2048, 148)
    try:
        for rows, split in ((32, 1), (32, 8), (64, 0), (64, -4), (64, 2), (64, 8)):
            ops.linear_f32_tiles(rows, split)
            assert ops.linear_f32_plan(310, 2048, 2048, 148) == (rows, split)
        for rows, split in ((32, 0), (32, 3), (64, 5), (64, 16), (64, -1), (48, 4), (0, 4)):
            with pytest.raises(ops.KernelError, match="no 32-bit tiles"):
                ops.linear_f32_tiles(rows, split)
            ops.library().tlc_linear_f32_tiles(rows, split)          # the library's own entry: as if nothing had been asked for
            assert ops.linear_f32_plan(310, 2048, 2048, 148) == chosen
    finally:
        ops.linear_f32_tiles(0)
    assert ops.linear_f32_plan(310, 2048, 2048, 148) == chosen


@pytest.mark.parametrize("K,N,M,plan", [
    # one block a tile where K is short: what a cluster costs is more than what it brings (microseconds, one block and the cluster)
    (32, 2048, 1200, (64, 0)), (256, 2048, 1200, (64, 0)), (128, 8192, 310, (64, 0)),          # 9.4 / 39.5, 43.1 / 58.6, 24.1 / 49.2
    (32, 512, 310, (64, -4)), (64, 2048, 48, (64, -4)), (256, 8192, 48, (64, -4)),             # 4.2 / 6.8, 5.0 / 6.2, 12.0 / 14.7
    # and where the output has no use for tiles of 256 columns, however long K is
    (1024, 64, 3000, (64, -4)), (12288, 64, 3000, (64, -4)),                                    # 36 / 56
    # clusters elsewhere, as the kernels were fitted
    (128, 64, 17, (32, 8)), (512, 2048, 17, (32, 8)), (1024, 2048, 48, (32, 8)),                # 6.6 / 3.3, 18.7 / 10.6, 35.3 / 19.7
    (1024, 2048, 130, (64, 8)), (2048, 2048, 310, (64, 8)), (4096, 2048, 310, (64, 8)),         # 36.6 / 34.5, 134 / 93, 264 / 179
    (2048, 8192, 17, (32, 8)), (2048, 8192, 130, (64, 4)), (2048, 8192, 1200, (64, 0)), (4096, 2048, 17, (32, 8))])
def test_tiles_of_32_bit_products_by_their_sizes(K, N, M, plan):
    assert ops.linear_f32_plan(M, N, K, 148) == plan


@pytest.mark.parametrize("N,K,takes", [
    (2368, 4096, False), (2384, 4096, True), (2384, 4064, False),               # 148 tiles and 149; a K of 127 steps
    (3328, 4096, True), (3329, 4096, False), (3552, 5384, False),               # 208 tiles are 104 clusters, all at once; 209
    (3552, 8192, True), (3553, 8192, False), (3552, 12288, True), (4064, 12288, False)])
def test_rings_of_17_to_32_rows_where_all_clusters_run_at_once(N, K, takes):
    """Beyond that a second round of clusters costs more than the ring brings, up to K = 8192 (figures beside the rule)."""
    assert bool(ops.library().tlc_linear_skinny_ring_takes(N, K, 148, 104)) == takes


@pytest.mark.parametrize("N,K,plain,activation", [
    (4736, 2048, False, False), (4752, 2048, True, False), (9472, 2048, True, True), (9488, 2048, False, False),   # 296, 297, 592, 593 tiles
    (8192, 1024, False, False), (8192, 1032, True, True), (8192, 2056, False, False),                              # one round of K
    (4752, 1032, True, True), (4752, 1280, True, False), (5600, 1280, True, True), (5600, 1800, True, False), (6400, 1800, True, True),
    (5600, 2048, True, False), (6400, 2048, True, True)])
def test_two_tiles_a_block_where_that_is_quicker(N, K, plain, activation):
    """With the gated activation a little later than without (figures beside the rule)."""
    takes = ops.library().tlc_linear_skinny_two_takes
    assert (bool(takes(N, K, 0, 148)), bool(takes(N, K, 1, 148))) == (plain, activation)
