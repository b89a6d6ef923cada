"""Quantised products whose codes go to the tensor pipe as integers (uzu_b200/csrc/qmm_scaled.cu, tiles of up to 64 rows, groups of 64 and more): chains
that are a block, two, or half a group; a chain cut off by the last block; rows at the edges of an epilogue warp's columns; a split k."""
import pytest

from tests.test_qmm_scaled_gpu import check

pytestmark = [pytest.mark.gpu]


@pytest.mark.parametrize("bits,gs,method", [(4, 64, "zero"), (4, 64, "symmetric"), (8, 64, "zero"), (4, 128, "zero"), (8, 128, "symmetric"), (4, 256, "zero"), (8, 256, "zero")])
@pytest.mark.parametrize("m,n,k", [(33, 9000, 768), (48, 2200, 1280), (64, 300, 2816), (63, 17000, 256), (41, 130, 14336)])
def test_integer_codes(ctx, bits, gs, method, m, n, k):
    check(ctx, m, n, k, bits, gs, method)


@pytest.mark.parametrize("splits", [1, 2, 4, 8])
@pytest.mark.parametrize("rows", [16, 32, 64])
def test_tiles_and_splits(ctx, rows, splits):
    """An odd number of blocks, so that the last rank's last chain of two is one."""
    try:
        assert ctx.lib.uzu_debug_set_qmm_tile(rows, splits)
        check(ctx, 90, 200, 27 * 64, 4, 64, "zero")
        check(ctx, 90, 200, 31 * 128, 8, 128, "zero")
    finally:
        ctx.lib.uzu_debug_set_qmm_tile(0, 0)
