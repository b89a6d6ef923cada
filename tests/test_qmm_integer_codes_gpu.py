"""Quantised products whose codes go to the tensor pipe as integers (uzu_b200/csrc/qmm_scaled.cu, tiles of up to 64 rows, groups of 64 and more): chains
that are a block, two, or half a group; a chain cut off by the last block; rows at the edges of an epilogue warp's columns; a split k."""
import numpy as np
import pytest

from oracle import oracle as O
from tests import gpu_ops as G
from tests.test_qmm_scaled_gpu import METHODS, check
from tests.util import f32_to_bf16

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


ENDS = [(2e36, 2e-3), (2e37, 2e-4), (1e-3, 1e35), (1e-32, 3e-3)]        # activations and scales near the ends of the range, products inside it


def check_ends(ctx, m, n, bits, gs, method, size, scale):
    """A group's unscaled sum stays in range where the product does: codes all at one end, activations of one sign. Tolerance: `check`'s for sums of k f32
    products, without its share of the root mean square (nothing cancels here)."""
    rng = np.random.default_rng(bits + gs)
    k = 512
    w = np.full((n, k * bits // 8), 0xFF, np.uint8)
    scales = (scale * rng.uniform(0.5, 1.0, (n, k // gs))).astype(np.float32)
    kw = {"scales": f32_to_bf16(scales), "method": METHODS[method], "bits": bits, "group_size": gs}
    if method == "zero":
        kw["zero_points"] = np.zeros((n, -(-(k // gs) // 2) if bits == 4 else k // gs), np.uint8)
    elif method == "mlx":
        kw["biases"] = f32_to_bf16(8 * scales)
    x = f32_to_bf16((size * rng.uniform(0.5, 1.0, (m, k))).astype(np.float32) / (1 if bits == 4 else 16))
    got = G.matmul(ctx, x, w, m=m, n=n, k=k, d_f32=True, **kw)
    ref = O.matmul(x, w, m=m, n=n, k=k, d_f32=True, threads=8, **kw)
    assert np.isfinite(ref).all()
    assert np.all(np.abs(got - ref) <= 1e-3 * np.abs(ref)), float(np.abs(got / ref - 1).max())


@pytest.mark.parametrize("size,scale", ENDS)
@pytest.mark.parametrize("bits,gs,method", [(4, 64, "zero"), (4, 128, "symmetric"), (8, 64, "symmetric"), (8, 256, "zero")])
@pytest.mark.parametrize("rows", [16, 32, 64])
def test_numbers_near_the_ends_of_the_range(ctx, rows, bits, gs, method, size, scale):
    try:
        assert ctx.lib.uzu_debug_set_qmm_tile(rows, 1)
        check_ends(ctx, 40, 4200, bits, gs, method, size, scale)       # more than 2^21 weights: smaller ones go 16 rows at a time on the kernel for few rows
    finally:
        ctx.lib.uzu_debug_set_qmm_tile(0, 0)


@pytest.mark.parametrize("size,scale", ENDS)
@pytest.mark.parametrize("bits,gs,method", [(4, 64, "zero"), (4, 128, "symmetric"), (4, 64, "mlx"), (8, 64, "symmetric"), (8, 128, "zero"), (8, 64, "mlx")])
@pytest.mark.parametrize("m", [2, 11, 32])
def test_few_rows_near_the_ends_of_the_range(ctx, m, bits, gs, method, size, scale):
    check_ends(ctx, m, 4200, bits, gs, method, size, scale)
