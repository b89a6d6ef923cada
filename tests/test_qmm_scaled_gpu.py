"""Quantised products of two and more rows (uzu_b200/csrc/qmm_scaled.cu: tcgen05, weights as bf16 planes in tensor memory; qmm_rows.cu: few rows) against
the oracle's matmul, at the sizes where tiles, splits and factor look-ahead can go wrong."""
import numpy as np
import pytest

from oracle import oracle as O
from tests import gpu_ops as G
from tests.util import assert_bf16_close, f32_to_bf16

pytestmark = [pytest.mark.gpu]

METHODS = {"mlx": O.QM_SCALE_BIAS, "zero": O.QM_ZERO_POINT, "symmetric": O.QM_SYMMETRIC}


def weights(rng, n, k, bits, gs, method):
    groups = k // gs
    w = rng.integers(0, 256, (n, k * bits // 8), dtype=np.uint8)
    kw = {"scales": f32_to_bf16(rng.uniform(0.01, 0.3, (n, groups)).astype(np.float32)), "method": METHODS[method], "bits": bits, "group_size": gs}
    if method == "mlx":
        kw["biases"] = f32_to_bf16(rng.uniform(-2, 0, (n, groups)).astype(np.float32))
    elif method == "zero":
        kw["zero_points"] = rng.integers(0, 256, (n, -(-groups // 2) if bits == 4 else groups), dtype=np.uint8)
    return w, kw


def check(ctx, m, n, k, bits, gs, method, seed=0, **extra):
    rng = np.random.default_rng(seed + m + n + k)
    w, kw = weights(rng, n, k, bits, gs, method)
    x = f32_to_bf16(rng.uniform(-0.5, 0.5, (m, k)).astype(np.float32))
    kw.update(extra)
    d = kw.pop("d", None)
    ref = O.matmul(x, w, m=m, n=n, k=k, d_f32=True, d=None if d is None else d.copy(), threads=8, **kw)
    got = G.matmul(ctx, x, w, m=m, n=n, k=k, d_f32=True, d=None if d is None else d.copy(), **kw)
    # sums of k f32 products in another order, the bound of the other tensor-core products: 1e-4 of the output's root mean square, 1e-3 relative
    scale = float(np.sqrt(np.mean(ref.astype(np.float64) ** 2)))
    assert np.isfinite(got).all()
    assert np.all(np.abs(got - ref) <= 1e-3 * np.abs(ref) + 1e-4 * scale), float(np.abs(got - ref).max() / scale)
    assert ctx.lib.uzu_debug_dense_umma_error() == 0


@pytest.mark.parametrize("bits,gs,method", [(4, 64, "zero"), (4, 32, "zero"), (4, 128, "symmetric"), (4, 32, "mlx"), (4, 256, "mlx"), (8, 64, "zero"), (8, 32, "symmetric"), (8, 128, "mlx")])
@pytest.mark.parametrize("m", [2, 17, 40, 129])
def test_formats_and_row_tiles(ctx, m, bits, gs, method):
    """Every format at a row count inside each kind of tile; features that leave the last tile ragged; a split k with a short last share."""
    check(ctx, m, 1700, 1280, bits, gs, method)


@pytest.mark.parametrize("m,n,k", [(2, 16, 64), (16, 128, 64), (33, 33000, 64), (49, 17000, 128), (64, 257, 192), (65, 8, 448), (128, 1000, 320), (193, 384, 576), (256, 130, 1088), (300, 128, 4096), (513, 640, 256)])
def test_edges(ctx, m, n, k):
    """One k block, odd block counts (a code tile that is not full, fewer blocks than the pipeline is deep), rows at both sides of a tile."""
    check(ctx, m, n, k, 4, 64, "zero")
    check(ctx, m, n, k, 8, 32, "zero")


@pytest.fixture
def tile(ctx):
    yield ctx.lib.uzu_debug_set_qmm_tile
    ctx.lib.uzu_debug_set_qmm_tile(0, 0)


@pytest.mark.parametrize("bits,gs,method", [(4, 64, "zero"), (8, 32, "mlx"), (4, 128, "mlx")])
@pytest.mark.parametrize("splits", [1, 2, 4, 8])
def test_every_tile_and_split(ctx, tile, splits, bits, gs, method):
    """Every width of a tile with every number of CTAs that share its k, the last of them with a short share. A width changes no bit, except
    that tiles of up to 64 rows add up chains of two blocks."""
    m, n, k = 150, 200, 61 * 64 if gs < 128 else 30 * 128
    rng = np.random.default_rng(bits + gs)
    w, kw = weights(rng, n, k, bits, gs, method)
    x = f32_to_bf16(rng.uniform(-0.5, 0.5, (m, k)).astype(np.float32))
    outs = []
    for rows in (16, 32, 64, 128, 192, 256):
        assert tile(rows, splits)
        check(ctx, m, n, k, bits, gs, method)
        outs.append(G.matmul(ctx, x, w, m=m, n=n, k=k, d_f32=True, **kw))
    assert all((o == outs[0]).all() for o in outs[:3]) and all((o == outs[3]).all() for o in outs[3:])


@pytest.mark.parametrize("bits,gs,method", [(4, 64, "zero"), (8, 64, "symmetric"), (4, 32, "mlx")])
@pytest.mark.parametrize("m,n,k", [(3, 130, 512), (21, 1700, 1024), (37, 257, 1024), (77, 384, 512), (150, 1000, 320), (300, 128, 512)])
def test_bf16_outputs(ctx, m, n, k, bits, gs, method):
    """The rounded sum stored straight from the accumulators: whole and ragged tiles, rows that are no multiple of 16."""
    rng = np.random.default_rng(m + n)
    w, kw = weights(rng, n, k, bits, gs, method)
    x = f32_to_bf16(rng.uniform(-0.5, 0.5, (m, k)).astype(np.float32))
    assert_bf16_close(G.matmul(ctx, x, w, m=m, n=n, k=k, **kw), O.matmul(x, w, m=m, n=n, k=k, threads=8, **kw), max_ulp=1, min_exact=0.97, what="bf16 rows")


def test_more_tiles_than_the_chip_holds(ctx):
    """CTAs that stay for several tiles, with and without neighbouring row tiles."""
    check(ctx, 20, 128 * 301, 256, 4, 64, "zero")
    check(ctx, 600, 128 * 80, 128, 4, 128, "symmetric")


def test_epilogue(ctx):
    rng = np.random.default_rng(5)
    for m in (3, 150):
        n, k = 192, 512
        d = rng.standard_normal((m, n)).astype(np.float32)
        bias = f32_to_bf16(rng.standard_normal(n).astype(np.float32))
        check(ctx, m, n, k, 4, 64, "zero", d=d, accumulate=True, bias=bias, ab_scale=0.5)
        check(ctx, m, n, k, 8, 64, "symmetric", soft_cap=3.0, bias=bias)
        check(ctx, m, n, k, 4, 64, "symmetric", signed_codes=True)


@pytest.mark.parametrize("bits,gs,method", [(4, 64, "zero"), (4, 128, "zero"), (4, 64, "mlx"), (4, 128, "symmetric"), (8, 64, "zero"), (8, 128, "zero"), (8, 64, "symmetric"), (8, 128, "mlx")])
@pytest.mark.parametrize("m,n,k", [(2, 1700, 2048), (8, 16, 512), (9, 130, 14336), (17, 5000, 1024), (25, 1700, 4096), (32, 4097, 1536), (5, 40, 4096), (8, 28672, 512)])
def test_few_rows(ctx, m, n, k, bits, gs, method):
    """The kernel of 2 to 32 rows (qmm_rows.cu): every width of its fragments, one step of k and several slices of it, fewer tiles than CTAs, a ragged tile."""
    check(ctx, m, n, k, bits, gs, method)


def test_few_rows_epilogue(ctx):
    """Accumulate, bias, scale and signed codes, with and without slices of k."""
    rng = np.random.default_rng(3)
    for n, k in ((16 * 160, 512), (48, 4096)):
        d = rng.uniform(-1, 1, (20, n)).astype(np.float32)
        check(ctx, 20, n, k, 4, 64, "zero", d=d, accumulate=True, bias=f32_to_bf16(rng.uniform(-1, 1, n).astype(np.float32)), ab_scale=0.5)
        check(ctx, 20, n, k, 8, 64, "symmetric", signed_codes=True)


@pytest.mark.parametrize("bits,k", [(4, 512), (4, 1536), (8, 256), (8, 768)])
@pytest.mark.parametrize("n", [1, 33, 4097])
def test_few_rows_zero_points_that_end_inside_a_word(ctx, bits, k, n):
    """Groups of 128 over an odd number of steps: a row's zero points are two bytes modulo four, and so is the array with an odd number of rows."""
    check(ctx, 7, n, k, bits, 128, "zero")
