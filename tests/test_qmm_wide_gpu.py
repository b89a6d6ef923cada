"""Quantised products of many rows with the codes as integers (uzu_b200/csrc/qmm_wide.cu): widths of one half and of two unequal ones, cut-off rows, features and code tiles, every epilogue, several tiles a CTA, and numbers near the ends of the range."""
import numpy as np
import pytest

from oracle import oracle as O
from tests import gpu_ops as G
from tests.test_qmm_integer_codes_gpu import ENDS, check_ends
from tests.test_qmm_scaled_gpu import check, weights
from tests.util import assert_bf16_close, f32_to_bf16
from uzu_b200.binding import UzuError

pytestmark = [pytest.mark.gpu]


@pytest.fixture(params=[16, 80, 128, 144, 256])
def width(ctx, request):
    assert ctx.lib.uzu_debug_set_qmm_tile(request.param, -1)
    yield request.param
    ctx.lib.uzu_debug_set_qmm_tile(0, 0)


@pytest.mark.parametrize("bits,gs,method", [(4, 128, "zero"), (4, 128, "symmetric"), (4, 256, "zero")])
def test_widths(ctx, width, bits, gs, method):
    check(ctx, 300, 200, 1280, bits, gs, method)
    check(ctx, 70, 130, 256 if gs == 256 else 5 * gs, bits, gs, method)


@pytest.mark.parametrize("bits,gs,method", [(4, 128, "zero"), (4, 256, "symmetric")])
@pytest.mark.parametrize("m,n,k", [(65, 9000, 512), (257, 4200, 2816), (1000, 2200, 256), (512, 17000, 256)])
def test_own_plan(ctx, bits, gs, method, m, n, k):
    check(ctx, m, n, k, bits, gs, method)


@pytest.mark.parametrize("size,scale", ENDS)
@pytest.mark.parametrize("bits,gs,method", [(4, 128, "symmetric"), (4, 256, "zero")])
def test_numbers_near_the_ends_of_the_range(ctx, size, scale, bits, gs, method):
    try:
        assert ctx.lib.uzu_debug_set_qmm_tile(80, -1)
        check_ends(ctx, 90, 4200, bits, gs, method, size, scale)
    finally:
        ctx.lib.uzu_debug_set_qmm_tile(0, 0)


def test_epilogue(ctx, width):
    rng = np.random.default_rng(5)
    m, n, k = 150, 192, 512
    d = rng.standard_normal((m, n)).astype(np.float32)
    bias = f32_to_bf16(rng.standard_normal(n).astype(np.float32))
    check(ctx, m, n, k, 4, 128, "zero", d=d, accumulate=True, bias=bias, ab_scale=0.5)
    check(ctx, m, n, k, 4, 128, "symmetric", signed_codes=True)
    w, kw = weights(rng, n, k, 4, 128, "zero")
    x = f32_to_bf16(rng.uniform(-0.5, 0.5, (m, k)).astype(np.float32))
    assert_bf16_close(G.matmul(ctx, x, w, m=m, n=n, k=k, **kw), O.matmul(x, w, m=m, n=n, k=k, threads=8, **kw), max_ulp=1, min_exact=0.97, what="bf16 rows")


@pytest.mark.parametrize("bits,gs,method", [(4, 64, "zero"), (8, 128, "zero"), (4, 128, "mlx")])
def test_what_it_does_not_take(ctx, width, bits, gs, method):
    """(so that no test above runs another kernel unseen)"""
    with pytest.raises(UzuError, match="qmm_wide"):
        check(ctx, 100, 128, 512, bits, gs, method)
