"""The recurrences that take four tokens at a time (uzu_b200/csrc/column_block.cuh) at the edges of their blocks: the shortest passes that go this way and the
longest that do not, passes that end inside a block or inside a CTA's step of four blocks, heads that do not fill the lanes, one and two columns per group of
lanes, CTAs that end between a pair's columns, against the plain recurrences in 64 bits. A sum runs over
at most 128 products and a state element carries the error of every token: 1e-5 and 1e-4 of the largest value, as for the token-by-token forms."""

import numpy as np
import pytest

from tests.test_punilix_gpu import close, general_delta_gpu, general_delta_plain
from tests.test_relidra_gpu import Delta, f32

pytestmark = [pytest.mark.gpu]


@pytest.mark.parametrize("dim,heads", [(36, 1), (64, 3), (68, 2), (128, 2), (36, 32), (64, 32), (100, 16), (128, 12)])       # from 32 heads of 36 on: two columns
@pytest.mark.parametrize("rows", [4, 9, 10, 16, 17, 47])
def test_general_delta_blocks(ctx, dim, heads, rows):
    rng = np.random.default_rng(rows * dim + heads)
    hd = heads * dim
    r, k, v, rate, decay = (rng.standard_normal((rows, hd), dtype=np.float32) for _ in range(5))
    rate_b, decay_b = rng.standard_normal(hd, dtype=np.float32), rng.standard_normal(hd, dtype=np.float32)
    state = rng.standard_normal((heads, dim, dim), dtype=np.float32)
    ref, ref_state = general_delta_plain(r, k, v, rate, decay, rate_b, decay_b, state, heads, dim)
    got, got_state = general_delta_gpu(ctx, r, k, v, rate, decay, rate_b, decay_b, state, heads, dim, True)
    close(got, ref, 1e-5, "output")
    close(got_state, ref_state, 1e-5, "state")


def test_general_delta_value_that_is_not_finite_reaches_no_earlier_token(ctx):
    rng = np.random.default_rng(5)
    rows, heads, dim = 11, 1, 128
    r, k, v, rate, decay = (rng.standard_normal((rows, dim), dtype=np.float32) for _ in range(5))
    zb, state = np.zeros(dim, np.float32), np.zeros((heads, dim, dim), np.float32)
    ref, _ = general_delta_plain(r, k, v, rate, decay, zb, zb, state, heads, dim)
    v[6, 3] = np.inf
    got, _ = general_delta_gpu(ctx, r, k, v, rate, decay, zb, zb, state, heads, dim, True)
    keep = np.ones((rows, dim), bool)
    keep[6:, 3] = False
    close(np.where(keep, got, 0.0), np.where(keep, ref, 0.0), 1e-5, "tokens before it and other columns")
    assert not np.isfinite(got[6:, 3]).any()


@pytest.mark.parametrize("heads,kv_heads,dim,vdim", [(2, 1, 36, 8), (2, 2, 64, 30), (4, 2, 100, 50), (2, 1, 128, 5), (40, 20, 64, 33), (16, 4, 100, 125), (16, 16, 128, 128)])       # from 40 heads on: two columns
@pytest.mark.parametrize("rows", [4, 11, 12, 18, 35, 36, 47])
def test_gated_delta_blocks(ctx, heads, kv_heads, dim, vdim, rows):
    D = Delta(ctx, heads, kv_heads, dim, vdim, 3, seed=rows + dim, start=0.3)
    proj = f32(D.rng, rows, D.stride)
    *_, o, S, _ = D.plain(proj)
    close(D.scan(proj), o.numpy(), 1e-4, "read-out")
    close(D.state(), S.numpy(), 1e-4, "state")
