"""Sampling of rows that are whole 16-byte pieces (uzu_b200/csrc/sampling.cu) at the edges of what a thread keeps of a row: ids are the oracle's."""
import numpy as np
import pytest

from oracle import oracle as O
from tests import gpu_ops as G
from tests.util import f32_to_bf16

pytestmark = [pytest.mark.gpu]


@pytest.mark.parametrize("V", [32768, 65528, 65536, 65544, 262144, 262152])       # too few pieces, one for every thread, a ragged second one, the most that is kept, one piece too many
@pytest.mark.parametrize("kw", [dict(top_k=37), dict(top_p=0.9, temperature=0.7), dict(min_p=0.05, top_k=3000)])
def test_filters(ctx, V, kw):
    """Values on a grid, so that the kept set ends inside a group of equals spread over threads, pieces and CTAs; masked entries among them."""
    rng = np.random.default_rng(V)
    logits = f32_to_bf16((np.round(rng.standard_normal((2, V)) * 8) / 4).astype(np.float32))
    mask = rng.integers(0, 2 ** 32, (2, (V + 31) // 32), dtype=np.uint64).astype(np.uint32) | np.uint32(1)
    seeds = rng.integers(0, 2 ** 63, 2).astype(np.uint64)
    for bitmask in (None, mask):
        assert np.array_equal(O.unified_sampling(logits, seeds=seeds, bitmask=bitmask, **kw), G.unified_sampling(ctx, logits, seeds=seeds, bitmask=bitmask, **kw))


@pytest.mark.parametrize("V", [8, 8184, 8192, 8200, 229376, 229384, 248320, 458752, 458760])       # a piece, the edges of a block, one and two pieces per thread and what is left over
def test_greedy_and_gumbel(ctx, V):
    rng = np.random.default_rng(V)
    logits = f32_to_bf16((np.round(rng.standard_normal((3, V)) * 8) / 4).astype(np.float32))
    logits[1, V // 2] = 0x7FC0                                        # NaN wins over no earlier element
    mask = rng.integers(0, 2 ** 32, (3, (V + 31) // 32), dtype=np.uint64).astype(np.uint32) | np.uint32(2)
    seeds = rng.integers(0, 2 ** 63, 3).astype(np.uint64)
    for kw in (dict(), dict(bitmask=mask), dict(seeds=seeds, temperature=0.7), dict(seeds=seeds, bitmask=mask)):
        assert np.array_equal(O.unified_sampling(logits, **kw), G.unified_sampling(ctx, logits, **kw)), kw
