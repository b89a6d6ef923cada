"""Prompt attention on tcgen05 (attention_umma.cu) wherever it can run: the cases of the mma.sync kernel, and against 64-bit sums the edges of its own tiles (128 rows of
(token, head) pairs, 64 keys), maxima that grow from tile to tile, and rows without a mask."""
import numpy as np
import pytest

from tests import gpu_ops as G
from tests import test_prefill_attention_gpu as P
from tests.util import bf16_to_f32, f32_to_bf16, off_the_rounding

pytestmark = [pytest.mark.gpu]


@pytest.fixture
def umma(ctx):
    ctx.lib.uzu_debug_set_prefill_attention(2)
    yield ctx
    ctx.lib.uzu_debug_set_prefill_attention(-1)


@pytest.mark.parametrize("H,Hkv,prefix,suffix,D", [(12, 2, 65, 9, 128), (32, 8, 1500, 16, 128), (3, 1, 130, 21, 64), (2, 1, 0, 31, 64), (8, 2, 0, 64, 256), (8, 2, 700, 33, 256), (4, 4, 63, 8, 256)])
@pytest.mark.parametrize("trie", [False, True])
def test_grouped_heads(umma, H, Hkv, prefix, suffix, D, trie):
    P.test_rows_of_grouped_heads(umma, H, Hkv, prefix, suffix, D, trie)


@pytest.mark.parametrize("bad", [np.nan, np.inf])
@pytest.mark.parametrize("H,Hkv,prefix,suffix,D,node", [(8, 2, 5, 15, 128, 14), (8, 2, 0, 70, 256, 3), (4, 4, 63, 8, 64, 5), (8, 2, 700, 9, 256, 4)])
@pytest.mark.parametrize("trie", [False, True])
def test_rows_that_a_token_does_not_see(umma, H, Hkv, prefix, suffix, D, node, trie, bad):
    P.test_rows_that_a_token_does_not_see(umma, H, Hkv, prefix, suffix, D, node, trie, bad)


def _reference(q, k, v, H, Hkv, prefix, suffix, D, causal, scale):
    q, k, v = (bf16_to_f32(x).astype(np.float64) for x in (q, k, v))
    k, v = k.reshape(-1, Hkv, D), v.reshape(-1, Hkv, D)
    out = np.empty((suffix, H, D))
    for h in range(H):
        s = q[h] @ k[:, h // (H // Hkv)].T * scale
        if causal:
            s[np.arange(prefix + suffix)[None] > prefix + np.arange(suffix)[:, None]] = -np.inf
        p = np.exp(s - s.max(1, keepdims=True))
        out[:, h] = p @ v[:, h // (H // Hkv)] / p.sum(1, keepdims=True)
    return out


@pytest.mark.parametrize("H,Hkv,prefix,suffix,D", [(32, 8, 0, 32, 128), (32, 8, 31, 33, 128), (32, 8, 512, 640, 128), (1, 1, 4000, 128, 128), (16, 4, 300, 129, 64), (3, 1, 1000, 300, 64), (8, 2, 1, 511, 256),
                                                   (8, 2, 1024, 1024, 256)])
@pytest.mark.parametrize("causal,grows", [(True, False), (True, True), (False, False)])
def test_against_64_bits(umma, H, Hkv, prefix, suffix, D, causal, grows):
    rng = np.random.default_rng(prefix + suffix + D)
    n = prefix + suffix
    q = rng.standard_normal((H, suffix, D)).astype(np.float32)
    k, v = (rng.standard_normal((n, Hkv * D)).astype(np.float32) for _ in range(2))
    if grows:                                    # scores of a later key are larger, by far more than a tile's maximum may move without a new one
        k *= (1 + 12 * np.arange(n, dtype=np.float32) / n)[:, None]
    q, k, v = f32_to_bf16(q), f32_to_bf16(k), f32_to_bf16(v)
    scale = D ** -0.5
    got = G.attention_single_pass(umma, q, k, v, head_dim=D, gqa_factor=H // Hkv, sequence_length=n, k_head_stride=D, k_seq_stride=Hkv * D, v_head_stride=D, v_seq_stride=Hkv * D,
                                  scale=float(scale), num_heads=H, suffix_length=suffix, is_causal=causal)
    want = _reference(q, k, v, H, Hkv, prefix, suffix, D, causal, scale)
    got = bf16_to_f32(got).astype(np.float64).reshape(want.shape)
    # one rounding to bf16, 2^-9 of a result on average and 2^-8 at most; weights of 16 bits and scores in f32 (2^-22 of up to 60 in the exponent) add 2^-16 of the values' size, about 5
    assert (np.abs(got - want) <= 2.0 ** -8 * np.abs(want) + 5 * 2.0 ** -14).all(), np.abs(got - want).max()


@pytest.mark.parametrize("H,Hkv,prefix,suffix,D,before", [(8, 2, 1500, 512, 256, 0), (8, 2, 64, 64, 256, 0), (32, 8, 1100, 256, 128, 1), (32, 8, 600, 512, 64, 1)])
def test_no_further_off_than_the_kernel_before(ctx, H, Hkv, prefix, suffix, D, before):
    """Results that are not the correctly rounded ones: with three planes no more than of the split-KV kernel, whose weights and sums are f32 (0), with two no more than of
    the mma.sync kernel, which has as many (1). (Sums of all keys in tensor memory, which cuts off what it adds, had half as many again and more.)"""
    rng = np.random.default_rng(D + suffix)
    n, off, count = prefix + suffix, [0, 0], 0
    while count < 1 << 20:
        q, k, v = (f32_to_bf16(rng.standard_normal(s).astype(np.float32)) for s in ((H, suffix, D), (n, Hkv * D), (n, Hkv * D)))
        want = _reference(q, k, v, H, Hkv, prefix, suffix, D, True, D ** -0.5)
        count += want.size
        for i, mode in enumerate((before, 2)):
            ctx.lib.uzu_debug_set_prefill_attention(mode)
            try:
                got = G.attention_single_pass(ctx, q, k, v, head_dim=D, gqa_factor=H // Hkv, sequence_length=n, k_head_stride=D, k_seq_stride=Hkv * D, v_head_stride=D,
                                              v_seq_stride=Hkv * D, scale=float(D ** -0.5), num_heads=H, suffix_length=suffix)
            finally:
                ctx.lib.uzu_debug_set_prefill_attention(-1)
            off[i] += off_the_rounding(got, want)
    assert off[1] <= off[0] + 4 * sum(off) ** 0.5, off      # (four standard deviations of the two counts)


@pytest.mark.parametrize("H,Hkv,prefix,suffix,D", [(8, 2, 130, 70, 256), (32, 8, 200, 40, 128), (8, 2, 100, 15, 128), (3, 1, 70, 33, 64)])
def test_values_that_are_not_finite(umma, H, Hkv, prefix, suffix, D):
    """An infinity that a row sees comes out as one, in its channel, and rows that do not see it have none of it."""
    rng, n, c = np.random.default_rng(prefix), prefix + suffix, 9
    q, k, v = (f32_to_bf16(rng.standard_normal(s).astype(np.float32)) for s in ((H, suffix, D), (n, Hkv, D), (n, Hkv, D)))
    kw = dict(head_dim=D, gqa_factor=H // Hkv, sequence_length=n, k_head_stride=D, k_seq_stride=Hkv * D, v_head_stride=D, v_seq_stride=Hkv * D, scale=float(D ** -0.5), num_heads=H,
              suffix_length=suffix)
    want = bf16_to_f32(G.attention_single_pass(umma, q, k, v, **kw)).copy()
    v[5, 0, c] = f32_to_bf16(np.array([-np.inf], np.float32))[0]
    v[prefix + 7, Hkv - 1, c + 1] = f32_to_bf16(np.array([np.inf], np.float32))[0]
    per = H // Hkv
    want[:, :per, c] = -np.inf
    want[7:, H - per:, c + 1] = np.inf
    got = bf16_to_f32(G.attention_single_pass(umma, q, k, v, **kw))
    odd = ~np.isfinite(want)
    assert np.array_equal(got[odd], want[odd])
    assert (np.abs(got[~odd] - want[~odd]) <= 2.0 ** -7 * np.abs(want[~odd]) + 1e-5).all()      # sums in another order, two planes of a weight: a neighbour at most, 2^-7 off
