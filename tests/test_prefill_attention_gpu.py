"""Parity of the tensor-core prefill attention (uzu_b200/csrc/attention_prefill.cu) against the CPU oracle's
AttentionSinglePass restatement (backends/cpu/kernel/attention/attention_single_pass.rs:49-126) and the independent float64 softmax of
tests/unit/encodable_block/attention_test.rs:26-124, on the reference tests' closed-form inputs (attention_single_pass_test.rs:33-78).

UZU_PREFILL_ATTN=0 takes the split-KV kernel for every pass."""
import os

import numpy as np
import pytest

from oracle import oracle as O
from tests import gpu_ops as G
from tests.test_oracle_pins import attention_inputs, softmax_reference
from tests.util import assert_bf16_close, bf16_to_f32, f32_to_bf16

pytestmark = [pytest.mark.gpu]


@pytest.fixture
def prefill_attn(ctx):
    ctx.lib.uzu_debug_set_prefill_attention(1)
    yield ctx
    ctx.lib.uzu_debug_set_prefill_attention(-1)


# (heads, kv heads, sequence, suffix, head_dim, causal)
CASES = [(4, 4, 64, 64, 64, True), (8, 2, 128, 128, 128, True), (8, 1, 200, 37, 128, True), (4, 2, 96, 16, 64, False),
         (8, 2, 300, 100, 64, True), (32, 8, 512, 256, 128, True)]


@pytest.mark.parametrize("H,Hkv,seq,suffix,D,causal", CASES)
def test_prefill_attention_head_major_inputs(prefill_attn, H, Hkv, seq, suffix, D, causal):
    ctx = prefill_attn
    q, k, v = attention_inputs(H, Hkv, seq, suffix, D)        # K / V laid out [kv_head, seq, D] like the reference's kernel tests
    kw = dict(head_dim=D, gqa_factor=H // Hkv, sequence_length=seq, k_head_stride=seq * D, k_seq_stride=D, v_head_stride=seq * D,
              v_seq_stride=D, scale=float(np.float32(1.0) / np.sqrt(np.float32(D))), num_heads=H, suffix_length=suffix, is_causal=causal)
    ref = O.attention_single_pass(q, k, v, **kw)
    got = G.attention_single_pass(ctx, q, k, v, **kw)
    assert_bf16_close(got, ref, max_ulp=1, min_exact=0.95, what="prefill attention vs oracle")
    ind = softmax_reference(q, k, v, H, Hkv, seq, suffix, D, causal)
    assert np.abs(bf16_to_f32(got).astype(np.float64) - ind).max() < 4e-3


def test_prefill_attention_token_major_cache_matches_decode_kernel(prefill_attn):
    """The engine's layout (token-major cache, head stride = D) with a prefix: the tensor-core path and the split-KV decode kernel
    (parity-tested in test_kernels_gpu.py) agree to bf16 rounding on random inputs."""
    ctx = prefill_attn
    rng = np.random.default_rng(31)
    H, Hkv, D, prefix, suffix = 8, 2, 128, 77, 45
    q = f32_to_bf16(rng.standard_normal((H, suffix, D)).astype(np.float32))
    k = f32_to_bf16(rng.standard_normal((prefix + suffix, Hkv * D)).astype(np.float32))
    v = f32_to_bf16(rng.standard_normal((prefix + suffix, Hkv * D)).astype(np.float32))
    kw = dict(head_dim=D, gqa_factor=H // Hkv, sequence_length=prefix + suffix, k_head_stride=D, k_seq_stride=Hkv * D, v_head_stride=D,
              v_seq_stride=Hkv * D, scale=float(1.0 / np.sqrt(D)), num_heads=H, suffix_length=suffix, is_causal=True)
    got = G.attention_single_pass(ctx, q, k, v, **kw)
    ctx.lib.uzu_debug_set_prefill_attention(0)
    base = G.attention_single_pass(ctx, q, k, v, **kw)
    ctx.lib.uzu_debug_set_prefill_attention(1)
    assert_bf16_close(got, base, max_ulp=1, min_exact=0.9, what="tensor-core vs split-KV kernel")
    assert_bf16_close(got, O.attention_single_pass(q, k, v, **kw), max_ulp=1, min_exact=0.95, what="vs oracle")


@pytest.mark.parametrize("H,Hkv,prefix,suffix,D", [(8, 2, 0, 64, 256), (8, 2, 700, 33, 256), (3, 1, 130, 21, 64), (12, 2, 65, 9, 128), (32, 8, 1500, 16, 128), (4, 4, 63, 8, 256), (2, 1, 0, 31, 64), (12, 2, 65, 5, 128), (4, 4, 63, 4, 256)])
@pytest.mark.parametrize("trie", [False, True])
def test_rows_of_grouped_heads(ctx, H, Hkv, prefix, suffix, D, trie):
    """Rows of (token, head) pairs: tiles that end inside a token's heads, head counts that do not divide a tile, 256 channels, few rows over
    many keys (a cluster shares them, some of its CTAs without a tile), and a trie's masks; the cache behind the last key is NaN."""
    rng = np.random.default_rng(H + prefix + suffix)
    n, G_ = prefix + suffix, H // Hkv
    if trie and suffix > 16:
        suffix, n = 16, prefix + 16
    q = f32_to_bf16(rng.standard_normal((H, suffix, D)).astype(np.float32))
    k, v = (f32_to_bf16(rng.standard_normal((n + 64, Hkv * D)).astype(np.float32)) for _ in range(2))
    k[n:], v[n:] = 0x7FC0, 0x7FC0
    kw = dict(head_dim=D, gqa_factor=G_, sequence_length=n, k_head_stride=D, k_seq_stride=Hkv * D, v_head_stride=D, v_seq_stride=Hkv * D,
              scale=float(D ** -0.5), num_heads=H, suffix_length=suffix, is_causal=True)
    if trie:
        heights = [0]
        for _ in range(suffix - 1):
            heights.append(int(rng.integers(1, heights[-1] + 2)))
        ends = [max(j for j in range(i, suffix) if all(heights[x] > heights[i] for x in range(i + 1, j + 1))) for i in range(suffix)]
        kw["trie"] = np.array([[i, ends[i], heights[i]] for i in range(suffix)], dtype=np.uint32)
    ref = O.attention_single_pass(q, k, v, **kw)
    got = G.attention_single_pass(ctx, q, k, v, **kw)
    assert_bf16_close(got, ref, max_ulp=1, min_exact=0.95, what="grouped rows vs oracle")


@pytest.mark.parametrize("H,Hkv,prefix,suffix,D", [(8, 2, 0, 64, 256), (8, 2, 700, 33, 256), (3, 1, 130, 21, 64), (12, 2, 65, 9, 128), (12, 2, 65, 5, 128), (4, 4, 63, 8, 256), (2, 1, 0, 31, 64)])
@pytest.mark.parametrize("trie", [False, True])
def test_rows_of_grouped_heads_on_the_tensor_pipe(prefill_attn, H, Hkv, prefix, suffix, D, trie):
    """The same where the rule would take the split-KV kernel."""
    test_rows_of_grouped_heads(prefill_attn, H, Hkv, prefix, suffix, D, trie)


@pytest.mark.parametrize("bad", [np.nan, np.inf])
@pytest.mark.parametrize("H,Hkv,prefix,suffix,D,node", [(8, 2, 5, 15, 128, 14), (8, 2, 0, 70, 256, 3), (4, 4, 63, 8, 64, 5), (8, 2, 700, 9, 256, 4)])
@pytest.mark.parametrize("trie", [False, True])
def test_rows_that_a_token_does_not_see(prefill_attn, H, Hkv, prefix, suffix, D, node, trie, bad):
    """A key or value that is not finite reaches the tokens that see it and no other: not those before it, not another branch of a trie."""
    ctx = prefill_attn
    rng = np.random.default_rng(H + prefix + suffix)
    if trie:
        suffix, node = 16, min(node, 7)
    n = prefix + suffix
    q = f32_to_bf16(rng.standard_normal((H, suffix, D)).astype(np.float32))
    k, v = (rng.standard_normal((n, Hkv * D)).astype(np.float32) for _ in range(2))
    kw = dict(head_dim=D, gqa_factor=H // Hkv, sequence_length=n, k_head_stride=D, k_seq_stride=Hkv * D, v_head_stride=D, v_seq_stride=Hkv * D,
              scale=float(D ** -0.5), num_heads=H, suffix_length=suffix, is_causal=True)
    sees = np.arange(suffix) >= node
    if trie:                                     # a root, and chains of three nodes each below it
        heights = [0] + [1 + i % 3 for i in range(suffix - 1)]
        ends = [max(j for j in range(i, suffix) if all(heights[x] > heights[i] for x in range(i + 1, j + 1))) for i in range(suffix)]
        kw["trie"] = np.array([[i, ends[i], heights[i]] for i in range(suffix)], dtype=np.uint32)
        sees = (np.arange(suffix) >= node) & (np.arange(suffix) <= ends[node])
    finite = G.attention_single_pass(ctx, q, f32_to_bf16(k), f32_to_bf16(v), **kw)
    k[prefix + node, ::7] = bad
    v[prefix + node] = bad
    got = G.attention_single_pass(ctx, q, f32_to_bf16(k), f32_to_bf16(v), **kw)
    assert_bf16_close(got[~sees], finite[~sees], max_ulp=1, min_exact=0.9, what="tokens that do not see the row")
    assert not np.isfinite(bf16_to_f32(got[sees])).all(axis=(1, 2)).any()
