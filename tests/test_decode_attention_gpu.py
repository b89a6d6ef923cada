"""A decoded row's attention (decode_attention.cu) at the edges of its tiles of 16 keys, of its ranks of 128 and behind eight ranks, for every channel count and for
heads of a key head that fill a CTA's rows or are shared out: the step's logits against those of the same tokens taken in as a prompt, which other kernels compute,
and the kernel's own results against sums in 64 bits."""
import ctypes as C
import dataclasses

import numpy as np
import pytest

from tests import gpu_ops as G
from tests.util import bf16_to_f32, f32_to_bf16, off_the_rounding
from uzu_b200 import binding as B
from uzu_b200 import synth

pytestmark = [pytest.mark.gpu]


def _spec(heads, groups, dim, kind):
    spec = synth.tiny(kind)
    rope = dict(spec.rope, head_dim=dim if kind == "llama-512" else dim // 2)
    return dataclasses.replace(spec, num_heads=heads, num_groups=groups, head_dim=dim, rope=rope, layer_kinds=["attn"] * 2)


@pytest.mark.parametrize("kind", ["llama-512", "qwen-hybrid-512"])      # the latter: normed queries and keys, half of the channels rotated, a gate
@pytest.mark.parametrize("heads,groups,dim", [(8, 2, 64), (8, 8, 64), (12, 1, 128), (16, 1, 64), (4, 1, 128), (2, 1, 256), (16, 2, 256)])
def test_steps_against_prompts(ctx, tmp_path, kind, heads, groups, dim):
    path = synth.write_model(_spec(heads, groups, dim, kind), tmp_path / "m", seed=7)
    tokens = np.random.default_rng(heads + dim).integers(0, 2048, 1100)
    with B.Engine(ctx, path, max_context_length=2048, use_cuda_graph=True) as eng, B.Engine(ctx, path, max_context_length=2048, use_cuda_graph=False) as eager:
        eng.set_persistent_decode(False)
        eager.set_persistent_decode(False)
        for n in (1, 15, 16, 127, 128, 129, 255, 1023, 1024, 1057):
            got = []
            for e in (eng, eager):
                e.reset()
                e.prefill(tokens[:n])
                for t in tokens[n:n + 2]:
                    e.step_host(int(t))
                got.append(e.last_logits())
            assert np.array_equal(*got), n
            eng.reset()
            eng.prefill(tokens[:n + 2])
            got, want = bf16_to_f32(got[0]), bf16_to_f32(eng.last_logits())
            assert np.linalg.norm(got - want) <= 0.03 * np.linalg.norm(want), (n, np.linalg.norm(got - want) / np.linalg.norm(want))      # bf16 rows in both


def _row(ctx, qkv, k, v, heads, groups, dim):
    """attention of a decoded row behind the cached ones; its key and value go to the end of k and v"""
    n = len(k)
    out = ctx.upload(np.zeros((heads, dim), np.uint16))
    bufs = [ctx.upload(np.ascontiguousarray(a)) for a in (qkv, k, v)]
    p = B.AttentionPrepareNormArgs()
    p.prepare = B.AttentionPrepareArgs(qkv=bufs[0].ptr, keys=bufs[1].ptr, values=bufs[2].ptr, num_q_heads=heads, num_kv_heads=groups, head_dim=dim, kv_token_offset=n - 1, batch_dim=1,
                                       has_kv=1)
    a = B.AttentionArgs(keys=bufs[1].ptr, values=bufs[2].ptr, out=out.ptr, gqa_factor=heads // groups, sequence_length=n, k_head_stride=dim, k_seq_stride=groups * dim, v_head_stride=dim,
                        v_seq_stride=groups * dim, scale=dim ** -0.5, num_heads=heads, suffix_length=1, head_dim=dim, is_causal=1)
    with ctx.command_buffer("decode-attention") as cmd:
        assert ctx.lib.uzu_debug_decode_attention_encode(cmd.h, C.byref(p), C.byref(a)) == 1
    return out.numpy(np.uint16, (heads, dim)), bufs[1].numpy(np.uint16, k.shape), bufs[2].numpy(np.uint16, v.shape)


@pytest.mark.parametrize("heads,groups,dim,n", [(64, 16, 256, 40), (64, 16, 256, 700), (48, 4, 256, 3000), (128, 32, 128, 700), (128, 16, 128, 2100), (128, 32, 64, 700)])
def test_no_further_off_than_sums_in_f32(ctx, heads, groups, dim, n):
    """Results that are not the correctly rounded ones: no more than of the split-KV kernel, which adds up its products in f32. (Chains of products on the tensor pipe, over
    a head's channels or from tile to tile, had up to twice as many.)"""
    rng, off, count, per = np.random.default_rng(dim + n), [0, 0], 0, heads // groups
    while count < 500000:
        qkv = f32_to_bf16(rng.standard_normal((heads + 2 * groups, dim)).astype(np.float32))
        k, v = (f32_to_bf16(rng.standard_normal((n, groups * dim)).astype(np.float32)) for _ in range(2))
        got, k, v = _row(ctx, qkv, k, v, heads, groups, dim)
        assert np.array_equal(k[-1], qkv[heads:heads + groups].ravel()) and np.array_equal(v[-1], qkv[heads + groups:].ravel())
        q, k64, v64 = (bf16_to_f32(x).astype(np.float64) for x in (qkv[:heads].reshape(groups, per, dim), k.reshape(n, groups, dim), v.reshape(n, groups, dim)))
        s = q @ k64.transpose(1, 2, 0) * dim ** -0.5
        w = np.exp(s - s.max(-1, keepdims=True))
        want = (w @ v64.transpose(1, 0, 2) / w.sum(-1, keepdims=True)).reshape(heads, dim)
        before = G.attention_single_pass(ctx, qkv[:heads], k, v, head_dim=dim, gqa_factor=per, sequence_length=n, k_head_stride=dim, k_seq_stride=groups * dim, v_head_stride=dim,
                                         v_seq_stride=groups * dim, scale=float(dim ** -0.5), num_heads=heads, suffix_length=1)
        count += want.size
        off[0] += off_the_rounding(before, want)
        off[1] += off_the_rounding(got, want)
    assert off[1] <= off[0] + 4 * sum(off) ** 0.5, off      # (four standard deviations of the two counts)


@pytest.mark.parametrize("heads,groups,dim,n", [(8, 2, 64, 700), (12, 2, 128, 40), (4, 1, 128, 2300), (8, 2, 256, 300), (12, 1, 256, 300)])
def test_values_that_are_not_finite(ctx, heads, groups, dim, n):
    """An infinity that a row sees comes out as one, and only in its channel, as sums in f32 give it: among the cached rows and as the new one."""
    rng, per = np.random.default_rng(n), heads // groups
    qkv = f32_to_bf16(rng.standard_normal((heads + 2 * groups, dim)).astype(np.float32))
    k, v = (f32_to_bf16(rng.standard_normal((n, groups, dim)).astype(np.float32)) for _ in range(2))
    clean, _, _ = _row(ctx, qkv, k.reshape(n, -1), v.reshape(n, -1), heads, groups, dim)
    want = bf16_to_f32(clean).copy()
    bad = {3: [np.inf], 5: [-np.inf], 6: [np.inf, -np.inf], dim - 1: [np.nan]}          # of the last key head: a channel's values, each of another key
    for c, values in bad.items():
        for i, x in enumerate(values):
            v[(7 * c + 11 * i) % (n - 1), groups - 1, c] = f32_to_bf16(np.array([x], np.float32))[0]
        want[heads - per:, c] = values[0] if len(values) == 1 else np.nan
    qkv[heads + 2 * groups - 1, 8] = f32_to_bf16(np.array([np.inf], np.float32))[0]
    want[heads - per:, 8] = np.inf
    got = bf16_to_f32(_row(ctx, qkv, k.reshape(n, -1), v.reshape(n, -1), heads, groups, dim)[0])
    odd = ~np.isfinite(want)
    assert np.array_equal(got[odd], want[odd], equal_nan=True)
    assert (np.abs(got[~odd] - want[~odd]) <= 2.0 ** -7 * np.abs(want[~odd]) + 1e-6).all()      # sums in another order: a neighbour at most, 2^-7 off
