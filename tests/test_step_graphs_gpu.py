"""Captured decode steps. Steps that go back and forth over the context lengths at which another one is taken (64, 128, ..), a change of the sampling method
and batches of other lengths and numbers of sequences: what is read back is what a fresh engine gives, and steps are captured no more often than they have to."""
import ctypes as C
import dataclasses

import numpy as np
import pytest

from uzu_b200 import binding as B
from uzu_b200 import synth

pytestmark = [pytest.mark.gpu]


@pytest.mark.parametrize("kind", ["llama", "qwen-hybrid"])
def test_restored_contexts_match_fresh_engines(ctx, tmp_path, kind):
    spec = synth.tiny(kind)
    path = synth.write_model(spec, tmp_path / "m", seed=3)
    prompt = np.random.default_rng(4).integers(0, spec.vocab_size, 1100)
    lengths = (62, 126, 254, 510, 1022)

    def steps(eng):
        out = []
        for tok in (1, 2, 3, 4):
            eng.step_host(tok)
            out.append(eng.last_logits().copy())
        return out

    def fresh(n):
        with B.Engine(ctx, path, max_context_length=2048, use_cuda_graph=True) as eng:
            eng.set_persistent_decode(False)
            eng.prefill(prompt[:n])
            return steps(eng)
    ref = {n: fresh(n) for n in lengths}
    with B.Engine(ctx, path, max_context_length=2048, use_cuda_graph=True) as eng:
        eng.set_persistent_decode(False)
        for _ in range(2):
            for n in lengths:
                eng.reset()
                eng.prefill(prompt[:n])
                eng.snapshot()
                for _ in range(2):
                    for got, want in zip(steps(eng), ref[n]):
                        assert np.array_equal(got, want)
                    eng.restore()


@pytest.mark.parametrize("fused", [True, False])
@pytest.mark.parametrize("kind", ["llama-512", "qwen-hybrid-512"])
def test_a_step_does_not_depend_on_the_length_it_was_captured_at(ctx, tmp_path, kind, fused):
    """The same bits from a graph captured at the start of its range, at this length, and without one. 4096 channels of attention in several layers and steps:
    sums in another order round differently in some of them."""
    spec = synth.tiny(kind, layers=4)
    spec = dataclasses.replace(spec, num_heads=32, num_groups=8, head_dim=128, rope=dict(spec.rope, head_dim=128 if kind == "llama-512" else 64))
    path = synth.write_model(spec, tmp_path / "m", seed=3)
    prompt = np.random.default_rng(5).integers(0, spec.vocab_size, 1000)
    results = []
    for graph, first in ((True, 520), (True, None), (False, None)):
        with B.Engine(ctx, path, max_context_length=4096, use_cuda_graph=graph, fused_decode=fused) as eng:
            eng.set_persistent_decode(False)
            if first:
                eng.prefill(prompt[:first])
                eng.step_host(1)
                eng.reset()
            eng.prefill(prompt)
            logits = []
            for tok in range(12):
                eng.step_host(tok)
                logits.append(eng.last_logits().copy())
            results.append(np.stack(logits))
    assert np.array_equal(results[0], results[1]) and np.array_equal(results[1], results[2])


@pytest.mark.parametrize("heads,groups,dim", [(8, 2, 64), (32, 8, 128), (8, 1, 256)])
def test_attention_at_a_device_position_is_cut_by_that_position(ctx, heads, groups, dim):
    """`sequence_length` is only the most there may be: the same bits for every bound. Keys come in pairs whose values cancel, so that an output is mostly
    the rounding of its sums."""
    rng = np.random.default_rng(dim)
    keys = 1000
    bf = lambda x: synth.f32_to_bf16_bits(np.asarray(x, np.float32))
    k, v = np.zeros((1024, groups, dim), np.float32), np.zeros((1024, groups, dim), np.float32)
    order = rng.permutation(keys)
    k[order] = rng.standard_normal((keys // 2, groups, dim)).repeat(2, axis=0)
    v[order] = rng.standard_normal((keys // 2, groups, dim)).repeat(2, axis=0) * np.where(np.arange(keys) % 2, -1.0, 1.0)[:, None, None]
    q, bk, bv = (ctx.upload(bf(x)) for x in (rng.standard_normal((heads, dim)), k, v))
    pos = ctx.upload(np.array([keys - 1], np.uint32))
    results = []
    for bound in (1000, 1024, 4096):
        out = ctx.upload(np.zeros(heads * dim, np.uint16))
        a = B.AttentionArgs(queries=q.ptr, keys=bk.ptr, values=bv.ptr, out=out.ptr, gqa_factor=heads // groups, sequence_length=bound, k_head_stride=dim,
                            k_seq_stride=groups * dim, v_head_stride=dim, v_seq_stride=groups * dim, scale=dim ** -0.5, num_heads=heads, suffix_length=1, head_dim=dim,
                            is_causal=1, dynamic_position=pos.ptr)
        with ctx.command_buffer("attention") as cmd:
            cmd.encode("uzu_attention_single_pass_encode", C.byref(a))
        results.append(out.numpy(np.uint16, (heads * dim,)))
    assert np.array_equal(results[1], results[0]) and np.array_equal(results[2], results[0])


def test_an_engine_keeps_the_steps_it_used_last(ctx, tmp_path):
    """Four of them: going back and forth over three ranges captures each once; five ranges in turn do not fit; a range in use survives others that come and go."""
    spec = synth.tiny("llama")
    path = synth.write_model(spec, tmp_path / "m", seed=3)
    prompt = np.random.default_rng(6).integers(0, spec.vocab_size, 1100)
    with B.Engine(ctx, path, max_context_length=2048, use_cuda_graph=True) as eng:
        eng.set_persistent_decode(False)

        def captures(*lengths):
            before = eng.step_captures
            for n in lengths:
                eng.reset()
                eng.prefill(prompt[:n])
                eng.step_host(1)
            return eng.step_captures - before
        assert captures(40, 100, 200) == 3
        assert captures(200, 40, 100, 40, 200) == 0
        assert captures(400) == 1                             # the fourth
        assert captures(800) == 1 and captures(100) == 1      # the fifth takes the place of the one used longest ago
        assert captures(800, 100, 200, 400) == 0
        assert captures(40, 800, 100, 200, 400) == 5          # five in turn: always the next one is gone


@pytest.mark.parametrize("kind", ["llama-512", "qwen-hybrid-512"])
def test_a_change_of_the_sampling_method(ctx, tmp_path, kind):
    """The method is part of a captured step: ids after greedy, two stochastic methods and greedy again at the same lengths are those of fresh engines, and a
    method that comes back finds its step."""
    spec = synth.tiny(kind)
    path = synth.write_model(spec, tmp_path / "m", seed=3)
    prompt = np.random.default_rng(7).integers(0, spec.vocab_size, 50)
    methods = [B.Engine.sampling(), B.Engine.sampling(seed=5, temperature=3.0, top_k=40), B.Engine.sampling(seed=5, temperature=30.0), B.Engine.sampling(seed=9, temperature=30.0)]

    def ids(eng, method):
        return [eng.prefill(prompt, method)] + [eng.step_host(tok) for tok in range(10)]

    def fresh(method):
        with B.Engine(ctx, path, max_context_length=512, use_cuda_graph=True) as eng:
            eng.set_persistent_decode(False)
            return ids(eng, method)
    ref = [fresh(m) for m in methods]
    assert ref[0] != ref[1] != ref[2] != ref[3]
    with B.Engine(ctx, path, max_context_length=512, use_cuda_graph=True) as eng:
        eng.set_persistent_decode(False)
        before = eng.step_captures
        for i in (0, 1, 2, 0, 3, 1, 0, 2):
            eng.reset()
            assert ids(eng, methods[i]) == ref[i], i
        assert eng.step_captures - before == 3                # a seed is no part of it: methods 2 and 3 share a step


@pytest.mark.parametrize("kind", ["llama-512", "qwen-hybrid-512"])
def test_batches_that_come_back_to_a_length(ctx, tmp_path, kind):
    """Kept batched steps over batch_begin: the same count of sequences keeps them, at other prompt lengths too; another count drops them."""
    spec = synth.tiny(kind)
    path = synth.write_model(spec, tmp_path / "m", seed=3)
    prompt = np.random.default_rng(8).integers(0, spec.vocab_size, 300)

    def batch(eng, lengths):
        eng.batch_begin(len(lengths))
        for b, n in enumerate(lengths):
            eng.batch_prefill(b, prompt[b:b + n])
        out = []
        for tok in range(4):
            out.append((eng.batch_step([tok + b for b in range(len(lengths))]), eng.batch_logits()))
        return out

    def fresh(lengths):
        with B.Engine(ctx, path, max_context_length=512, use_cuda_graph=True) as eng:
            return batch(eng, lengths)
    shapes = [(60, 20, 62), (120, 126, 5), (250, 7, 9)]       # the longest goes over 64, over 128, stays below 256
    ref = {s: fresh(s) for s in shapes + [(60, 20)]}
    with B.Engine(ctx, path, max_context_length=512, use_cuda_graph=True) as eng:
        def captures(s):
            before = eng.step_captures
            for (ids, logits), (want, want_logits) in zip(batch(eng, s), ref[s]):
                assert ids == want and np.array_equal(logits, want_logits), s
            return eng.step_captures - before
        assert [captures(s) for s in shapes] == [2, 1, 0]     # 64 and 128, then 256
        assert [captures(s) for s in shapes] == [0, 0, 0]
        assert captures((60, 20)) == 1                        # below 64 only
        assert captures(shapes[0]) == 2


@pytest.mark.parametrize("mode", [True, False])
@pytest.mark.parametrize("lookahead", [1, 257])
def test_fed_steps_behind_steps_in_flight(ctx, tmp_path, mode, lookahead):
    """A fed step after steps that nobody waited for (their tokens land in the ring that it reads): alone, and behind a reset that counts from zero again."""
    spec = synth.tiny("llama", layers=1)
    path = synth.write_model(spec, tmp_path / "m", seed=11)
    prompt = np.arange(9) * 5 % spec.vocab_size
    with B.Engine(ctx, path, max_context_length=1024, use_cuda_graph=mode) as eng:
        eng.prefill(prompt)
        eng.decode_device(lookahead)
        ctx.synchronize()
        want = eng.step_host(3)
        eng.reset()
        again = eng.step_host(7)
        eng.prefill(prompt)
        eng.reset()
        eng.prefill(prompt)
        eng.decode_device(lookahead)
        assert eng.step_host(3) == want
        eng.decode_device(lookahead - 1)
        eng.reset()
        assert eng.step_host(7) == again


@pytest.mark.parametrize("kind", ["llama-512", "qwen-hybrid-512"])
def test_chained_steps_without_a_graph(ctx, tmp_path, kind):
    """Steps that follow one another on the device alone, launch by launch as in captured ones: a step's first kernel stands behind the whole step before it. The products of
    these models have fewer tiles than the chip has room for."""
    spec = synth.tiny(kind)
    path = synth.write_model(spec, tmp_path / "m", seed=5)
    prompt = np.random.default_rng(6).integers(0, spec.vocab_size, 60)
    logits = []
    for graph in (True, False):
        with B.Engine(ctx, path, max_context_length=1024, use_cuda_graph=graph) as eng:
            eng.set_persistent_decode(False)
            eng.prefill(prompt)
            eng.decode_device(300)
            logits.append(eng.last_logits().copy())
    assert np.array_equal(*logits)


def test_engines_of_two_threads_on_one_core(tmp_path):
    """A fed step watches for its token in host memory; another engine's thread on the same core comes to its turn all the same."""
    import os
    import threading
    spec = synth.tiny("llama", layers=1)
    path = synth.write_model(spec, tmp_path / "m", seed=12)
    out = {}

    def run(name, core=None):
        if core is not None:
            os.sched_setaffinity(0, {core})      # (of this thread)
        with B.Context(0) as own, B.Engine(own, path, max_context_length=1024) as eng:
            eng.set_persistent_decode(False)
            token, out[name] = eng.prefill(np.arange(5)), []
            for _ in range(200):
                token = eng.step_host(token)
                out[name].append(token)

    core = min(os.sched_getaffinity(0))
    for names, where in ((["alone"], None), (["a", "b"], core)):
        threads = [threading.Thread(target=run, args=(n, where)) for n in names]
        for t in threads:
            t.start()
        for t in threads:
            t.join(60)
    assert len(out["alone"]) == 200 and out["a"] == out["b"] == out["alone"]
