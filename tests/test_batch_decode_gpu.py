"""Multi-sequence batched decode (extension API uzu_engine_batch_*): B independent sequences sharing one pass
over the weights per step, against B independent oracle models (the reference decodes one sequence at a time: N independent reference runs
are the oracle for an N-sequence batch)."""
import os

import numpy as np
import pytest

from oracle.model import OracleModel
from tests.test_engine_gpu import _logit_check
from tests.util import bf16_to_f32
from uzu_b200 import binding as B
from uzu_b200 import synth

pytestmark = [pytest.mark.gpu]


@pytest.mark.parametrize("graph", [False, True])
@pytest.mark.parametrize("kind,nseq", [("llama", 3), ("qwen-hybrid", 2), ("llama-512", 8)])
def test_batched_decode_matches_independent_oracles(ctx, tmp_path, kind, nseq, graph):
    """graph=True: the batched step is captured once into a CUDA graph and replayed with per-sequence positions read from the device."""
    spec = synth.tiny(kind)
    path = synth.write_model(spec, tmp_path / "m", seed=41)
    rng = np.random.default_rng(9)
    prompts = [rng.integers(0, spec.vocab_size, 5 + 7 * b) for b in range(nseq)]        # different lengths -> different positions per row
    refs = [OracleModel(path, max_context=128) for _ in range(nseq)]
    ref_logits = [r.prefill(p) for r, p in zip(refs, prompts)]
    with B.Engine(ctx, path, max_context_length=128, use_cuda_graph=graph) as eng:
        eng.batch_begin(nseq)
        firsts = [eng.batch_prefill(b, prompts[b]) for b in range(nseq)]
        toks = []
        for b in range(nseq):
            l = np.sort(bf16_to_f32(ref_logits[b][0]))[::-1]
            want = int(np.argmax(bf16_to_f32(ref_logits[b][0])))
            if l[0] - l[1] > 0.05 * abs(l[0]):
                assert firsts[b] == want, (b, firsts[b], want)
            toks.append(want)                                                             # teacher forcing with the oracle's tokens
        for step in range(5):
            got = eng.batch_step(toks)
            lg = eng.batch_logits()
            nxt = []
            for b in range(nseq):
                lr = refs[b].forward([toks[b]])
                _logit_check(lg[b:b + 1], lr, f"{kind} seq {b} step {step}")
                want = int(np.argmax(bf16_to_f32(lr[0])))
                l = np.sort(bf16_to_f32(lr[0]))[::-1]
                if l[0] - l[1] > 0.05 * abs(l[0]):
                    assert got[b] == want, (b, step, got[b], want)
                nxt.append(want)
            toks = nxt
        for b in range(nseq):
            assert ctx.lib.uzu_engine_batch_context_length(eng.h, b) == len(prompts[b]) + 5
        assert eng.batch_decode_timed(toks, 4) > 0.0                                     # device-chained steps run


def test_batch_resize_frees_sequences_and_recaptures_the_graph(ctx, tmp_path):
    """batch_begin with a different sequence count: dropped sequences release their state, re-created ones get fresh buffers, and the captured
    batched step (which holds every sequence's buffer addresses) is re-captured -- the logits after 4 -> 2 -> 4 sequences equal those of a
    fresh 4-sequence engine bit for bit."""
    spec = synth.tiny("qwen-hybrid-512")
    path = synth.write_model(spec, tmp_path / "m", seed=43)
    rng = np.random.default_rng(10)
    prompts = [rng.integers(0, spec.vocab_size, 6 + 3 * b) for b in range(4)]

    def run(eng, nseq, steps=3):
        eng.batch_begin(nseq)
        toks = [eng.batch_prefill(b, prompts[b]) for b in range(nseq)]
        out = []
        for _ in range(steps):
            toks = eng.batch_step(toks)
            out.append(eng.batch_logits()[:nseq].copy())
        return out

    with B.Engine(ctx, path, max_context_length=128, use_cuda_graph=True) as eng:
        first = run(eng, 4)
        two = run(eng, 2)
        again = run(eng, 4)
    with B.Engine(ctx, path, max_context_length=128, use_cuda_graph=True) as fresh:
        want = run(fresh, 4)
    for a, b, c in zip(first, again, want):
        assert (a == c).all() and (b == c).all()
    with B.Engine(ctx, path, max_context_length=128, use_cuda_graph=True) as fresh2:
        want2 = run(fresh2, 2)
    for a, c in zip(two, want2):
        assert (a == c).all()


LENGTHS = [1, 70, 900, 3000]       # one cached row, two splits of the keys, a launch's worth of them, as many as there are


@pytest.fixture(scope="module")
def uneven(tmp_path_factory):
    spec = synth.tiny("llama")
    path = synth.write_model(spec, tmp_path_factory.mktemp("uneven") / "m", seed=44)
    rng = np.random.default_rng(11)
    prompts = [rng.integers(0, spec.vocab_size, n) for n in LENGTHS]
    tokens = rng.integers(0, spec.vocab_size, (3, len(LENGTHS)))
    refs = [OracleModel(path, max_context=4096) for _ in LENGTHS]
    for r, p in zip(refs, prompts):
        r.prefill(p)
    return spec, path, prompts, tokens, [[r.forward([t[b]]) for b, r in enumerate(refs)] for t in tokens]


@pytest.mark.parametrize("graph", [False, True])
def test_sequences_of_uneven_lengths(ctx, uneven, graph):
    """Every sequence's keys are cut by its own length: sequences with one split, a few and the most there are share a launch."""
    _, path, prompts, tokens, want = uneven
    with B.Engine(ctx, path, max_context_length=4096, use_cuda_graph=graph) as eng:
        eng.batch_begin(len(prompts))
        for b, p in enumerate(prompts):
            eng.batch_prefill(b, p)
        for step, toks in enumerate(tokens):
            eng.batch_step(toks)
            got = eng.batch_logits()
            for b in range(len(prompts)):
                _logit_check(got[b:b + 1], want[step][b], f"{LENGTHS[b]} rows, step {step}")


def test_a_sequence_does_not_depend_on_its_neighbours_lengths(ctx, uneven):
    """The same bits beside short and long neighbours, eager and from a graph."""
    spec, path, _, tokens, _ = uneven
    rng = np.random.default_rng(12)
    prompt = rng.integers(0, spec.vocab_size, 300)
    results = []
    for graph in (False, True):
        for others in ((3, 5), (1500, 40), (64, 3000)):
            with B.Engine(ctx, path, max_context_length=4096, use_cuda_graph=graph) as eng:
                eng.batch_begin(3)
                for b, p in enumerate([prompt] + [rng.integers(0, spec.vocab_size, n) for n in others]):
                    eng.batch_prefill(b, p)
                for toks in tokens[:, :3]:
                    eng.batch_step([int(tokens[0, 0])] + [int(t) for t in toks[1:]])
                results.append(eng.batch_logits()[0].copy())
    assert all((r == results[0]).all() for r in results)


@pytest.mark.parametrize("graph", [False, True])
def test_a_batch_samples_greedily_whatever_the_engines_own_sequence_does(ctx, tmp_path, graph):
    """The engine's own sequence takes a stochastic method after batch_begin: prompts and steps of the batch still return their largest logit, from steps
    captured before the change, while it lasts and after it."""
    spec = synth.tiny("llama-512")
    path = synth.write_model(spec, tmp_path / "m", seed=41)
    rng = np.random.default_rng(10)
    hot = B.Engine.sampling(seed=7, temperature=50.0)
    prompts = [rng.integers(0, spec.vocab_size, 60) for _ in range(3)]
    largest = lambda logits: [int(t) for t in bf16_to_f32(logits).argmax(-1)]
    with B.Engine(ctx, path, max_context_length=512, use_cuda_graph=graph) as eng:
        eng.batch_begin(3)
        for sampling in (None, hot, B.Engine.sampling()):
            eng.prefill(prompts[0], sampling)
            for b, p in enumerate(prompts):
                assert eng.batch_prefill(b, p) == largest(eng.last_logits())[-1]
            for step in range(40):                  # lengths that share a captured step and lengths that do not
                got = eng.batch_step([1, 2, 3])
                assert got == largest(eng.batch_logits()), (step, sampling)


@pytest.mark.parametrize("graph", [False, True])
def test_more_slots_than_a_batched_step_takes(ctx, tmp_path, graph):
    """Sequence slots lie in the batch's list, and there may be 64 of them: a batched step over more than 16 is refused before anything is written."""
    spec = synth.tiny("llama", layers=1)
    path = synth.write_model(spec, tmp_path / "m", seed=42)
    with B.Engine(ctx, path, max_context_length=64, use_cuda_graph=graph) as eng:
        slots = [eng.slot_acquire() for _ in range(17)]
        eng._batch = 17
        for call in (lambda: eng.batch_step([1] * 17), eng.batch_logits, lambda: eng.batch_decode_timed([1] * 17, 2)):
            with pytest.raises(B.UzuError, match="at most 16"):
                call()
        for s in slots:
            eng.slot_release(s)
        eng.batch_begin(2)
        firsts = [eng.batch_prefill(b, [3, 1, 4]) for b in range(2)]
        got = eng.batch_step(firsts)
        assert firsts[0] == firsts[1] and got[0] == got[1]
