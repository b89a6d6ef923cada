"""A decoded row's attention (decode_attention.cu) at the edges of its tiles of 16 keys, of its ranks of 128 and behind eight ranks, for every channel count and for
heads of a key head that fill a CTA's rows or are shared out: the step's logits against those of the same tokens taken in as a prompt, which other kernels compute."""
import dataclasses

import numpy as np
import pytest

from tests.util import bf16_to_f32
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
