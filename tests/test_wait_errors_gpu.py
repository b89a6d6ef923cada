"""A barrier wait that ran out inside a tensor-memory product is an error of the call that waits for it. No kernel is made to fail: the test stores the
word that such a kernel stores."""
import pytest

from uzu_b200 import binding as B
from uzu_b200 import synth

pytestmark = [pytest.mark.gpu]


@pytest.fixture
def ran_out(ctx):
    yield lambda: ctx.lib.uzu_debug_set_wait_error(ctx.h, 0x106)
    ctx.lib.uzu_debug_set_wait_error(ctx.h, 0)


def test_command_buffer_fails(ctx, ran_out):
    with pytest.raises(B.UzuError, match="0x106"):
        with ctx.command_buffer("fails"):
            ran_out()
    assert ctx.lib.uzu_debug_dense_umma_error() == 0x106
    with ctx.command_buffer("works"):
        pass


def test_context_fails(ctx, ran_out):
    ran_out()
    assert ctx.lib.uzu_context_synchronize(ctx.h) != 0
    assert ctx.lib.uzu_context_synchronize(ctx.h) == 0


@pytest.mark.parametrize("graph", [False, True])
def test_engine_calls_fail_once(ctx, ran_out, tmp_path, graph):
    path = synth.write_model(synth.tiny("llama"), tmp_path / "m", seed=3)
    with B.Engine(ctx, path, max_context_length=128, use_cuda_graph=graph) as eng:
        ran_out()
        with pytest.raises(B.UzuError, match="0x106"):
            eng.prefill([1, 2, 3])
        eng.prefill([1, 2, 3])
        ran_out()
        with pytest.raises(B.UzuError, match="0x106"):
            eng.step_host(4)
        eng.step_host(4)
        eng.batch_begin(2)
        for i in range(2):
            eng.batch_prefill(i, [1, 2, 3])
        ran_out()
        with pytest.raises(B.UzuError, match="0x106"):
            eng.batch_step([4, 5])
        eng.batch_step([4, 5])
