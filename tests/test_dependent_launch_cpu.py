"""Kernels started through `launch()` may run under programmatic dependent launch, beside their predecessor: each has to wait for it (pdl_wait)
before it touches memory. Read from the sources: no GPU can show a missing wait reliably."""
import re
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parents[1] / "uzu_b200" / "csrc"
COOPERATIVE = {"decode_mega_kernel"}      # a cooperative launch: stream-ordered, never a dependent one
KERNEL = re.compile(r"__global__\s+void\s+(?:__cluster_dims__\([^)]*\)\s*)?(?:__launch_bounds__\([^{;]*?\)\s*)?(\w+)\s*\(")


def _body(text, at):
    """the braces that open behind `at`"""
    start = text.index("{", text.index(")", at))
    depth = 0
    for i in range(start, len(text)):
        depth += {"{": 1, "}": -1}.get(text[i], 0)
        if depth == 0:
            return text[start:i + 1]
    raise AssertionError("unbalanced braces")


def _kernels():
    for path in sorted(CSRC.glob("*.cu")):
        text = re.sub(r"//[^\n]*", "", path.read_text())
        for m in KERNEL.finditer(text):
            # the stream-ordered form <<<..>>> waits for the kernels before it by itself
            ordered = re.search(rf"\b{m.group(1)}\s*(<[^;(]*>)?\s*<<<", text)
            yield pytest.param(_body(text, m.end()), bool(ordered) or m.group(1) in COOPERATIVE, id=f"{path.name}-{m.group(1)}")


@pytest.mark.parametrize("body,ordered", list(_kernels()))
def test_kernel_waits_for_its_predecessor(body, ordered):
    assert ordered or "pdl_wait();" in body or "griddepcontrol.wait" in body


def test_copies_and_fills_are_ordered_with_the_contexts_stream():
    """The stream of a context does not wait for the legacy stream. A fill or a copy on the device that goes to the latter returns before it is done, so that a kernel
    launched next may not see it."""
    for path in sorted(CSRC.iterdir()):
        text = re.sub(r"//[^\n]*", "", path.read_text())
        assert not re.search(r"\bcudaMemset\s*\(", text), path.name
        assert not re.search(r"\bcudaMemcpy\s*\([^;]*cudaMemcpyDeviceToDevice", text), path.name


def test_the_first_launch_of_a_buffer_waits_for_the_buffer_before():
    """Kernels read ahead of their wait what earlier steps left behind (a decoded row's position, cached rows, recurrent states), and a dependent launch orders nothing
    before its wait: every launch asks the buffer whether it may be one, and the first one may not."""
    struct = re.search(r"struct uzu_command_buffer \{.*?\n\};", (CSRC / "common.cuh").read_text(), re.S).group(0)
    assert re.search(r"bool dependent\(\) const \{ return use_pdl && launches > 0; \}", struct)
    for path in sorted([*CSRC.glob("*.cu"), *CSRC.glob("*.cuh"), *CSRC.glob("*.inl")]):
        text = re.sub(r"//[^\n]*", "", path.read_text())
        for m in re.finditer(r"= cudaLaunchAttributeProgrammaticStreamSerialization", text):
            guard = text.rfind("if (", 0, m.start())
            assert text[guard:].startswith("if (cmd->dependent())") and "}" not in text[guard:m.start()], path.name


@pytest.mark.parametrize("body", [pytest.param(p.values[0], id=p.id) for p in _kernels() if "tcgen05.alloc" in p.values[0]])
def test_tensor_memory_is_taken_before_dependents_may_start(body):
    """A dependent's CTA beside this one could take the tensor memory that this one still waits for, and wait itself for this kernel's end. One thread's call lets
    dependents start: it stands behind the barrier that every warp passes once the memory is there."""
    if "pdl_launch_dependents" in body:
        taken = body.index("tcgen05.alloc")
        assert body.index("__syncthreads", taken) < body.index("pdl_launch_dependents") < body.index("tcgen05.dealloc")


def test_scores_are_not_written_over_weights_that_products_still_read():
    """attention_umma.cu: scores that go where weights of an earlier tile were wait for that tile's products, or go elsewhere. (Only products of the same shape into the
    same sum are in order by themselves.)"""
    text = re.sub(r"//[^\n]*", "", (CSRC / "attention_umma.cu").read_text())
    issue = text[text.index("if (i + 1 < tiles)"):text.index("au_commit(o_done)")]
    over = "tmem + s * 64u + pl * 32u" in issue                        # weights in the columns of scores
    assert not over or issue.index("au_wait(o_done") < issue.index("scores(i + 1)")


@pytest.mark.parametrize("body", [pytest.param(p.values[0], id=p.id) for p in _kernels() if "tcgen05.alloc" in p.values[0]])
def test_products_in_flight_are_waited_for_before_tensor_memory_is_given_back(body):
    """Also where a wait ran out: the role that issues products then commits what it has issued and waits, with a limit, for that."""
    end = body.index("tcgen05.dealloc")
    assert re.search(r"(_commit\(last_products\);\s*\}?\s*__syncwarp\(\);\s*\w+_settle\(last_products, 0\)|\(accum_bar\)[^;]*;\s*__syncwarp\(\);\s*if \(!ok\)\s*for \([^)]*try_wait\(accum_bar, 0\))", body[:end])
