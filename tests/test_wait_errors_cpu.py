"""What the host reports when a barrier wait inside a kernel ran out (uzu_b200/csrc/wait_errors.h, compiled for the host): the word is set by the test."""
import ctypes
import subprocess
from pathlib import Path

import pytest

HEADER = Path(__file__).resolve().parents[1] / "uzu_b200" / "csrc" / "wait_errors.h"
SOURCE = f'''#include "{HEADER}"
static unsigned int word;
static uzu::WaitErrors e;
static uint64_t seen[2];
extern "C" {{
void begin() {{ word = 0; e.word = &word; seen[0] = seen[1] = e.found(); }}
void ran_out(unsigned c) {{ word = c; }}
uint64_t start() {{ return e.start(); }}
unsigned finished(uint64_t n) {{ return e.finished(n); }}
unsigned since(int who) {{ return e.since(seen[who]); }}
}}'''


@pytest.fixture(scope="module")
def errors(tmp_path_factory):
    out = tmp_path_factory.mktemp("we") / "libwe.so"
    subprocess.run(["g++", "-std=c++17", "-shared", "-fPIC", "-pthread", "-x", "c++", "-", "-o", str(out)], input=SOURCE.encode(), check=True)
    lib = ctypes.CDLL(str(out))
    lib.start.restype = ctypes.c_uint64
    lib.finished.argtypes = [ctypes.c_uint64]
    return lib


def test_every_buffer_that_had_started_reports_it_and_later_ones_do_not(errors):
    errors.begin()
    a, b = errors.start(), errors.start()
    assert errors.finished(a) == 0
    errors.ran_out(0x106)
    assert errors.finished(a) == 0x106        # the word does not say whose kernel it was
    assert errors.finished(b) == 0x106        # though the first look took the word
    c = errors.start()
    assert errors.finished(c) == 0


def test_every_watcher_reports_it_once(errors):
    errors.begin()
    errors.ran_out(3)
    assert [errors.since(0), errors.since(1)] == [3, 3]
    assert [errors.since(0), errors.since(1)] == [0, 0]
    n = errors.start()
    errors.ran_out(5)
    assert errors.finished(n) == 5
    assert errors.since(0) == 5 and errors.since(0) == 0
