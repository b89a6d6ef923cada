"""The zero-point fetch of the few-row quantised product (uzu_b200/csrc/qmm_rows_index.h), compiled for the host: every copy stays inside the array
and brings the step's zero points, for strides that are no multiple of the four bytes it copies."""
import ctypes
import subprocess
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parents[1] / "uzu_b200" / "csrc"


@pytest.fixture(scope="module")
def fetch(tmp_path_factory):
    out = tmp_path_factory.mktemp("qr") / "libqr.so"
    source = f'#include "{CSRC / "qmm_rows_index.h"}"\nextern "C" void fetch(uint32_t* r, const uint32_t* a) {{ auto f = uzu::qr_zero_fetch(a[0], a[1], a[2], a[3], a[4]); r[0] = f.offset; r[1] = f.bytes; r[2] = f.shift; }}'
    subprocess.run(["g++", "-std=c++17", "-shared", "-fPIC", "-x", "c++", "-", "-o", str(out)], input=source.encode(), check=True)
    lib = ctypes.CDLL(str(out))

    def call(*args):
        r = (ctypes.c_uint32 * 3)()
        lib.fetch(r, (ctypes.c_uint32 * 5)(*args))
        return tuple(r)
    return call


@pytest.mark.parametrize("bits,group", [(4, 64), (4, 128), (8, 64), (8, 128)])
@pytest.mark.parametrize("steps", [1, 2, 3, 5])
@pytest.mark.parametrize("n", [1, 2, 17, 33, 4097])
def test_copies_stay_inside_the_zero_points(fetch, bits, group, steps, n):
    k = steps * (512 if bits == 4 else 256)
    groups = k // group
    stride = -(-groups // 2) if bits == 4 else groups
    step_bytes = stride // steps
    for row in {0, 1, n // 2, n - 1} & set(range(n)):
        for step in range(steps):
            offset, size, shift = fetch(row, step, n, stride, step_bytes)
            at = row * stride + step * step_bytes
            assert offset % 4 == 0 and 0 < size <= 4 and offset + size <= n * stride
            assert offset + shift // 8 == at and shift // 8 + step_bytes <= size
