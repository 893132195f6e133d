"""The split average pooling's stretches of a window, compiled for the host: whole windows are covered once, for windows
of more pixels than 32-bit products hold as well (a 16384 x 16384 plane has 2^28)."""
import ctypes
import subprocess

import pytest

from flagdnn_b200 import build


@pytest.fixture(scope="module")
def begin(tmp_path_factory):
    d = tmp_path_factory.mktemp("stretch")
    (d / "s.cpp").write_text('#include "pool_stretch.h"\n'
                             'extern "C" long long begin(long long n, int i, int s) { return fdnn::stretch_begin(n, i, s); }\n')
    subprocess.run(["g++", "-O1", "-std=c++17", "-shared", "-fPIC", f"-I{build.CSRC}", "-o", str(d / "s.so"), str(d / "s.cpp")],
                   check=True)
    f = ctypes.CDLL(str(d / "s.so")).begin
    f.restype = ctypes.c_longlong
    f.argtypes = [ctypes.c_longlong, ctypes.c_int, ctypes.c_int]
    return f


@pytest.mark.parametrize("count", [1, 7, 8, 9, 16, 36, 49, 2 ** 28 - 1, 2 ** 28, 2 ** 28 + 3, 2 ** 31 + 5, 2 ** 33, 2 ** 61 + 1])
def test_stretches_cover_a_window_once(begin, count):
    for slices in (1, 8):
        starts = [begin(count, i, slices) for i in range(slices + 1)]
        assert starts == [count * i // slices for i in range(slices + 1)]
