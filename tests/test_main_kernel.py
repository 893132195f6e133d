"""fdnn_conv2d_main_kernel: which kernel a problem runs on, where the plan's tiles leave it open."""
import ctypes

import pytest

from flagdnn_b200 import _native as nat
from test_abi import _desc

DIRECT, IGEMM, PAIR, ROWS = range(4)


def kernel_of(lib, d, w=None):
    k = nat.ConvKernel()
    assert lib.fdnn_conv2d_main_kernel(ctypes.byref(d), None, w, None, ctypes.byref(k)) == nat.FDNN_OK
    return k.kernel, k.tile_m, k.tile_n


@pytest.mark.parametrize("case,want", [
    (dict(n=256, c=256, h=14, w=14, k=256), (ROWS, 256, 256)),                                  # 3x3, W stride 1
    (dict(n=128, c=64, h=56, w=56, k=64), (ROWS, 256, 64)),                                     # planned with grouped pixels
    (dict(n=256, c=256, h=56, w=56, k=64, r=1, s=1, pad=0), (IGEMM, 128, 64)),                  # one tap
    (dict(n=128, c=256, h=28, w=28, k=256, stride=2), (PAIR, 256, 256)),                        # W stride 2
    (dict(n=256, c=3, h=224, w=224, k=64, r=7, s=7, stride=2, pad=3), (PAIR, 256, 256)),        # the stem
    (dict(n=4, c=64, h=56, w=56, k=64, dtype=nat.F32, channels_last=False), (ROWS, 256, 64)),
    (dict(n=256, c=256, h=14, w=14, k=256, algo=nat.ALGO_IGEMM), (IGEMM, 128, 256)),            # as asked for
    (dict(n=2, c=8, h=6, w=6, k=8), (DIRECT, 0, 0)),
    (dict(n=32, c=64, h=28, w=28, k=64, groups=64), (DIRECT, 0, 0)),                            # depthwise
    (dict(n=2, c=8, h=6, w=6, k=8, dtype=nat.F64), (DIRECT, 0, 0)),
])
def test_kernels(native_lib, case, want):
    assert kernel_of(native_lib, _desc(**case)) == want


def test_groups_in_channel_blocks(native_lib):
    d = _desc(n=256, c=64, h=56, w=56, k=128, groups=2)
    assert kernel_of(native_lib, d) == (ROWS, 256, 128)                  # the dense filter in front of the packed one
    assert kernel_of(native_lib, d, w=256) == (ROWS, 256, 128)           # in place
    d = _desc(n=64, c=512, h=14, w=14, k=512, groups=16)
    assert kernel_of(native_lib, d, w=256) == (ROWS, 256, 64)
    assert kernel_of(native_lib, d)[0] == IGEMM                          # too many groups for the dense filter


def test_what_the_query_refuses_is_refused(native_lib):
    k = nat.ConvKernel()
    d = _desc(c=8, k=8, groups=3)
    assert native_lib.fdnn_conv2d_main_kernel(ctypes.byref(d), None, None, None, ctypes.byref(k)) == nat.FDNN_BAD_PARAM
    assert native_lib.fdnn_conv2d_main_kernel(ctypes.byref(_desc()), None, None, None, None) == nat.FDNN_BAD_PARAM
