"""Arguments of grouped layers that run in one launch: refused like those of one launch per group, before anything is
launched."""
import ctypes

import pytest
import torch

from flagdnn_b200 import _native as nat


def _desc(n, c, h, w, k, groups, x_strides, w_strides, y_strides):
    d = nat.ConvDesc()
    d.dtype = nat.BF16
    d.n, d.c, d.h, d.w, d.k, d.r, d.s, d.groups = n, c, h, w, k, 3, 3, groups
    d.stride_h = d.stride_w = d.dil_h = d.dil_w = 1
    d.pad_top = d.pad_bottom = d.pad_left = d.pad_right = 1
    d.algo = nat.ALGO_AUTO
    d.x_strides[:], d.w_strides[:], d.y_strides[:] = x_strides, w_strides, y_strides
    return d


def _nchw(groups=32):
    c, k, h, w = 24 * groups, 48 * groups, 21, 21
    return _desc(3, c, h, w, k, groups, (c * h * w, h * w, w, 1), (24 * 9, 1, 72, 24), (k * h * w, h * w, w, 1))


@pytest.mark.skipif(torch.cuda.is_available(), reason="the addresses are made up; without a device nothing can use them")
@pytest.mark.parametrize("offset", [2, 8, 16, 128])
def test_scratch_off_256_bytes_is_refused(native_lib, offset):
    d, plan = _nchw(), nat.ConvPlan()
    x, w, y, packed, scratch = 0x10000, 0x4000000, 0x8000000, 0x10000000, 0x20000000
    assert native_lib.fdnn_conv2d_query(ctypes.byref(d), x, w, y, ctypes.byref(plan)) == nat.FDNN_OK
    assert plan.x_repacked == 1 and plan.workspace_bytes > 0
    status = native_lib.fdnn_conv2d_fwd(ctypes.byref(d), x, w, packed if plan.w_packed else None, None, None, nat.ACT_NONE, y,
                                        scratch + offset, plan.workspace_bytes, None)
    assert status == nat.FDNN_BAD_PARAM
    assert b"workspace must be 256-byte aligned" in native_lib.fdnn_last_error()
