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


@pytest.mark.gpu
def test_filters_packed_for_another_layer_are_refused(native_lib):
    """Two layers whose packed filters take the same bytes per group (24 and 32 channels are both padded to 32): each
    call takes its own buffer and refuses the other's."""
    groups, k, n, hw = 32, 48 * 32, 3, 21
    g = torch.Generator().manual_seed(3)
    layers = []
    for cg in (24, 32):
        x = torch.randn((n, cg * groups, hw, hw), generator=g).to(torch.bfloat16).cuda()
        w = (torch.randn((k, cg, 3, 3), generator=g) * (cg * 9) ** -0.5).to(torch.bfloat16).cuda()      # NCHW: needs packing
        y = torch.full((n, k, hw, hw), -7.0, dtype=torch.bfloat16, device="cuda")
        d, plan = _desc(n, cg * groups, hw, hw, k, groups, x.stride(), w.stride(), y.stride()), nat.ConvPlan()
        nat.check(native_lib.fdnn_conv2d_query(ctypes.byref(d), x.data_ptr(), w.data_ptr(), y.data_ptr(), ctypes.byref(plan)))
        assert plan.w_packed == 1
        packed = torch.empty(plan.packed_weight_bytes, dtype=torch.uint8, device="cuda")
        nat.check(native_lib.fdnn_conv2d_pack_weight(ctypes.byref(d), w.data_ptr(), y.data_ptr(), packed.data_ptr(), packed.numel(), None))
        layers.append((d, plan, x, w, y, packed))
    assert layers[0][5].numel() == layers[1][5].numel()
    scratch = torch.empty(max(l[1].workspace_bytes for l in layers), dtype=torch.uint8, device="cuda")

    def run(i, packed):
        d, plan, x, w, y, _ = layers[i]
        return native_lib.fdnn_conv2d_fwd(ctypes.byref(d), x.data_ptr(), w.data_ptr(), packed.data_ptr(), None, None, nat.ACT_NONE,
                                          y.data_ptr(), scratch.data_ptr(), scratch.numel(), None)

    for i in (0, 1):
        assert run(i, layers[1 - i][5]) == nat.FDNN_BAD_PARAM
        assert b"pack again" in native_lib.fdnn_last_error()
        torch.cuda.synchronize()
        assert bool((layers[i][4] == -7.0).all()), "a refused call must not write"
    for i in (0, 1):
        nat.check(run(i, layers[i][5]))
        want = torch.nn.functional.conv2d(layers[i][2].double(), layers[i][3].double(), None, 1, 1, 1, groups)
        torch.testing.assert_close(layers[i][4].double(), want, rtol=2.0 ** -8, atol=2.0 ** -8 * want.abs().max().item())


def test_a_filter_read_in_place_is_not_asked_for_packed(native_lib):
    """Eight groups of 64 channels: planned as one dense layer, run as one launch over the groups that reads w itself."""
    c = k = 512
    d = _desc(16, c, 28, 28, k, 8, (c * 784, 1, 28 * c, c), (64 * 9, 1, 192, 64), (k * 784, 1, 28 * k, k))
    plan = nat.ConvPlan()
    for w, packed in ((0x1000, 0), (None, 1), (0x1002, 1)):     # in place; not known yet; off 16 bytes
        nat.check(native_lib.fdnn_conv2d_query(ctypes.byref(d), 0x100000, w, 0x2000000, ctypes.byref(plan)))
        assert plan.w_packed == packed and (plan.packed_weight_bytes > 0) == bool(packed)
    # two groups of 32 channels stay one dense layer, and [K, C, R, S] filters are packed for it
    d = _desc(256, 64, 56, 56, 128, 2, (64 * 3136, 1, 56 * 64, 64), (32 * 9, 1, 96, 32), (128 * 3136, 1, 56 * 128, 128))
    nat.check(native_lib.fdnn_conv2d_query(ctypes.byref(d), 0x100000, 0x1000, 0x2000000, ctypes.byref(plan)))
    assert plan.w_packed == 1


@pytest.mark.gpu
@pytest.mark.parametrize("groups", [4, 8])
def test_layers_in_one_launch_leave_no_packed_filter_behind(native_lib, groups):
    import flagdnn_b200 as fd

    g = torch.Generator().manual_seed(groups)
    fmt = torch.channels_last
    x = torch.randn((4, 64 * groups, 28, 28), generator=g).to(torch.bfloat16).cuda().contiguous(memory_format=fmt)
    w = (torch.randn((64 * groups, 64, 3, 3), generator=g) / 24).to(torch.bfloat16).cuda().contiguous(memory_format=fmt)
    before = set(fd.conv_host._PACKED_WEIGHT_CACHE)
    y = fd.conv2d(x, w, None, 1, 1, 1, groups)
    assert fd.conv_host.conv2d_plan(x, w, 1, 1, 1, groups)["w_packed"] == 0
    assert set(fd.conv_host._PACKED_WEIGHT_CACHE) <= before
    want = torch.nn.functional.conv2d(x.double(), w.double(), None, 1, 1, 1, groups)
    torch.testing.assert_close(y.double(), want, rtol=2.0 ** -8, atol=2.0 ** -8 * want.abs().max().item())


@pytest.mark.skipif(torch.cuda.is_available(), reason="the addresses are made up; without a device nothing can use them")
@pytest.mark.parametrize("scratch_bytes", [0, 256, 64 * 784 * 2])
def test_too_little_scratch_is_called_that(native_lib, scratch_bytes):
    """Eight groups of 64 channels in NCHW, filter read in place: scratch for less than two relaid-out groups."""
    c = k = 512
    d, plan = _desc(1, c, 28, 28, k, 8, (c * 784, 784, 28, 1), (64 * 9, 1, 192, 64), (k * 784, 784, 28, 1)), nat.ConvPlan()
    x, w, y, scratch = 0x100000, 0x1000000, 0x2000000, 0x3000000
    nat.check(native_lib.fdnn_conv2d_query(ctypes.byref(d), x, w, y, ctypes.byref(plan)))
    assert plan.x_repacked == 1 and plan.w_packed == 0 and plan.workspace_bytes >= 8 * 64 * 784 * 2
    status = native_lib.fdnn_conv2d_fwd(ctypes.byref(d), x, w, None, None, None, nat.ACT_NONE, y,
                                        scratch if scratch_bytes else None, scratch_bytes, None)
    assert status == nat.FDNN_WORKSPACE_TOO_SMALL
