"""Small layers of few channels: which kernels take them, and that a pixel reaches the outputs whose windows hold it and
no others, as on the direct kernel."""
import ctypes

import pytest
import torch

from flagdnn_b200 import _native as nat

# n, c, h, w, k, r, stride, pad
SMALL = [(1, 3, 32, 32, 16, 5, 1, 2), (1, 4, 32, 32, 32, 5, 1, 2), (1, 3, 64, 64, 32, 7, 2, 3), (2, 2, 24, 40, 6, 6, 1, 2),
         (1, 3, 32, 32, 16, 11, 1, 5), (1, 3, 56, 56, 8, 9, 1, 4)]


def _plan(lib, case, channels_last, dtype=nat.F16):
    n, c, h, w, k, r, stride, pad = case
    oh, ow = ((e + 2 * pad - r) // stride + 1 for e in (h, w))
    d, plan = nat.ConvDesc(), nat.ConvPlan()
    d.dtype, d.groups, d.algo = dtype, 1, nat.ALGO_AUTO
    d.n, d.c, d.h, d.w, d.k, d.r, d.s = n, c, h, w, k, r, r
    d.stride_h = d.stride_w = stride
    d.pad_top = d.pad_bottom = d.pad_left = d.pad_right = pad
    d.dil_h = d.dil_w = 1

    def strides(ch, e, f):
        return (ch * e * f, 1, f * ch, ch) if channels_last else (ch * e * f, e * f, f, 1)

    d.x_strides[:], d.w_strides[:], d.y_strides[:] = strides(c, h, w), strides(c, r, r), strides(k, oh, ow)
    nat.check(lib.fdnn_conv2d_query(ctypes.byref(d), None, None, None, ctypes.byref(plan)))
    return plan


@pytest.mark.parametrize("channels_last", [True, False])
@pytest.mark.parametrize("case", SMALL)
def test_small_layers_take_no_quads_and_no_thin_rows(native_lib, case, channels_last):
    plan = _plan(native_lib, case, channels_last)
    assert plan.flops < 2e7 and plan.low_channel == 0
    # filters of up to eight taps a row run as pixel windows, wider ones on the direct kernel
    assert plan.algo == (nat.ALGO_IGEMM if case[5] <= 8 else nat.ALGO_DIRECT)


def test_larger_layers_keep_their_quads(native_lib):
    assert _plan(native_lib, (4, 3, 64, 64, 32, 7, 2, 3), True).low_channel == 1
    assert _plan(native_lib, (32, 3, 224, 224, 64, 7, 2, 3), True).low_channel == 2


@pytest.mark.gpu
@pytest.mark.parametrize("layout", [torch.channels_last, torch.contiguous_format])
@pytest.mark.parametrize("case", SMALL)
def test_an_infinite_pixel_stays_in_its_windows(native_lib, case, layout):
    import flagdnn_b200 as fd

    n, c, h, w, k, r, stride, pad = case
    g = torch.Generator().manual_seed(c * r)
    x = torch.randn((n, c, h, w), generator=g).half()
    x[0, c - 1, h // 2, w // 2 + 1] = float("inf")
    x = x.cuda().contiguous(memory_format=layout)
    wt = (torch.randn((k, c, r, r), generator=g) * (c * r * r) ** -0.5).half().cuda().contiguous(memory_format=layout)
    y = fd.conv2d(x, wt, None, stride, pad)
    want = torch.nn.functional.conv2d(x.double(), wt.double(), None, stride, pad)
    finite = torch.isfinite(want)
    assert torch.equal(torch.isfinite(y), finite) and not bool(finite.all())
    # one rounding of an fp32 sum
    size = want[finite].abs().max().item()
    torch.testing.assert_close(y.double()[finite], want[finite], rtol=2.0 ** -11, atol=2.0 ** -11 * size)


@pytest.mark.gpu
@pytest.mark.parametrize("layout", [torch.channels_last, torch.contiguous_format])
@pytest.mark.parametrize("case", SMALL)
def test_residuals_are_taken(native_lib, case, layout):
    """Through the C ABI, which refuses a residual where quads are planned."""
    n, c, h, w, k, r, stride, pad = case
    g = torch.Generator().manual_seed(k * r)
    x = torch.randn((n, c, h, w), generator=g).half().cuda().contiguous(memory_format=layout)
    wt = (torch.randn((k, c, r, r), generator=g) * (c * r * r) ** -0.5).half().cuda().contiguous(memory_format=layout)
    want = torch.nn.functional.conv2d(x.double(), wt.double(), None, stride, pad)
    res = torch.randn(want.shape, generator=g).half().cuda().contiguous(memory_format=layout)
    y = torch.empty_like(res)
    d, plan = nat.ConvDesc(), nat.ConvPlan()
    d.dtype, d.groups, d.algo = nat.F16, 1, nat.ALGO_AUTO
    d.n, d.c, d.h, d.w, d.k, d.r, d.s = n, c, h, w, k, r, r
    d.stride_h = d.stride_w = stride
    d.pad_top = d.pad_bottom = d.pad_left = d.pad_right = pad
    d.dil_h = d.dil_w = 1
    d.x_strides[:], d.w_strides[:], d.y_strides[:] = x.stride(), wt.stride(), y.stride()
    nat.check(native_lib.fdnn_conv2d_query(ctypes.byref(d), x.data_ptr(), wt.data_ptr(), y.data_ptr(), ctypes.byref(plan)))
    packed = torch.empty(max(plan.packed_weight_bytes, 1), dtype=torch.uint8, device="cuda")
    scratch = torch.empty(max(plan.workspace_bytes, 1), dtype=torch.uint8, device="cuda")
    stream = torch.cuda.current_stream().cuda_stream
    if plan.w_packed:
        nat.check(native_lib.fdnn_conv2d_pack_weight(ctypes.byref(d), wt.data_ptr(), y.data_ptr(), packed.data_ptr(), packed.numel(), stream))
    nat.check(native_lib.fdnn_conv2d_fwd_residual(
        ctypes.byref(d), x.data_ptr(), wt.data_ptr(), packed.data_ptr() if plan.w_packed else None, None, None, res.data_ptr(),
        nat.ACT_RELU, y.data_ptr(), scratch.data_ptr(), plan.workspace_bytes, stream))
    want = torch.relu(want + res.double())
    torch.testing.assert_close(y.double(), want, rtol=2.0 ** -11, atol=2.0 ** -11 * want.max().item())   # one rounding
