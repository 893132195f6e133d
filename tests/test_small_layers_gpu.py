"""Small layers: the 16-bit ones that go to the tensor-core kernel, the direct kernel's split reductions (fp32, fp64,
groups), depthwise planes of odd sizes and the channels-last depthwise kernel's tiles, against torch in fp64; and the C
ABI called for a small layer without packed filter and scratch."""
import ctypes

import pytest
import torch

from flagdnn_b200 import _native as nat

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def fd(native_lib):
    import flagdnn_b200

    assert torch.cuda.is_available()
    yield flagdnn_b200
    assert flagdnn_b200.device_status() == 0, "a kernel recorded a bounded-wait incident"


# the rounding of the result type, and fp32 sums (3xTF32 products: 4e-6 of the result's size, as measured everywhere)
_EPS = {torch.bfloat16: 2.0 ** -8, torch.float16: 2.0 ** -11, torch.float32: 2e-5, torch.float64: 1e-12}


def _check(y, x, w, b, stride, pad, groups):
    want = torch.nn.functional.conv2d(x.double(), w.double(), None if b is None else b.double(), stride, pad, 1, groups)
    scale = want.abs().max().item()
    torch.testing.assert_close(y.double(), want, rtol=_EPS[y.dtype], atol=_EPS[y.dtype] * scale)


@pytest.mark.parametrize("layout", ["nchw", "nhwc"])
@pytest.mark.parametrize("dtype", list(_EPS))
@pytest.mark.parametrize("case", [(1, 64, 14, 14, 64, 3, 1, 1, 1), (4, 152, 7, 13, 48, 3, 2, 1, 1), (1, 3, 30, 31, 10, 7, 2, 3, 1),
                                  (2, 97, 5, 5, 33, 1, 1, 0, 1), (1, 256, 3, 3, 8, 3, 1, 0, 1), (1, 96, 9, 9, 12, 3, 1, 1, 3),
                                  (1, 24, 6, 6, 5, 2, 1, 0, 1)])
def test_small_layers_match_fp64(fd, case, dtype, layout):
    n, c, h, w, k, r, stride, pad, groups = case
    g = torch.Generator().manual_seed(c * 7 + k)
    fmt = torch.channels_last if layout == "nhwc" else torch.contiguous_format
    x = torch.randn((n, c, h, w), generator=g).to(dtype).cuda().contiguous(memory_format=fmt)
    wt = (torch.randn((k, c // groups, r, r), generator=g) * (c // groups * r * r) ** -0.5).to(dtype).cuda().contiguous(memory_format=fmt)
    b = torch.randn(k, generator=g).to(dtype).cuda()
    _check(fd.conv2d(x, wt, b, stride, pad, 1, groups), x, wt, b, stride, pad, groups)


@pytest.mark.parametrize("layout", ["nchw", "nhwc"])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16, torch.float32])
@pytest.mark.parametrize("case", [(1, 64, 7, 7, 3, 1), (3, 104, 9, 17, 3, 1), (2, 64, 8, 8, 3, 2), (5, 200, 13, 5, 3, 2),
                                  (2, 96, 11, 10, 5, 1), (3, 64, 15, 9, 5, 2), (2, 130, 1, 1, 3, 1), (300, 128, 3, 2, 3, 1),
                                  (2, 7, 33, 31, 3, 1), (3, 109, 14, 15, 3, 2), (2, 37, 9, 8, 5, 1), (1, 50, 111, 109, 3, 1), (40, 99, 7, 5, 5, 2)])
def test_depthwise_tiles_match_fp64(fd, case, dtype, layout):
    n, c, h, w, r, stride = case
    g = torch.Generator().manual_seed(c + h)
    fmt = torch.channels_last if layout == "nhwc" else torch.contiguous_format
    x = torch.randn((n, c, h, w), generator=g).to(dtype).cuda().contiguous(memory_format=fmt)
    wt = (torch.randn((c, 1, r, r), generator=g) / r).to(dtype).cuda()
    b = torch.randn(c, generator=g).to(dtype).cuda()
    _check(fd.conv2d(x, wt, b, stride, r // 2, 1, c), x, wt, b, stride, r // 2, c)
    # scale, residual and GELU take the other epilogue of the same kernels
    scale = (torch.rand(c, generator=g) + 0.5).to(dtype).cuda()
    y0 = fd.conv2d(x, wt, None, stride, r // 2, 1, c)
    res = torch.randn(y0.shape, generator=g).to(dtype).cuda().contiguous(memory_format=fmt)
    for act in ("relu", "gelu"):
        y = fd.conv_host.conv2d_bias_act(x, wt, b, stride=stride, padding=r // 2, groups=c, scale=scale, residual=res, activation=act)
        pre = torch.nn.functional.conv2d(x.double(), wt.double(), None, stride, r // 2, 1, c)
        pre = pre * scale.double().view(1, -1, 1, 1) + b.double().view(1, -1, 1, 1) + res.double()
        want = torch.relu(pre) if act == "relu" else torch.nn.functional.gelu(pre)
        size = want.abs().max().item()
        torch.testing.assert_close(y.double(), want, rtol=2 * _EPS[dtype], atol=2 * _EPS[dtype] * size)


def test_small_layer_without_packed_filter_and_scratch(native_lib):
    x = torch.randn(1, 64, 14, 14, device="cuda").half()          # NCHW: the tensor-core plan needs both
    w = (torch.randn(64, 64, 3, 3, device="cuda") / 24).half()
    y = torch.empty(1, 64, 14, 14, device="cuda").half()
    d = nat.ConvDesc()
    d.dtype, d.n, d.c, d.h, d.w, d.k, d.r, d.s = nat.F16, 1, 64, 14, 14, 64, 3, 3
    d.stride_h = d.stride_w = d.dil_h = d.dil_w = d.groups = 1
    d.pad_top = d.pad_bottom = d.pad_left = d.pad_right = 1
    for i in range(4):
        d.x_strides[i], d.w_strides[i], d.y_strides[i] = x.stride(i), w.stride(i), y.stride(i)
    stream = torch.cuda.current_stream().cuda_stream
    nat.check(native_lib.fdnn_conv2d_fwd(ctypes.byref(d), x.data_ptr(), w.data_ptr(), None, None, None, nat.ACT_NONE,
                                         y.data_ptr(), None, 0, stream))
    _check(y, x, w, None, 1, 1, 1)


@pytest.mark.parametrize("c, dtype, code", [(136, torch.bfloat16, nat.BF16), (3, torch.float16, nat.F16), (20, torch.float32, nat.F32)])
def test_scratch_of_the_tightest_layout_is_enough(native_lib, c, dtype, code):
    """The plan asks scratch for line-sized rows (or windows); rows of 16-byte multiples are still accepted, less is not."""
    n, h, w_, k = 4, 40, 46, 64
    x = torch.randn(n, c, h, w_, device="cuda").to(dtype)
    w = (torch.randn(k, c, 3, 3, device="cuda") / (3 * c ** 0.5)).to(dtype)
    y = torch.empty(n, k, h, w_, device="cuda", dtype=dtype)
    d = nat.ConvDesc()
    d.dtype, d.n, d.c, d.h, d.w, d.k, d.r, d.s = code, n, c, h, w_, k, 3, 3
    d.stride_h = d.stride_w = d.dil_h = d.dil_w = d.groups = 1
    d.pad_top = d.pad_bottom = d.pad_left = d.pad_right = 1
    d.algo = nat.ALGO_IGEMM
    for i in range(4):
        d.x_strides[i], d.w_strides[i], d.y_strides[i] = x.stride(i), w.stride(i), y.stride(i)
    plan = nat.ConvPlan()
    nat.check(native_lib.fdnn_conv2d_query(ctypes.byref(d), x.data_ptr(), w.data_ptr(), y.data_ptr(), ctypes.byref(plan)))
    stream = torch.cuda.current_stream().cuda_stream
    packed = torch.empty(plan.packed_weight_bytes, dtype=torch.uint8, device="cuda")
    nat.check(native_lib.fdnn_conv2d_pack_weight(ctypes.byref(d), w.data_ptr(), y.data_ptr(), packed.data_ptr(),
                                                 packed.numel(), stream))
    es = x.element_size()
    tight = (2 if dtype == torch.float32 else 1) * n * h * w_ * -(-c * es // 16) * 16
    assert tight < plan.workspace_bytes
    for nbytes in (plan.workspace_bytes, tight):
        ws = torch.full((nbytes + 256,), 0x55, dtype=torch.uint8, device="cuda")
        y.zero_()
        nat.check(native_lib.fdnn_conv2d_fwd(ctypes.byref(d), x.data_ptr(), w.data_ptr(), packed.data_ptr(), None, None,
                                             nat.ACT_NONE, y.data_ptr(), ws.data_ptr(), nbytes, stream))
        _check(y, x, w, None, 1, 1, 1)
        assert (ws[nbytes:] == 0x55).all(), "scratch written past its end"
    status = native_lib.fdnn_conv2d_fwd(ctypes.byref(d), x.data_ptr(), w.data_ptr(), packed.data_ptr(), None, None,
                                        nat.ACT_NONE, y.data_ptr(), ws.data_ptr(), tight - 16, stream)
    assert status == nat.FDNN_WORKSPACE_TOO_SMALL
