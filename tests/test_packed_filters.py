"""Packed filters kept between calls: one filter tensor used by layers of different group counts, padding or data."""
import ctypes

import pytest
import torch

import flagdnn_b200 as fd
from flagdnn_b200 import conv_host

# One filter [K, C/G, R, R] for two group counts, and what the layer of the first count is planned as.
GROUP_PAIRS = [
    # (dtype, K, C/G, R, spatial, images, two group counts)
    pytest.param(torch.bfloat16, 192, 32, 3, 56, 64, (3, 4), id="dense-bf16"),     # 96 and 128 channels: the same c_padded
    pytest.param(torch.float16, 48, 8, 3, 56, 32, (6, 8), id="dense-f16"),
    pytest.param(torch.bfloat16, 96, 16, 3, 56, 16, (3, 4), id="pixel-grouped"),
    pytest.param(torch.bfloat16, 120, 20, 3, 40, 16, (2, 3), id="ragged-bf16"),    # 40 and 60 channels: packed behind the dense filter
    pytest.param(torch.float32, 120, 20, 3, 40, 16, (2, 3), id="ragged-f32"),
]


def _plan(x, w, pad, groups):
    n, _, h, wd = x.shape
    out = torch.empty((n, w.shape[0], h, wd), dtype=x.dtype, device="meta", memory_format=torch.channels_last)
    return conv_host._plan_for(x, w, out, (1, 1), (pad, pad, pad, pad), (1, 1), groups, conv_host.nat.ALGO_AUTO)


@pytest.mark.parametrize("dtype,k,cg,r,hw,n,counts", GROUP_PAIRS)
def test_two_group_counts_never_share_a_packed_filter(native_lib, dtype, k, cg, r, hw, n, counts):
    w = torch.empty((k, cg, r, r), dtype=dtype, device="meta").contiguous(memory_format=torch.channels_last)
    layouts = []
    for g in counts:
        x = torch.empty((n, cg * g, hw, hw), dtype=dtype, device="meta", memory_format=torch.channels_last)
        d, plan = _plan(x, w, r // 2, g)
        if plan.w_packed:
            layouts.append(conv_host._packed_layout(d, plan))
    assert len(set(layouts)) == len(layouts)


def test_left_paddings_of_a_stem_never_share_a_packed_filter(native_lib):
    # quads of pixels: the filter is stored shifted by what the left padding leaves of a 16-byte piece
    w = torch.empty((64, 3, 7, 7), dtype=torch.bfloat16, device="meta")
    x = torch.empty((32, 3, 224, 224), dtype=torch.bfloat16, device="meta", memory_format=torch.channels_last)
    layouts = set()
    for pad in (2, 3):
        out = torch.empty((32, 64, 112, 112), dtype=x.dtype, device="meta", memory_format=torch.channels_last)
        d, plan = conv_host._plan_for(x, w, out, (2, 2), (pad, 5 - pad, pad, 5 - pad), (1, 1), 1, conv_host.nat.ALGO_AUTO)
        assert plan.low_channel
        layouts.add(conv_host._packed_layout(d, plan))
    assert len(layouts) == 2


@pytest.mark.gpu
@pytest.mark.parametrize("dtype,k,cg,r,hw,n,counts", GROUP_PAIRS)
def test_one_filter_under_two_group_counts(native_lib, dtype, k, cg, r, hw, n, counts):
    g = torch.Generator().manual_seed(k + cg)
    w = (torch.randn((k, cg, r, r), generator=g) * (cg * r * r) ** -0.5).to(dtype).cuda().contiguous(memory_format=torch.channels_last)
    eps = {torch.bfloat16: 2.0 ** -8, torch.float16: 2.0 ** -11, torch.float32: 2e-5}[dtype]   # one rounding; split TF32
    for groups in counts + counts:
        x = torch.randn((n, cg * groups, hw, hw), generator=g).to(dtype).cuda().contiguous(memory_format=torch.channels_last)
        y = fd.conv2d(x, w, None, 1, r // 2, 1, groups)
        want = torch.nn.functional.conv2d(x.double(), w.double(), None, 1, r // 2, 1, groups)
        torch.testing.assert_close(y.double(), want, rtol=eps, atol=eps * want.abs().max().item())


@pytest.mark.gpu
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("c,k,groups", [(32, 32, 2), (96, 96, 12), (24, 40, 4)])
def test_a_small_grouped_filter_is_packed_for_the_tensor_core_route(native_lib, dtype, c, k, groups):
    """Planned as the direct kernel, which reads w itself; the packed form is that of the route a forced call takes, and
    packing reads C / groups channels of each filter."""
    nat = conv_host.nat
    cg, hw, r = c // groups, 6, 3
    g = torch.Generator().manual_seed(c + k)
    fmt = torch.channels_last
    x = torch.randn((1, c, hw, hw), generator=g).to(dtype).cuda().contiguous(memory_format=fmt)
    w = (torch.randn((k, cg, r, r), generator=g) * (cg * r * r) ** -0.5).to(dtype).cuda()
    y = torch.empty((1, k, hw, hw), dtype=dtype, device="cuda", memory_format=fmt)
    args = (x, w, y, (1, 1), (1, 1, 1, 1), (1, 1), groups)
    d, plan = conv_host._plan_for(*args, nat.ALGO_AUTO)
    assert plan.algo == nat.ALGO_DIRECT
    forced, want_plan = conv_host._plan_for(*args, nat.ALGO_IGEMM)
    assert want_plan.w_packed
    packed = torch.empty(want_plan.packed_weight_bytes, dtype=torch.uint8, device="cuda")
    stream = torch.cuda.current_stream().cuda_stream
    nat.check(native_lib.fdnn_conv2d_pack_weight(ctypes.byref(d), w.data_ptr(), y.data_ptr(), packed.data_ptr(), packed.numel(), stream))
    scratch = torch.empty(max(want_plan.workspace_bytes, 256), dtype=torch.uint8, device="cuda")
    nat.check(native_lib.fdnn_conv2d_fwd(ctypes.byref(forced), x.data_ptr(), w.data_ptr(), packed.data_ptr(), None, None, nat.ACT_NONE,
                                         y.data_ptr(), scratch.data_ptr(), scratch.numel(), stream))
    want = torch.nn.functional.conv2d(x.double(), w.double(), None, 1, 1, 1, groups)
    eps = {torch.bfloat16: 2.0 ** -8, torch.float32: 2e-5}[dtype]   # one rounding; split TF32
    torch.testing.assert_close(y.double(), want, rtol=eps, atol=eps * want.abs().max().item())
