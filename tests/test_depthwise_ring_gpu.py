"""Depthwise layers on dense NCHW tensors, whole planes through a ring in shared memory (csrc/conv_depthwise_ring.cu)."""
import pytest
import torch

pytestmark = pytest.mark.gpu

EPS = {torch.bfloat16: 2.0 ** -8, torch.float16: 2.0 ** -11, torch.float32: 2.0 ** -24}

# n, c, h, w, k, stride: a megabyte of 16-bit values and more, where this kernel is the one chosen
LAYERS = {
    "rows_of_16_bytes": (45, 64, 56, 56, 3, 1),
    "rows_of_16_bytes_odd": (1, 4001, 44, 48, 3, 1),   # the last plane has no partner
    "rows_of_words": (17, 43, 30, 26, 3, 1),
    "odd_rows": (61, 41, 17, 13, 3, 1),                # planes start anywhere, groups end off 16 bytes
    "odd_planes": (1, 2051, 15, 18, 3, 1),
    "tiny_planes": (107, 333, 3, 5, 3, 1),
    "single_row": (1200, 30, 1, 17, 3, 1),
    "single_column": (1200, 30, 17, 1, 3, 1),
    "many_groups": (50, 64, 50, 50, 3, 1),             # every slot of the ring several times over
    "two_slots": (4, 14, 110, 110, 3, 1),
    "stride_2": (9, 40, 56, 50, 3, 2),
    "stride_2_odd": (31, 35, 15, 33, 3, 2),
    "five": (19, 40, 28, 30, 5, 1),
    "five_odd": (70, 81, 11, 9, 5, 1),
    "five_stride_2": (33, 26, 27, 24, 5, 2),
    "five_stride_2_odd": (33, 27, 27, 25, 5, 2),
    "channels_wrap": (500, 3, 20, 19, 3, 1),           # partners of different images
    "another_kernel": (2, 24, 24, 24, 3, 1),           # too small a layer
}


@pytest.mark.parametrize("dtype", list(EPS), ids=["bf16", "f16", "f32"])
@pytest.mark.parametrize("name", LAYERS)
def test_planes_match_fp64(native_lib, name, dtype):
    import flagdnn_b200 as fd

    n, c, h, w, k, stride = LAYERS[name]
    g = torch.Generator().manual_seed(n * 1000 + c + h)
    x = torch.randn(n, c, h, w, generator=g).to(dtype).cuda()
    wt = torch.randn(c, 1, k, k, generator=g).to(dtype).cuda()
    b = torch.randn(c, generator=g).to(dtype).cuda()
    got = fd.conv2d(x, wt, b, stride=stride, padding=k // 2, groups=c)
    relu = fd.conv2d_bias_act(x, wt, b, stride=stride, padding=k // 2, groups=c, relu=True)
    args = (stride, k // 2, 1, c)
    ref = torch.nn.functional.conv2d(x.cpu().double(), wt.cpu().double(), b.cpu().double(), *args)
    size = torch.nn.functional.conv2d(x.cpu().double().abs(), wt.cpu().double().abs(), b.cpu().double().abs(), *args)
    # one rounding to the type, and k * k + 1 fp32 additions of at most `size` in all
    bound = EPS[dtype] * ref.abs() + (k * k + 2) * 2.0 ** -24 * size + 2.0 ** -24
    assert bool(((got.cpu().double() - ref).abs() <= bound).all())
    assert torch.equal(relu, torch.relu(got))
    assert fd.device_status() == 0


def test_an_infinite_plane_stays_in_its_channel(native_lib):
    """Two planes share an instruction, not their values."""
    import flagdnn_b200 as fd

    x = torch.randn(200, 8, 18, 18).bfloat16().cuda()
    wt = torch.randn(8, 1, 3, 3).bfloat16().cuda()
    clean = fd.conv2d(x, wt, None, padding=1, groups=8)
    x[0, 2] = float("inf")
    x[1, 5, 3, 3] = float("nan")
    got = fd.conv2d(x, wt, None, padding=1, groups=8)
    same = torch.ones(200, 8, dtype=torch.bool)
    same[0, 2] = same[1, 5] = False
    assert torch.equal(got[same], clean[same])
    assert bool(torch.isnan(got[1, 5, 2:5, 2:5]).all()) and bool(torch.isfinite(got[1, 5, 6:]).all())
