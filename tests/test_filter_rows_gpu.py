"""Layers whose activations are copied once per filter row (csrc/conv_rows_sm100.cu): the sums are those of the kernel that
copies them for every tap, in the same order, so that both must agree bit for bit."""
import pytest
import torch

import oracle

pytestmark = pytest.mark.gpu

# n, c, h, w, k, (r, s), padding, dilation, stride; long reductions or many tiles, where this kernel is the one chosen
LAYERS = {
    "one_tile": (1, 256, 9, 13, 64, (3, 3), 1, 1, 1),
    "two_tiles_full": (1, 256, 16, 15, 64, (3, 3), 1, 1, 1),               # 16 x 16 = 256 walk rows: one pair tile, full
    "one_walk_row_more": (1, 512, 1, 256, 64, (1, 3), (0, 1), 1, 1),       # 257: the second pair holds one
    "images_inside_a_tile": (37, 256, 5, 6, 64, (3, 3), 1, 1, 1),
    "no_padding": (3, 256, 12, 20, 128, (3, 3), 0, 1, 1),
    "wide_padding": (2, 256, 7, 9, 64, (3, 3), (3, 4), 1, 1),
    "two_taps_same": (2, 512, 11, 18, 72, (2, 2), "same", 1, 1),           # right padding above left
    "four_taps_same": (2, 296, 11, 18, 72, (4, 4), "same", 1, 1),
    "dilation_4": (2, 256, 20, 21, 64, (3, 3), 4, 4, 1),
    "nine_taps": (2, 256, 12, 30, 64, (1, 9), (0, 4), 1, 1),
    "ten_taps": (2, 256, 12, 30, 64, (1, 10), (0, 4), 1, 1),               # one more than a copy holds: the other kernel
    "five_by_five": (2, 104, 17, 19, 136, (5, 5), 2, 1, 1),
    "stride_h": (3, 256, 21, 22, 64, (3, 3), 1, 1, (2, 1)),
    "channels_8": (60, 8, 30, 30, 96, (3, 3), 1, 1, 1),
    "channels_24": (1, 24, 112, 112, 24, (3, 3), 1, 1, 1),
    "channels_264": (2, 264, 13, 17, 128, (3, 3), 1, 1, 1),
    "filters_150": (3, 328, 13, 17, 150, (3, 3), 1, 1, 1),                 # rows of 300 bytes
    "filters_264": (3, 320, 14, 14, 264, (3, 3), 1, 1, 1),
    "filters_272": (3, 320, 14, 14, 272, (3, 3), 1, 1, 1),                 # 16 columns of the last tile
    "resident_128": (20, 64, 56, 56, 128, (3, 3), 1, 1, 1),                # several tiles per pair, whole filter kept
    "streamed_128": (28, 128, 28, 28, 128, (3, 3), 1, 1, 1),
    "streamed_256": (60, 192, 28, 28, 256, (3, 3), 1, 1, 1),
    "grouped_pixels": (20, 64, 56, 56, 64, (3, 3), 1, 1, 1),               # the plan packs its filter for grouped pixels
    "images_cut_by_warps": (9, 256, 7, 7, 96, (3, 3), 1, 1, 1),
}


def _tensors(case, dtype, filter_format):
    n, c, h, w, k, rs, _, _, _ = case
    g = torch.Generator().manual_seed(n * 7919 + c * 31 + k)
    x = torch.randn(n, c, h, w, generator=g).to(dtype).cuda().contiguous(memory_format=torch.channels_last)
    wt = (torch.randn(k, c, *rs, generator=g) * (c * rs[0] * rs[1]) ** -0.5).to(dtype).cuda().contiguous(memory_format=filter_format)
    b = (torch.randn(k, generator=g) * 0.1).to(dtype).cuda()
    sc = (torch.rand(k, generator=g) + 0.5).to(dtype).cuda()
    return x, wt, b, sc


def _both(fd, call):
    got = call()
    fd.set_algo("igemm")
    try:
        return got, call()
    finally:
        fd.set_algo("auto")


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16, torch.float32], ids=["bf16", "f16", "f32"])
@pytest.mark.parametrize("filter_format", [torch.channels_last, torch.contiguous_format], ids=["krsc", "kcrs"])
@pytest.mark.parametrize("layout", ["nhwc", "nchw"])
@pytest.mark.parametrize("name", LAYERS)
def test_bit_equal_to_a_copy_per_tap(native_lib, name, layout, filter_format, dtype):
    import flagdnn_b200 as fd

    case = LAYERS[name]
    n, c, h, w, k, rs, pad, dil, stride = case
    x, wt, b, sc = _tensors(case, dtype, filter_format)
    if layout == "nchw":
        x = x.contiguous()
    got, per_tap = _both(fd, lambda: fd.conv2d(x, wt, b, stride=stride, padding=pad, dilation=dil))
    assert torch.equal(got, per_tap)
    assert got.is_contiguous(memory_format=torch.channels_last if layout == "nhwc" else torch.contiguous_format) or 1 in got.shape
    if isinstance(pad, str):
        return
    pd, dl, st = ((v, v) if isinstance(v, int) else v for v in (pad, dil, stride))
    for act in ("relu", "none"):
        call = lambda: fd.fused_conv2d_bias_relu(x, wt, b, stride=st, padding=pd, dilation=dl, scale=sc, activation=act)
        got, per_tap = _both(fd, call)
        assert torch.equal(got, per_tap)
    ref = oracle.conv2d_torch_cpu(x[-1:], wt, b, st, pd, dl, 1, scale=sc, relu=False)
    tol = 1e-4 if dtype == torch.float32 else 1e-2      # the suite's bounds for three TF32 products and for 16 bits
    torch.testing.assert_close(got[-1:].float().cpu(), ref, rtol=tol, atol=tol)
    assert fd.device_status() == 0


def test_outputs_on_any_boundary(native_lib):
    """y as a view: base and pixel pitch on 32, 16, 4 and 2 bytes; nothing beside the view is written."""
    import flagdnn_b200 as fd
    from flagdnn_b200 import conv_host

    x, wt, b, _ = _tensors(LAYERS["images_inside_a_tile"], torch.bfloat16, torch.channels_last)
    want = fd.conv2d(x, wt, b, padding=1)
    n, k, oh, ow = want.shape
    for offset, pitch in ((0, 64), (16, 80), (8, 72), (2, 66), (1, 65)):
        store = torch.full((n * oh * ow * pitch + 64,), 7.0, dtype=torch.bfloat16, device="cuda")
        view = store[offset:offset + n * oh * ow * pitch].view(n, oh, ow, pitch)
        out = view[..., :k].permute(0, 3, 1, 2)
        conv_host.fused_conv2d_bias_relu(x, wt, b, stride=1, padding=1, activation="none", out=out)
        assert torch.equal(out, want), (offset, pitch)
        assert bool((view[..., k:] == 7.0).all()) and bool((store[:offset] == 7.0).all()) and bool((store[-32:] == 7.0).all())


# groups of 16 and 32 channels inside 64-channel blocks: n, c, hw, k, groups, stride_h, padding
GROUPED = {
    "two_of_32": (9, 64, 14, 128, 2, 1, 1),
    "two_of_32_narrow": (9, 64, 14, 64, 2, 1, 1),
    "two_of_32_wide": (5, 64, 15, 256, 2, 1, 1),
    "blocks_of_two": (3, 256, 13, 256, 8, 1, 1),
    "blocks_of_four": (3, 256, 13, 512, 16, 1, 0),
    "four_of_16": (40, 64, 28, 128, 4, 1, 1),
    "stride_h": (9, 64, 15, 128, 2, 2, 1),
    "sixteen_filters": (9, 64, 14, 64, 4, 1, 1),      # too few filters per group: another route
    "block_of_96": (9, 96, 14, 192, 3, 1, 1),         # ... not whole blocks
}


@pytest.mark.parametrize("filter_format", [torch.channels_last, torch.contiguous_format], ids=["krsc", "kcrs"])
@pytest.mark.parametrize("name", GROUPED)
def test_groups_in_channel_blocks(native_lib, name, filter_format):
    import flagdnn_b200 as fd

    n, c, hw, k, groups, stride_h, pad = GROUPED[name]
    g = torch.Generator().manual_seed(c + k + groups)
    x = torch.randn(n, c, hw, hw, generator=g).bfloat16().cuda().contiguous(memory_format=torch.channels_last)
    wt = (torch.randn(k, c // groups, 3, 3, generator=g) * (c // groups * 9) ** -0.5).bfloat16().cuda().contiguous(memory_format=filter_format)
    b = torch.randn(k, generator=g).bfloat16().cuda()
    got = fd.conv2d(x, wt, b, stride=(stride_h, 1), padding=pad, groups=groups)
    ref = torch.nn.functional.conv2d(x.cpu().float(), wt.cpu().float(), b.cpu().float(), (stride_h, 1), pad, 1, groups)
    # fp32 sums of up to 288 products of unit variance in all, rounded once to 8 bits of mantissa
    torch.testing.assert_close(got.float().cpu(), ref, rtol=2 ** -8, atol=2 ** -12)
    # an infinite channel reaches the outputs of its own group only
    x[:, 0] = float("inf")
    other = fd.conv2d(x, wt, b, stride=(stride_h, 1), padding=pad, groups=groups)
    if filter_format == torch.channels_last and name in ("two_of_32", "blocks_of_two", "four_of_16"):
        assert torch.equal(other[:, k // groups:], got[:, k // groups:])
    assert fd.device_status() == 0
