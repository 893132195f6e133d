"""1x1 layers with a shortcut on tiles of 256 columns: three staging buffers, the next tile's box asked for ahead."""
import ctypes

import pytest
import torch

from flagdnn_b200 import _native as nat, device_status

pytestmark = pytest.mark.gpu

CODE = {torch.float16: nat.F16, torch.bfloat16: nat.BF16}
EPS = {torch.bfloat16: 2.0 ** -8, torch.float16: 2.0 ** -11}

# n, c, h, w, k.  A tile is 128 pixels x 256 columns, two epilogue warps take 128 columns each, an SM has several tiles
# where there are more than 148.
LAYERS = {
    "several_tiles": (16, 64, 56, 56, 256),            # 392 tiles
    "two_column_tiles": (33, 128, 28, 28, 512),        # 203 x 2 tiles, the last row tile of 16 pixels
    "four_steps": (100, 256, 14, 14, 256),             # 154 tiles: some SMs have one, some two
    "one_tile": (3, 64, 28, 28, 256),                  # nothing to ask for ahead
    "eight_columns_left": (25, 64, 28, 28, 264),       # the second half of every other tile has no columns
    "one_half_left": (25, 128, 28, 28, 328),           # 72 columns: a box and an eighth of one
    "into_the_second_half": (25, 64, 28, 28, 392),     # 136 columns
    "odd_pixels": (7, 40, 53, 59, 264),                # 172 row tiles, the last one of 1 pixel, a step that is not full
    "narrow": (40, 192, 28, 28, 136),                  # 245 tiles, the second half of 8 columns
}


@pytest.mark.parametrize("act", [nat.ACT_NONE, nat.ACT_RELU], ids=["linear", "relu"])
@pytest.mark.parametrize("dtype", list(EPS), ids=["bf16", "f16"])
@pytest.mark.parametrize("name", LAYERS)
def test_three_buffers_match_fp64_and_two(native_lib, name, dtype, act):
    """Every operand is summed in the same order whatever the tile, so that the widths agree bit for bit; against fp64: one
    rounding to the type, and fp32 sums of at most 256 products, which are far below it."""
    n, c, h, w, k = LAYERS[name]
    g = torch.Generator().manual_seed(n * 1000 + c + k)
    def nhwc(t):
        return t.to(dtype).cuda().contiguous(memory_format=torch.channels_last)
    x = nhwc(torch.randn(n, c, h, w, generator=g))
    wt = (torch.randn(k, c, 1, 1, generator=g) * c ** -0.5).to(dtype).cuda()
    scale, bias = (torch.randn(k, generator=g).to(dtype).cuda() for _ in range(2))
    shortcut = nhwc(torch.randn(n, k, h, w, generator=g))
    pixels = n * h * w
    guard = 4096    # elements on either side of y
    memory = torch.empty(pixels * k + 2 * guard, dtype=dtype, device="cuda")
    y = memory[guard:-guard].view(n, h, w, k).permute(0, 3, 1, 2)
    d = nat.ConvDesc()
    d.dtype, d.n, d.c, d.h, d.w, d.k, d.r, d.s, d.groups = CODE[dtype], n, c, h, w, k, 1, 1, 1
    d.stride_h = d.stride_w = d.dil_h = d.dil_w = 1
    for i in range(4):
        d.x_strides[i], d.w_strides[i], d.y_strides[i] = x.stride(i), wt.stride(i), y.stride(i)
    got = {}
    for width in (nat.ALGO_FLAG_TILE_N_256, nat.ALGO_FLAG_TILE_N_128):
        d.algo = nat.ALGO_IGEMM | width
        plan = nat.ConvPlan()
        nat.check(native_lib.fdnn_conv2d_query(ctypes.byref(d), x.data_ptr(), wt.data_ptr(), y.data_ptr(), ctypes.byref(plan)))
        assert (plan.tile_n, plan.x_repacked, plan.w_packed) == (256 if width == nat.ALGO_FLAG_TILE_N_256 else 128, 0, 0)
        memory.fill_(-7.0)
        nat.check(native_lib.fdnn_conv2d_fwd_residual(
            ctypes.byref(d), x.data_ptr(), wt.data_ptr(), None, bias.data_ptr(), scale.data_ptr(), shortcut.data_ptr(), act,
            y.data_ptr(), None, 0, torch.cuda.current_stream().cuda_stream))
        assert device_status() == 0
        assert bool((memory[:guard] == -7.0).all()) and bool((memory[-guard:] == -7.0).all())
        got[width] = y.clone()
    wide = got[nat.ALGO_FLAG_TILE_N_256]
    assert torch.equal(wide, got[nat.ALGO_FLAG_TILE_N_128])
    want = torch.nn.functional.conv2d(x.double(), wt.double()) * scale.double().view(1, k, 1, 1) + bias.double().view(1, k, 1, 1)
    want = want + shortcut.double()
    if act == nat.ACT_RELU:
        want = want.relu()
    eps = EPS[dtype]
    torch.testing.assert_close(wide.double(), want, rtol=eps, atol=eps * want.abs().max().item())
