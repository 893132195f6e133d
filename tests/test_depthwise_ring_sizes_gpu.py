"""Depthwise layers on dense NCHW tensors: the sizes from which whole planes go through a ring in shared memory."""
import pytest
import torch

pytestmark = pytest.mark.gpu

EPS = {torch.bfloat16: 2.0 ** -8, torch.float16: 2.0 ** -11, torch.float32: 2.0 ** -24}

# n, c, h, w, k, stride: just past the lines between the kernels, for one type or for all
LAYERS = {
    "rows_of_16_bytes": (89, 451, 24, 24, 3, 1),
    "large_rows_of_16_bytes": (113, 143, 56, 56, 3, 1),
    "rows_of_8_bytes": (17, 129, 26, 28, 3, 1),
    "two_slots": (11, 14, 110, 110, 3, 1),
    "stride_2": (25, 41, 56, 50, 3, 2),
    "stride_2_odd": (110, 35, 15, 33, 3, 2),
    "stride_2_odd_planes": (73, 61, 31, 31, 3, 2),
    "five": (31, 41, 28, 30, 5, 1),
    "five_rows_of_8_bytes": (40, 41, 26, 28, 5, 1),
    "five_stride_2": (97, 27, 27, 26, 5, 2),
    "five_stride_2_odd": (97, 27, 27, 25, 5, 2),
    "five_stride_2_rows_of_16_bytes": (33, 81, 40, 40, 5, 2),
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
    args = (stride, k // 2, 1, c)
    ref = torch.nn.functional.conv2d(x.double(), wt.double(), b.double(), *args)
    size = torch.nn.functional.conv2d(x.double().abs(), wt.double().abs(), b.double().abs(), *args)
    # one rounding to the type, and k * k + 1 fp32 additions of at most `size` in all
    bound = EPS[dtype] * ref.abs() + (k * k + 2) * 2.0 ** -24 * size + 2.0 ** -24
    assert bool(((got.double() - ref).abs() <= bound).all())
    assert fd.device_status() == 0


def test_an_infinite_plane_stays_in_its_channel(native_lib):
    """Two planes share an instruction, not their values: in a layer large enough for the ring."""
    import flagdnn_b200 as fd

    x = torch.randn(400, 8, 18, 18).bfloat16().cuda()
    wt = torch.randn(8, 1, 3, 3).bfloat16().cuda()
    clean = fd.conv2d(x, wt, None, padding=1, groups=8)
    x[0, 2] = float("inf")
    x[1, 5, 3, 3] = float("nan")
    got = fd.conv2d(x, wt, None, padding=1, groups=8)
    same = torch.ones(400, 8, dtype=torch.bool)
    same[0, 2] = same[1, 5] = False
    assert torch.equal(got[same], clean[same])
    assert bool(torch.isnan(got[1, 5, 2:5, 2:5]).all()) and bool(torch.isfinite(got[1, 5, 6:]).all())


@pytest.mark.parametrize("n,c,hw,k,stride,dtype", [(2, 96, 57, 3, 1, torch.bfloat16), (2, 96, 57, 3, 2, torch.bfloat16),
                                                   (3, 64, 57, 5, 1, torch.bfloat16), (2, 96, 57, 5, 2, torch.bfloat16),
                                                   (7, 96, 57, 3, 2, torch.float32)])
def test_a_few_large_planes_take_no_longer_than_unaligned_ones(native_lib, n, c, hw, k, stride, dtype):
    """Odd rows are read by single elements or words whatever the base's alignment, but only an aligned base can go through the
    ring: where there is little for it to overlap it must not be taken (these were 1.4 to 1.8 times as long there)."""
    import flagdnn_b200 as fd

    def microseconds(offset):
        memory = torch.randn(n * c * hw * hw + offset, device="cuda").to(dtype)
        x = memory[offset:].view(n, c, hw, hw)
        wt = torch.randn(c, 1, k, k, device="cuda").to(dtype)
        fd.conv2d(x, wt, None, stride=stride, padding=k // 2, groups=c)
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph):
            for _ in range(40):
                y = fd.conv2d(x, wt, None, stride=stride, padding=k // 2, groups=c)
        times = []
        for _ in range(9):
            a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            a.record()
            graph.replay()
            b.record()
            b.synchronize()
            times.append(a.elapsed_time(b) * 25)
        return sorted(times)[4]

    aligned, unaligned = microseconds(0), microseconds(1)
    assert aligned < 1.2 * unaligned, (aligned, unaligned)
