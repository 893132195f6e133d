"""Layers of fewer than eight channels on the window mode: output widths of every remainder, several and single rows per
tile, both layouts of x and y, ragged filter counts, residuals (which take the other path), against torch in fp64."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def fd(native_lib):
    import flagdnn_b200

    assert torch.cuda.is_available()
    yield flagdnn_b200
    assert flagdnn_b200.device_status() == 0, "a kernel recorded a bounded-wait incident"


# n, c, h, w, k, r, s, stride, pad
CASES = [(3, 3, 30, 46, 32, 7, 7, 2, 3), (2, 3, 62, 254, 64, 7, 7, 2, 3), (2, 3, 33, 170, 32, 7, 7, 2, 3), (1, 3, 224, 130, 64, 7, 7, 2, 3),
         (5, 1, 28, 27, 40, 5, 5, 1, 2), (4, 6, 19, 21, 33, 3, 3, 1, 1), (2, 4, 40, 128, 130, 3, 3, 1, 1), (3, 7, 17, 9, 24, 5, 8, 1, 3),
         (9, 2, 12, 50, 16, 3, 4, 3, 0), (2, 3, 96, 96, 64, 7, 7, 2, 3)]


@pytest.mark.parametrize("x_layout", ["nchw", "nhwc"])
@pytest.mark.parametrize("y_layout", ["nchw", "nhwc"])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("case", CASES)
def test_few_channel_layers_match_fp64(fd, case, dtype, x_layout, y_layout):
    n, c, h, w, k, r, s, stride, pad = case
    g = torch.Generator().manual_seed(w * 10 + k)
    fmt = {"nhwc": torch.channels_last, "nchw": torch.contiguous_format}
    x = torch.randn((n, c, h, w), generator=g).to(dtype).cuda().contiguous(memory_format=fmt[x_layout])
    wt = (torch.randn((k, c, r, s), generator=g) * (c * r * s) ** -0.5).to(dtype).cuda()
    b = torch.randn(k, generator=g).to(dtype).cuda()
    want = torch.nn.functional.conv2d(x.double(), wt.double(), b.double(), stride, pad)
    eps = 2.0 ** -8 if dtype == torch.bfloat16 else 2.0 ** -11
    size = want.abs().max().item()
    out = torch.empty(want.shape, dtype=dtype, device="cuda").contiguous(memory_format=fmt[y_layout])
    prev = fd.set_algo("igemm")
    try:
        out.fill_(9.0)
        fd.conv2d(x, wt, b, stride, pad, out=out)
        torch.testing.assert_close(out.double(), want, rtol=eps, atol=eps * size)
        res = torch.randn(want.shape, generator=g).to(dtype).cuda().contiguous(memory_format=fmt[y_layout])
        z = fd.conv_host.conv2d_bias_act(x, wt, b, stride=stride, padding=pad, residual=res, relu=True,
                                         out=torch.empty_like(out))
        torch.testing.assert_close(z.double(), torch.relu(want + res.double()), rtol=2 * eps, atol=2 * eps * size)
    finally:
        fd.set_algo(prev)


def test_neighbouring_pixels_do_not_leak(fd):
    """An infinite pixel reaches exactly the outputs whose windows hold it."""
    x = torch.randn(1, 3, 64, 170, device="cuda").half()
    wt = torch.randn(32, 3, 7, 7, device="cuda").half() * 0.1
    x[0, 1, 30, 77] = float("inf")
    y = fd.conv2d(x, wt, None, 2, 3)
    want = torch.nn.functional.conv2d(x.double(), wt.double(), None, 2, 3)
    assert torch.equal(torch.isfinite(y), torch.isfinite(want))
