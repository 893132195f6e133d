"""The packed max-pooling and the split average-pooling kernels at the edges of their ranges: odd and single output rows,
windows that reach past the image on every side, NaN, -inf planes, few and many outputs."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def fd(native_lib):
    import flagdnn_b200

    assert torch.cuda.is_available()
    return flagdnn_b200


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("shape", [(2, 8, 1, 1), (1, 16, 2, 3), (3, 64, 7, 9), (2, 24, 112, 112), (5, 8, 13, 6)])
@pytest.mark.parametrize("window", [(3, 2, 1), (3, 2, 0), (3, 1, 1), (2, 2, 0)])
def test_max_pool_equals_torch(fd, dtype, shape, window):
    kernel, stride, pad = window
    n, c, h, w = shape
    if min(h, w) + 2 * pad < kernel:
        pytest.skip("the window does not fit")
    g = torch.Generator().manual_seed(h * 100 + w)
    x = torch.randn(shape, generator=g).to(dtype)
    x.view(-1)[::37] = float("nan")
    x[0, 0] = float("-inf")
    x = x.cuda().contiguous(memory_format=torch.channels_last)
    y = fd.max_pool2d(x, kernel, stride, pad)
    want = torch.nn.functional.max_pool2d(x.cpu().float(), kernel, stride, pad)
    torch.testing.assert_close(y.cpu().float(), want, rtol=0, atol=0, equal_nan=True)


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("shape", [(1, 8, 7, 7), (2, 2048, 6, 6), (3, 24, 5, 9), (64, 40, 16, 3), (300, 512, 4, 4)])
@pytest.mark.parametrize("out", [1, 2])
def test_average_pool_matches_fp64(fd, dtype, shape, out):
    g = torch.Generator().manual_seed(sum(shape))
    x = torch.randn(shape, generator=g).to(dtype).cuda().contiguous(memory_format=torch.channels_last)
    y = fd.adaptive_avg_pool2d(x, out)
    want = torch.nn.functional.adaptive_avg_pool2d(x.double().cpu(), out)
    # one rounding of an fp32 mean: half a unit of the type, and sums within a few 1e-7
    eps = 2.0 ** -8 if dtype == torch.bfloat16 else 2.0 ** -11
    torch.testing.assert_close(y.double().cpu(), want, rtol=eps, atol=1e-6)
