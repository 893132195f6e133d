"""The relayouts in front of the tensor-core kernels (NCHW planes and padded rows, channels-last pixels of any pitch and
alignment, strided views) against the oracle: channel counts that fill no 16-byte piece, tiles with remainders on both
sides, bases one element off."""
import pytest
import torch

import oracle
from cases import TOL

pytestmark = pytest.mark.gpu


def _tol(dtype):
    return TOL[str(dtype).split(".")[1]]


@pytest.fixture(scope="module")
def fd(native_lib):
    import flagdnn_b200

    assert torch.cuda.is_available()
    yield flagdnn_b200
    assert flagdnn_b200.device_status() == 0, "a kernel recorded a bounded-wait incident"


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("case", ["nchw_odd", "nchw_padded_rows", "nhwc_odd", "nhwc_offset", "nhwc_pitch", "strided", "column", "nchw_aligned"])
def test_relayouts_match_oracle(fd, dtype, case):
    g = torch.Generator().manual_seed(5)
    n, c, h, w, k = 3, 51, 11, 13, 24
    if case == "nchw_odd":
        x = torch.randn((n, c, h, w), generator=g).to(dtype).cuda()
    elif case == "nchw_padded_rows":
        x = torch.randn((n, c, h, w + 3), generator=g).to(dtype).cuda()[..., :w]
    elif case == "nhwc_odd":
        x = torch.randn((n, h, w, c), generator=g).to(dtype).cuda().permute(0, 3, 1, 2)
    elif case == "nhwc_offset":
        x = torch.randn((n * h * w * c + 1,), generator=g).to(dtype).cuda()[1:].view(n, h, w, c).permute(0, 3, 1, 2)
    elif case == "nhwc_pitch":
        x = torch.randn((n, h, w, c + 5), generator=g).to(dtype).cuda()[..., :c].permute(0, 3, 1, 2)
    elif case == "column":
        w = 1
        x = torch.randn((n, c, h, w), generator=g).to(dtype).cuda()
    elif case == "nchw_aligned":
        h, w = 24, 16
        x = torch.randn((n, c, h, w), generator=g).to(dtype).cuda()
    else:
        x = torch.randn((n, 2 * c, h, 2 * w), generator=g).to(dtype).cuda()[:, ::2, :, ::2]
    wt = (torch.randn((k, c, 3, 3), generator=g) / (3 * c ** 0.5)).to(dtype).cuda()
    prev = fd.set_algo("igemm")
    try:
        y = fd.conv2d(x, wt, None, padding=1)
    finally:
        fd.set_algo(prev)
    ref = oracle.conv2d_torch_cpu(x, wt, None, 1, 1, 1, 1, relu=False)
    torch.testing.assert_close(y.float().cpu(), ref, **_tol(dtype))


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16, torch.float32])
@pytest.mark.parametrize("shape", [(65, 64, 64), (130, 72, 200), (40, 33, 61), (64, 128, 8), (300, 9, 130)])
def test_mm_matches_fp64(fd, dtype, shape):
    m, k, n = shape
    g = torch.Generator().manual_seed(m + k + n)
    a = torch.randn((m, k), generator=g).to(dtype).cuda()
    b = (torch.randn((k, n), generator=g) / k ** 0.5).to(dtype).cuda()
    prev = fd.set_algo("igemm")
    try:
        y = fd.mm(a, b)
    finally:
        fd.set_algo(prev)
    torch.testing.assert_close(y.double(), a.double() @ b.double(), **_tol(dtype))
