"""Grouped layers in one launch: against one launch per group (the same sums, bit for bit), against torch in fp64, with
ragged channel counts, every epilogue, both layouts, and a non-finite value that stays in its group."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def fd(native_lib):
    import flagdnn_b200

    assert torch.cuda.is_available()
    yield flagdnn_b200
    assert flagdnn_b200.device_status() == 0, "a kernel recorded a bounded-wait incident"


def _tensors(case, dtype, layout):
    n, c, h, w, k, r, stride, groups = case
    g = torch.Generator().manual_seed(c * 3 + k)
    fmt = torch.channels_last if layout == "nhwc" else torch.contiguous_format
    x = torch.randn((n, c, h, w), generator=g).to(dtype).cuda().contiguous(memory_format=fmt)
    wt = (torch.randn((k, c // groups, r, r), generator=g) * (c // groups * r * r) ** -0.5).to(dtype).cuda()
    b = torch.randn(k, generator=g).to(dtype).cuda()
    return x, wt.contiguous(memory_format=fmt), b


CASES = [(3, 768, 21, 21, 1536, 3, 1, 32), (2, 256, 14, 14, 256, 3, 1, 16), (5, 384, 9, 11, 384, 3, 2, 16),
         (4, 640, 13, 13, 1280, 3, 1, 16), (7, 1152, 8, 8, 1152, 1, 1, 12), (40, 512, 28, 30, 512, 3, 1, 32), (2, 512, 30, 17, 2304, 5, 1, 16)]


@pytest.mark.parametrize("layout", ["nhwc", "nchw"])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16, torch.float32])
@pytest.mark.parametrize("case", CASES)
def test_one_launch_equals_one_per_group(fd, case, dtype, layout):
    n, c, h, w, k, r, stride, groups = case
    x, wt, b = _tensors(case, dtype, layout)
    assert fd.conv_host.conv2d_plan(x, wt, stride, r // 2, 1, groups)["algo"] != 1 or dtype == torch.float32
    scale = torch.rand(k, device="cuda").to(dtype) + 0.5
    y = fd.conv2d(x, wt, b, stride, r // 2, 1, groups)
    res = torch.randn_like(y)
    z = fd.conv_host.conv2d_bias_act(x, wt, b, stride=stride, padding=r // 2, groups=groups, scale=scale, residual=res, relu=True)
    want = torch.nn.functional.conv2d(x.double(), wt.double(), b.double(), stride, r // 2, 1, groups)
    eps = {torch.bfloat16: 2.0 ** -8, torch.float16: 2.0 ** -11, torch.float32: 2e-5}[dtype]
    torch.testing.assert_close(y.double(), want, rtol=eps, atol=eps * want.abs().max().item())
    if dtype == torch.float32:
        return   # one launch per group, or exact products where a group is small
    prev = fd.set_algo("igemm")
    try:
        y_loop = fd.conv2d(x, wt.clone(memory_format=torch.preserve_format), b, stride, r // 2, 1, groups)
        z_loop = fd.conv_host.conv2d_bias_act(x, wt.clone(memory_format=torch.preserve_format), b, stride=stride,
                                              padding=r // 2, groups=groups, scale=scale, residual=res, relu=True)
    finally:
        fd.set_algo(prev)
    assert torch.equal(y, y_loop)
    assert torch.equal(z, z_loop)


@pytest.mark.parametrize("groups", [2, 4, 8, 16])
def test_few_groups_match_fp64(fd, groups):
    case = (6, 48 * groups, 19, 23, 40 * groups, 3, 1, groups)
    x, wt, b = _tensors(case, torch.bfloat16, "nhwc")
    y = fd.conv2d(x, wt, b, 1, 1, 1, groups)
    want = torch.nn.functional.conv2d(x.double(), wt.double(), b.double(), 1, 1, 1, groups)
    torch.testing.assert_close(y.double(), want, rtol=2.0 ** -8, atol=2.0 ** -8 * want.abs().max().item())


def test_a_non_finite_value_stays_in_its_group(fd):
    case = CASES[1]
    x, wt, b = _tensors(case, torch.bfloat16, "nhwc")
    clean = fd.conv2d(x, wt, b, 1, 1, 1, 16)
    x[:, 16 * 5 + 3] = float("inf")
    y = fd.conv2d(x, wt, b, 1, 1, 1, 16)
    other = [i for i in range(256) if i // 16 != 5]
    assert torch.equal(y[:, other], clean[:, other])
