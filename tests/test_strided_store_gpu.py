"""The tensor-core epilogue's stores into y layouts that have no TMA map (NCHW planes, channels-last rows of a pitch
that is not a multiple of 16 bytes).  The reference of each case is the same kernel
writing a dense channels-last y of padded channels: the same accumulations, so results agree bit for bit."""
import pytest
import torch

from cases import TOL

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def fd(native_lib):
    import flagdnn_b200

    assert torch.cuda.is_available()
    yield flagdnn_b200
    assert flagdnn_b200.device_status() == 0, "a kernel recorded a bounded-wait incident"


def _tol(dtype):
    return TOL[str(dtype).split(".")[1]]


def _padded_reference(fd, x, w, bias, pad, residual=None, act="none"):
    """[N, K, OH, OW] computed into a dense channels-last y whose channels are a multiple of eight."""
    k = w.shape[0]
    kp = (k + 7) // 8 * 8
    wp = torch.zeros((kp, *w.shape[1:]), dtype=w.dtype, device=w.device)
    wp[:k] = w
    bp = torch.zeros(kp, dtype=w.dtype, device=w.device)
    bp[:k] = bias
    xc = x.contiguous(memory_format=torch.channels_last)
    rp = None
    if residual is not None:
        rp = torch.zeros((x.shape[0], kp, *residual.shape[2:]), dtype=x.dtype, device=x.device)
        rp[:, :k] = residual
        rp = rp.contiguous(memory_format=torch.channels_last)
    y = fd.conv_host.conv2d_bias_act(xc, wp, bp, padding=pad, residual=rp, activation=act)
    return y[:, :k]


# (n, c, h, w, k): OH * OW divisible by 8, 4, 2, 1; images smaller than a warp's 32 rows; K across tiles and ragged
SHAPES = [(3, 16, 16, 16, 64), (2, 24, 14, 14, 72), (3, 16, 10, 13, 40), (5, 24, 7, 7, 33), (9, 8, 3, 5, 130),
          (2, 20, 1, 301, 257), (4, 12, 9, 11, 50), (2, 100, 21, 19, 150), (40, 16, 1, 1, 17), (2, 16, 13, 1, 30)]


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16, torch.float32])
@pytest.mark.parametrize("shape", SHAPES)
@pytest.mark.parametrize("layout", ["nchw", "nhwc", "offset"])
def test_strided_stores_match_dense_channels_last(fd, dtype, shape, layout):
    n, c, h, w, k = shape
    g = torch.Generator().manual_seed(n * 1000 + k)
    x = torch.randn((n, c, h, w), generator=g).to(dtype).cuda()
    wt = (torch.randn((k, c, 3, 3), generator=g) / (3 * c ** 0.5)).to(dtype).cuda()
    bias = torch.randn(k, generator=g).to(dtype).cuda()
    if layout == "nchw":
        out = torch.full((n, k, h, w), 7.0, dtype=dtype, device="cuda")
    elif layout == "nhwc":
        out = torch.full((n, h, w, k), 7.0, dtype=dtype, device="cuda").permute(0, 3, 1, 2)
    else:   # one element past an aligned base, rows of K + 3 channels
        base = torch.full((n * h * w * (k + 3) + 1,), 7.0, dtype=dtype, device="cuda")
        out = base[1:].view(n, h, w, k + 3)[..., :k].permute(0, 3, 1, 2)
    xin = x if layout == "nchw" else x.contiguous(memory_format=torch.channels_last)
    prev = fd.set_algo("igemm")
    try:
        for act, residual in (("none", False), ("relu", True), ("gelu", False)):
            res = torch.randn((n, k, h, w), generator=g).to(dtype).cuda() if residual else None
            res_in = None
            if residual:
                res_in = torch.empty_strided(out.shape, out.stride(), dtype=dtype, device="cuda")
                res_in.copy_(res)
            out.fill_(7.0)
            fd.conv_host.conv2d_bias_act(xin, wt, bias, padding=1, residual=res_in, activation=act, out=out)
            want = _padded_reference(fd, x, wt, bias, 1, res, act)
            if residual and (layout == "offset" or h * w == 1):
                # the residual's alignment (or, over extents of one, its strides) differ from y's: it is added in a
                # second step on one side, which rounds twice
                torch.testing.assert_close(out.float(), want.float(), **_tol(dtype))
            else:
                assert torch.equal(out, want), (act, residual, (out.float() - want.float()).abs().max())
    finally:
        fd.set_algo(prev)
    if layout == "offset":
        gap = base[1:].view(n, h, w, k + 3)[..., k:]
        assert (gap == 7.0).all() and base[0] == 7.0, "elements between the rows of y were written"
