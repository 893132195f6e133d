"""The native host path of the eager operators against the Python code it stands in for."""
import contextlib

import pytest
import torch

import flagdnn_b200 as fd
from flagdnn_b200 import conv_host

pytestmark = pytest.mark.gpu


@contextlib.contextmanager
def python_only():
    """The eager operators without the native host path."""
    loaded = conv_host._load_fast()
    conv_host._fast = False
    try:
        yield
    finally:
        conv_host._fast = loaded


def _both(call):
    """The call natively and through the Python code."""
    native = call()
    with python_only():
        return native, call()


def _huge(kind):
    """Calls whose output alone (3 to 4 TB) no device holds; the operands are one element each, expanded."""
    one = torch.ones((), dtype=torch.bfloat16, device="cuda")
    if kind == "conv2d":
        return lambda: fd.conv2d(one.expand(1, 64, 40000, 40000), one.expand(1024, 64, 1, 1))
    if kind == "conv1d":
        return lambda: fd.conv1d(one.expand(1, 64, 2000000000), one.expand(1024, 64, 1))
    return lambda: fd.mm(one.expand(2000000000, 8), one.expand(8, 1024))


@pytest.mark.parametrize("kind", ["conv2d", "conv1d", "mm"])
def test_out_of_memory_keeps_its_type(native_lib, kind):
    call = _huge(kind)
    with pytest.raises(torch.OutOfMemoryError):
        call()
    with python_only(), pytest.raises(torch.OutOfMemoryError):
        call()


class _Spy:
    """The native module, noting for each call whether it took it."""

    def __init__(self, fast):
        self.fast, self.taken = fast, []

    def __getattr__(self, name):
        fn = getattr(self.fast, name)

        def call(*args):
            y = fn(*args)
            self.taken.append(y is not None)
            return y
        return call


def _routes(monkeypatch, call):
    """(did the native path take it, its result or exception, the Python code's)"""
    def outcome():
        try:
            return call()
        except Exception as exc:
            return exc

    spy = _Spy(conv_host._load_fast())
    monkeypatch.setattr(conv_host, "_fast", spy)
    native = outcome()
    monkeypatch.setattr(conv_host, "_fast", False)
    python = outcome()
    monkeypatch.setattr(conv_host, "_fast", spy.fast)
    return spy.taken == [True], native, python


def _same(native, python):
    assert type(native) is type(python)
    if isinstance(native, Exception):
        assert str(native) == str(python)
        return
    assert native.dtype == python.dtype and native.shape == python.shape and native.stride() == python.stride()
    assert native.requires_grad == python.requires_grad
    assert torch.equal(native, python)


def _tensors(n, c, h, w, k, r, groups, dtype, layout):
    g = torch.Generator().manual_seed(n + c + k)
    x = torch.randn((n, c, h, w), generator=g).to(dtype).cuda().contiguous(memory_format=layout)
    wt = (torch.randn((k, c // groups, r, r), generator=g) / r).to(dtype).cuda().contiguous(memory_format=layout)
    b = torch.randn(k, generator=g).to(dtype).cuda()
    return x, wt, b


LAYOUTS = [torch.channels_last, torch.contiguous_format]
# n, c, h, w, k, r, groups, stride, padding, dilation: in place, relaid out, few channels, depthwise, grouped, small, 1x1
CONVS = [(4, 64, 28, 28, 64, 3, 1, 1, 1, 1), (3, 50, 21, 17, 42, 3, 1, 2, 1, 1), (2, 3, 64, 64, 32, 7, 1, 2, 3, 1),
         (2, 64, 14, 14, 64, 3, 64, 1, 1, 1), (4, 96, 20, 20, 48, 3, 3, 1, 1, 1), (1, 16, 8, 8, 16, 3, 1, 1, 0, 2),
         (8, 256, 14, 14, 64, 1, 1, 1, 0, 1)]


@pytest.mark.parametrize("layout", LAYOUTS)
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16, torch.float32])
@pytest.mark.parametrize("case", CONVS)
def test_conv2d_is_the_same_call(native_lib, monkeypatch, case, dtype, layout):
    n, c, h, w, k, r, groups, stride, pad, dil = case
    x, wt, b = _tensors(n, c, h, w, k, r, groups, dtype, layout)
    taken, native, python = _routes(monkeypatch, lambda: fd.conv2d(x, wt, b, (stride, stride), pad, (dil, dil), groups))
    assert taken
    _same(native, python)
    res = torch.randn_like(python)
    sc = torch.rand(k, device="cuda").to(dtype)
    for act in ("none", "relu", "gelu", "gelu_tanh"):
        taken, native, python = _routes(monkeypatch, lambda: conv_host.conv2d_bias_act(
            x, wt, b, stride=stride, padding=(pad, pad), dilation=dil, groups=groups, scale=sc, residual=res, activation=act))
        assert taken == (c > 4), "a residual on pixel quads is added in a second step, by the Python code"
        _same(native, python)
    if groups == 1:
        taken, native, python = _routes(monkeypatch, lambda: conv_host.fused_conv2d_bias_relu(
            x, wt, b, stride=stride, padding=pad, dilation=dil, scale=sc))
        assert taken
        _same(native, python)


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("rows", [False, True])
@pytest.mark.parametrize("case", [(2, 33, 201, 40, 3, 1, 2, 1, 1), (4, 64, 96, 64, 5, 1, 1, 2, 4), (3, 32, 64, 32, 3, 32, 1, 1, 1)])
def test_conv1d_is_the_same_call(native_lib, monkeypatch, case, rows, dtype):
    n, c, length, k, r, groups, stride, dil, pad = case
    x = torch.randn(n, c, length, device="cuda").to(dtype)
    if rows:
        x = x.transpose(1, 2).contiguous().transpose(1, 2)
    wt, b = torch.randn(k, c // groups, r, device="cuda").to(dtype), torch.randn(k, device="cuda").to(dtype)
    taken, native, python = _routes(monkeypatch, lambda: fd.conv1d(x, wt, b, stride, pad, dil, groups))
    assert taken
    _same(native, python)


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("form", ["plain", "first transposed", "second transposed", "strided", "one row"])
def test_mm_is_the_same_call(native_lib, monkeypatch, form, dtype):
    m, k, n = (1 if form == "one row" else 130), 72, 104
    a, b = torch.randn(m, k, device="cuda").to(dtype), torch.randn(k, n, device="cuda").to(dtype)
    if form == "first transposed":
        a = a.t().contiguous().t()
    elif form == "second transposed":
        b = b.t().contiguous().t()
    elif form == "strided":
        a, b = torch.randn(m, 2 * k, device="cuda").to(dtype)[:, ::2], torch.randn(k, 3 * n, device="cuda").to(dtype)[:, 5:5 + n]
    taken, native, python = _routes(monkeypatch, lambda: fd.mm(a, b))
    assert taken
    _same(native, python)


def test_calls_left_to_the_python_code(native_lib, monkeypatch):
    x, wt, b = _tensors(2, 32, 15, 15, 24, 3, 1, torch.bfloat16, torch.channels_last)
    far = torch.randn(48, device="cuda").to(torch.bfloat16)[::2]
    nchw = torch.randn(2, 24, 15, 15, device="cuda").to(torch.bfloat16)
    sub = torch.nn.Parameter(wt)
    calls = {
        "list": lambda: fd.conv2d(x, wt, b, [1, 1], [1, 1]),
        "same": lambda: fd.conv2d(x, wt, b, 1, "same"),
        "bias apart": lambda: fd.conv2d(x, wt, far, 1, 1),
        "fp64": lambda: fd.conv2d(x.double(), wt.double(), b.double(), 1, 1),
        "empty": lambda: fd.conv2d(x[:0], wt, b, 1, 1),
        "no output": lambda: fd.conv2d(x[:, :, :2, :2], wt, b, 1, 0),
        "residual of another layout": lambda: conv_host.conv2d_bias_act(x, wt, b, padding=1, residual=nchw, relu=True),
    }
    for name, call in calls.items():
        taken, native, python = _routes(monkeypatch, call)
        assert not taken, name
        _same(native, python)
    taken, native, python = _routes(monkeypatch, lambda: fd.conv2d(x, sub, b, 1, 1))     # parameters are plain tensors
    assert taken and not native.requires_grad
    _same(native, python)


def test_refused_calls_end_in_the_same_errors(native_lib, monkeypatch):
    x, wt, b = _tensors(2, 32, 15, 15, 24, 3, 1, torch.bfloat16, torch.channels_last)
    row = torch.randn(2, 32, 40, device="cuda").to(torch.bfloat16)
    calls = [
        lambda: fd.conv2d(x[0], wt, b), lambda: fd.conv2d(x, wt.half(), b), lambda: fd.conv2d(x, wt.cpu(), b),
        lambda: fd.conv2d(x.cpu(), wt.cpu(), b.cpu()), lambda: fd.conv2d(x, wt, b[:3]), lambda: fd.conv2d(x, wt, b.half()),
        lambda: fd.conv2d(x, wt, b, 0), lambda: fd.conv2d(x, wt, b, 1, -1), lambda: fd.conv2d(x, wt, b, 1, 1, 0),
        lambda: fd.conv2d(x, wt, b, 1, 1, 1, 0), lambda: fd.conv2d(x, wt, b, 1, 1, 1, 5), lambda: fd.conv2d(x, wt, b, (1, 2, 3)),
        lambda: fd.conv2d(x, wt, b, 1, "other"), lambda: fd.conv2d(x.int(), wt.int()), lambda: fd.conv2d(x[:, :, :1, :1], wt, b),
        lambda: conv_host.fused_conv2d_bias_relu(x, wt, b, activation="tanh"),
        lambda: conv_host.conv2d_bias_act(x, wt, b, scale=b.float()),
        lambda: conv_host.conv2d_bias_act(x, wt, b, padding=1, residual=x),
        lambda: fd.conv1d(row, wt[:, :, 0], b, 0), lambda: fd.conv1d(row, wt[:, :, 0], b, 1, -1),
        lambda: fd.conv1d(row[0, 0], wt[:, :, 0], b), lambda: fd.conv1d(row[:, :, :2], wt[:, :, 0], b),
        lambda: fd.conv1d(row, torch.nn.Parameter(wt[:, :, 0]), b),
        lambda: fd.mm(row[0], row[0]), lambda: fd.mm(row[0], row[0].t().half()), lambda: fd.mm(row, row[0].t()),
    ]
    for i, call in enumerate(calls):
        taken, native, python = _routes(monkeypatch, call)
        assert not taken and isinstance(python, Exception), i
        _same(native, python)


def test_forced_kernels_and_streams_reach_the_native_path(native_lib, monkeypatch):
    x, wt, b = _tensors(4, 64, 28, 28, 64, 3, 1, torch.bfloat16, torch.channels_last)
    for algo in ("direct", "igemm"):
        prev = fd.set_algo(algo)
        try:
            taken, native, python = _routes(monkeypatch, lambda: fd.conv2d(x, wt, b, 1, 1))
        finally:
            fd.set_algo(prev)
        assert taken
        _same(native, python)
    side = torch.cuda.Stream()
    side.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(side):
        taken, native, python = _routes(monkeypatch, lambda: fd.conv2d(x, wt, b, 1, 1))
    torch.cuda.current_stream().wait_stream(side)
    assert taken
    _same(native, python)
