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
