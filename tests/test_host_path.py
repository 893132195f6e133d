"""The native host path is there, is the one this torch needs, and refuses a library of another ABI."""
import ctypes

import pytest
import torch

from flagdnn_b200 import _native as nat
from flagdnn_b200 import build, conv_host


def test_the_host_path_loads(native_lib):
    fast = conv_host._load_fast()
    assert fast and fast.built_for == build.host_tag()
    assert torch.__version__ in fast.built_for


def test_a_host_path_of_another_torch_is_stale(native_lib, monkeypatch):
    assert not build._host_stale()
    monkeypatch.setattr(torch, "__version__", "2.0.0")
    assert build._host_stale()


def test_a_host_path_of_another_torch_is_not_used(native_lib, monkeypatch):
    monkeypatch.setattr(conv_host, "_fast", None)
    monkeypatch.setattr(build, "host_tag", lambda: "flagdnn host path for torch 2.0.0")
    with pytest.warns(RuntimeWarning, match="native host path is not used"):
        assert conv_host._load_fast() is False


@pytest.mark.parametrize("wrong", [dict(version=1), dict(desc=8), dict(plan=8)])
def test_another_abi_is_refused(native_lib, wrong):
    from flagdnn_b200 import _fastcall

    version = native_lib.fdnn_abi_version() + wrong.get("version", 0)
    desc = ctypes.sizeof(nat.ConvDesc) + wrong.get("desc", 0)
    plan = ctypes.sizeof(nat.ConvPlan) + wrong.get("plan", 0)
    with pytest.raises(ImportError, match="of the C ABI"):
        _fastcall.bind(1, 2, 3, None, version, desc, plan)


def test_calls_that_are_not_the_native_paths_are_left_to_python(native_lib):
    fast = conv_host._load_fast()
    x, w = torch.randn(1, 3, 8, 8), torch.randn(4, 3, 3, 3)
    assert fast.conv(x, w, None, None, None, 1, 1, 1, 1, nat.ALGO_AUTO, nat.ACT_NONE) is None           # no CUDA tensors
    assert fast.conv1d(x[0], w[0], None, 1, 1, 1, 1, nat.ALGO_AUTO) is None
    assert fast.mm(x[0, 0], x[0, 1], nat.ALGO_AUTO) is None
    assert fast.conv(None, "w", None, None, None, 1, 1, 1, 1, nat.ALGO_AUTO, nat.ACT_NONE) is None
