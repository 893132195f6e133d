"""NCHW layers in a captured graph: the filter is packed on the way, so that replays read it as it is by then."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,c,hw,k", [(1, 64, 14, 64), (32, 128, 28, 128)], ids=["small", "medium"])
def test_replays_read_the_current_filter(native_lib, n, c, hw, k):
    import flagdnn_b200 as fd

    x = torch.randn(n, c, hw, hw, device="cuda").half()
    w = (torch.randn(k, c, 3, 3, device="cuda") * (c * 9) ** -0.5).half()
    fd.conv2d(x, w, None, padding=1)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        y = fd.conv2d(x, w, None, padding=1)
    graph.replay()
    assert torch.equal(y, fd.conv2d(x, w, None, padding=1))
    w.copy_(torch.randn_like(w) * (c * 9) ** -0.5)
    graph.replay()
    assert torch.equal(y, fd.conv2d(x, w.clone(), None, padding=1))
    assert fd.device_status() == 0
