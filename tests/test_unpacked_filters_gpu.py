"""fdnn_conv2d_fwd_unpacked: the filter is packed on the way, and the buffer then serves fdnn_conv2d_fwd."""
import ctypes
import gc

import pytest
import torch

from flagdnn_b200 import _native as nat, device_status

pytestmark = pytest.mark.gpu

CODE = {torch.float16: nat.F16, torch.bfloat16: nat.BF16, torch.float32: nat.F32}
EPS = {torch.bfloat16: 2.0 ** -8, torch.float16: 2.0 ** -11, torch.float32: 2e-5}   # one rounding; split TF32
F16, BF16, F32 = torch.float16, torch.bfloat16, torch.float32


class Layer:
    def __init__(self, dtype, n, c, h, w, k, r, s, stride=1, groups=1, x_format="nchw", w_format="kcrs", seed=0):
        g = torch.Generator().manual_seed(seed + c * 31 + k)
        fmt = {"nchw": torch.contiguous_format, "nhwc": torch.channels_last}[x_format]
        self.pad, self.stride, self.groups = (r // 2, s // 2), stride, groups
        self.x = torch.randn(n, c, h, w, generator=g).to(dtype).cuda().contiguous(memory_format=fmt)
        self.w = (torch.randn(k, c // groups, r, s, generator=g) * (c // groups * r * s) ** -0.5).to(dtype).cuda()
        if w_format == "ck":      # the K dimension contiguous
            self.w = self.w.view(k, c).t().contiguous().t().view(k, c, 1, 1)
        oh, ow = (h + 2 * self.pad[0] - r) // stride + 1, (w + 2 * self.pad[1] - s) // stride + 1
        self.y = torch.empty((n, k, oh, ow), dtype=dtype, device="cuda", memory_format=fmt)
        d = self.d = nat.ConvDesc()
        d.dtype, d.n, d.c, d.h, d.w, d.k, d.r, d.s, d.groups = CODE[dtype], n, c, h, w, k, r, s, groups
        d.stride_h = d.stride_w = stride
        d.dil_h = d.dil_w = 1
        d.pad_top = d.pad_bottom = self.pad[0]
        d.pad_left = d.pad_right = self.pad[1]
        for i in range(4):
            d.x_strides[i], d.w_strides[i], d.y_strides[i] = self.x.stride(i), self.w.stride(i), self.y.stride(i)
        self.plan = nat.ConvPlan()
        nat.check(nat.load().fdnn_conv2d_query(ctypes.byref(d), self.x.data_ptr(), self.w.data_ptr(), self.y.data_ptr(),
                                               ctypes.byref(self.plan)))
        self.scratch = torch.empty(max(self.plan.workspace_bytes, 256), dtype=torch.uint8, device="cuda")

    def buffer(self):
        return torch.full((self.plan.packed_weight_bytes,), 0x2A, dtype=torch.uint8, device="cuda")

    def unpacked(self, packed, nbytes=None, scratch=True, residual=None, act=nat.ACT_NONE):
        self.y.fill_(-7.0)
        return nat.load().fdnn_conv2d_fwd_unpacked(
            ctypes.byref(self.d), self.x.data_ptr(), self.w.data_ptr(), packed if packed is None or isinstance(packed, int) else packed.data_ptr(),
            self.plan.packed_weight_bytes if nbytes is None else nbytes, None, None, None if residual is None else residual.data_ptr(),
            act, self.y.data_ptr(), self.scratch.data_ptr() if scratch else None, self.scratch.numel() if scratch else 0,
            torch.cuda.current_stream().cuda_stream)

    def packed_call(self, packed):
        """fdnn_conv2d_fwd with nothing but the packed filter."""
        self.y.fill_(-7.0)
        return nat.load().fdnn_conv2d_fwd(ctypes.byref(self.d), self.x.data_ptr(), None, packed.data_ptr(), None, None, nat.ACT_NONE,
                                          self.y.data_ptr(), self.scratch.data_ptr(), self.scratch.numel(),
                                          torch.cuda.current_stream().cuda_stream)

    def pack(self, packed):
        nat.check(nat.load().fdnn_conv2d_pack_weight(ctypes.byref(self.d), self.w.data_ptr(), self.y.data_ptr(), packed.data_ptr(),
                                                     packed.numel(), torch.cuda.current_stream().cuda_stream))
        return packed

    def check(self, residual=None):
        want = torch.nn.functional.conv2d(self.x.double(), self.w.double(), None, self.stride, self.pad, 1, self.groups)
        if residual is not None:
            want = want + residual.double()
        eps = EPS[self.x.dtype]
        torch.testing.assert_close(self.y.double(), want, rtol=eps, atol=eps * want.abs().max().item())


LAYERS = {
    "in_the_relayout": dict(dtype=F16, n=4, c=64, h=20, w=22, k=96, r=3, s=3),
    "in_the_relayout_f32": dict(dtype=F32, n=4, c=64, h=20, w=22, k=96, r=3, s=3),
    "in_the_relayout_odd_rows": dict(dtype=BF16, n=3, c=40, h=17, w=19, k=72, r=5, s=5),
    "in_the_relayout_1x1": dict(dtype=F16, n=3, c=300, h=15, w=16, k=130, r=1, s=1),
    "by_itself": dict(dtype=BF16, n=4, c=20, h=30, w=30, k=64, r=3, s=3, x_format="nhwc"),
    "by_itself_f32": dict(dtype=F32, n=4, c=24, h=30, w=30, k=64, r=3, s=3, x_format="nhwc"),
    "k_contiguous": dict(dtype=BF16, n=1, c=264, h=1, w=500, k=133, r=1, s=1, x_format="nhwc", w_format="ck"),
    "windows": dict(dtype=BF16, n=8, c=3, h=64, w=64, k=32, r=7, s=7, stride=2),
    "quads": dict(dtype=BF16, n=8, c=3, h=64, w=64, k=32, r=7, s=7, stride=2, x_format="nhwc"),
    "quads_pairs": dict(dtype=F16, n=32, c=3, h=112, w=112, k=64, r=7, s=7, stride=2, x_format="nhwc"),
    "pixel_groups": dict(dtype=BF16, n=20, c=64, h=56, w=56, k=64, r=3, s=3, stride=1, x_format="nhwc"),
    "pixel_groups_stride_2": dict(dtype=BF16, n=60, c=32, h=112, w=112, k=64, r=3, s=3, stride=2, x_format="nhwc"),
    "two_groups": dict(dtype=BF16, n=9, c=64, h=14, w=14, k=128, r=3, s=3, groups=2, x_format="nhwc"),
    "three_groups": dict(dtype=BF16, n=9, c=120, h=24, w=24, k=120, r=3, s=3, groups=3),
    "many_groups": dict(dtype=F16, n=3, c=768, h=21, w=21, k=1536, r=3, s=3, groups=32),
    "small": dict(dtype=F16, n=1, c=64, h=14, w=14, k=64, r=3, s=3),
}


@pytest.mark.parametrize("name", LAYERS)
def test_the_buffer_serves_later_calls(native_lib, name):
    layer = Layer(**LAYERS[name])
    assert layer.plan.w_packed == 1
    packed = layer.buffer()
    nat.check(layer.unpacked(packed))
    layer.check()
    assert torch.equal(packed, layer.pack(layer.buffer()))
    nat.check(layer.packed_call(packed))
    layer.check()
    assert device_status() == 0


def test_a_small_layer_without_scratch_packs_too(native_lib):
    """Without scratch the direct kernel computes the layer, from w itself."""
    layer = Layer(**LAYERS["small"])
    packed = layer.buffer()
    nat.check(layer.unpacked(packed, scratch=False))
    layer.check()
    assert torch.equal(packed, layer.pack(layer.buffer()))
    nat.check(layer.packed_call(packed))
    layer.check()


def test_few_channels_with_a_residual_pack_too(native_lib):
    layer = Layer(F16, 2, 3, 24, 24, 16, 5, 5)
    assert layer.plan.w_packed == 1 and layer.plan.algo != nat.ALGO_DIRECT
    packed, residual = layer.buffer(), torch.randn_like(layer.y)
    nat.check(layer.unpacked(packed, residual=residual))
    layer.check(residual)
    assert torch.equal(packed, layer.pack(layer.buffer()))
    nat.check(layer.packed_call(packed))
    layer.check()


def test_what_is_refused(native_lib):
    layer = Layer(**LAYERS["in_the_relayout"])
    packed = layer.buffer()
    assert layer.unpacked(None) == nat.FDNN_BAD_PARAM
    assert layer.unpacked(packed, nbytes=packed.numel() - 1) == nat.FDNN_WORKSPACE_TOO_SMALL
    assert layer.unpacked(packed.data_ptr() + 8) == nat.FDNN_BAD_PARAM
    torch.cuda.synchronize()
    assert bool((packed == 0x2A).all()) and bool((layer.y == -7.0).all())
    small = Layer(**LAYERS["small"])         # the direct kernel needs no buffer, and none is written off its boundary
    packed = torch.full((small.plan.packed_weight_bytes + 16,), 0x2A, dtype=torch.uint8, device="cuda")
    nat.check(small.unpacked(packed.data_ptr() + 8, scratch=False))
    small.check()
    assert bool((packed == 0x2A).all())


def test_the_record_follows_what_the_buffer_holds(native_lib):
    """Two layers of one packed size: a buffer serves the one that was packed into it last, and a call that was refused
    leaves it as it was."""
    a, b = Layer(F16, 3, 40, 20, 20, 64, 3, 3), Layer(F16, 3, 64, 20, 20, 64, 3, 3)
    assert a.plan.packed_weight_bytes == b.plan.packed_weight_bytes
    packed = a.pack(a.buffer())
    assert b.unpacked(packed, act=9) == nat.FDNN_BAD_PARAM
    nat.check(a.packed_call(packed))
    a.check()
    nat.check(b.unpacked(packed))
    b.check()
    nat.check(b.packed_call(packed))
    b.check()
    assert a.packed_call(packed) == nat.FDNN_BAD_PARAM
    assert b"pack again" in native_lib.fdnn_last_error()
    assert a.unpacked(packed, scratch=False) == nat.FDNN_WORKSPACE_TOO_SMALL
    nat.check(b.packed_call(packed))
    b.check()


@pytest.mark.parametrize("name", LAYERS)
def test_a_buffer_inside_the_workspace_is_scratch(native_lib, name):
    """Nothing is remembered of it: afterwards it may hold any layer's packed filter."""
    layer, other = Layer(**LAYERS[name]), Layer(BF16, 3, 64, 20, 20, 64, 3, 3)
    begin, nbytes = -(-layer.plan.workspace_bytes // 256) * 256, layer.plan.packed_weight_bytes
    arena = torch.full((begin + max(nbytes, other.plan.packed_weight_bytes) + 256,), 0x2A, dtype=torch.uint8, device="cuda")
    layer.scratch = arena[:begin + nbytes]
    region = arena[begin:begin + other.plan.packed_weight_bytes]
    other.pack(region)     # whatever lay at this address before is forgotten
    arena.fill_(0x2A)
    nat.check(layer.unpacked(arena.data_ptr() + begin))
    layer.check()
    assert bool((arena[begin + nbytes:] == 0x2A).all())
    region.copy_(other.pack(other.buffer()))
    nat.check(other.packed_call(region))
    other.check()


def test_calls_that_pack_on_the_way_leave_the_records_alone(native_lib):
    """More of them than there are records, each with scratch of its own: a buffer packed for another layer is refused still."""
    import flagdnn_b200 as fd

    a, b = Layer(F16, 3, 40, 20, 20, 64, 3, 3), Layer(F16, 3, 64, 20, 20, 64, 3, 3)
    packed = a.pack(a.buffer())
    x, w = torch.randn(1, 64, 50, device="cuda").half(), torch.randn(64, 64, 3, device="cuda").half()
    x2, w2 = torch.randn(1, 64, 14, 14, device="cuda").half(), torch.randn(64, 64, 3, 3, device="cuda").half()
    held = []
    gc.collect()     # what other tests left for it is not freed in between
    for _ in range(300):
        before = torch.cuda.memory_allocated()
        fd.conv1d(x, w, padding=1)
        fd.conv2d(x2, w2, padding=1)
        assert torch.cuda.memory_allocated() == before
        held.append([torch.empty(n, dtype=torch.uint8, device="cuda") for n in (32 << 10, 128 << 10)])   # where the scratch was
    assert b.packed_call(packed) == nat.FDNN_BAD_PARAM
    nat.check(a.packed_call(packed))
    a.check()
