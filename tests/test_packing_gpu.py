"""Filters packed tap by tap: every tap lands in its place whatever their number, and many taps cost what few do."""
import ctypes

import pytest
import torch

from flagdnn_b200 import _native as nat, device_status

pytestmark = pytest.mark.gpu

CODE = {torch.float16: nat.F16, torch.bfloat16: nat.BF16, torch.float32: nat.F32}


class Packing:
    def __init__(self, lib, dtype, k, c, r, s, strided=False):
        g = torch.Generator().manual_seed(k + c + r * s)
        self.lib, self.dtype = lib, dtype
        self.x = torch.randn(2, c, r + 6, s + 9, generator=g).to(dtype).cuda()
        self.w = torch.randn(k, c, r, s, generator=g).to(dtype).cuda()
        if strided:   # taps and channels apart
            self.w = torch.randn(k, c, r, s + 3, generator=g).to(dtype).cuda()[..., :s]
        self.y = torch.empty(2, k, 7, 10, dtype=dtype, device="cuda")
        d = self.d = nat.ConvDesc()
        d.dtype, d.n, d.c, d.h, d.w, d.k, d.r, d.s, d.groups = CODE[dtype], 2, c, r + 6, s + 9, k, r, s, 1
        d.stride_h = d.stride_w = d.dil_h = d.dil_w = 1
        d.algo = nat.ALGO_IGEMM | nat.ALGO_FLAG_NO_PIXEL_GROUP
        for i in range(4):
            d.x_strides[i], d.w_strides[i], d.y_strides[i] = self.x.stride(i), self.w.stride(i), self.y.stride(i)
        self.plan = nat.ConvPlan()
        nat.check(lib.fdnn_conv2d_query(ctypes.byref(d), self.x.data_ptr(), self.w.data_ptr(), self.y.data_ptr(), ctypes.byref(self.plan)))
        assert (self.plan.algo, self.plan.w_packed, self.plan.pixel_group, self.plan.low_channel) == (nat.ALGO_IGEMM, 1, 0, 0)
        self.packed = torch.full((self.plan.packed_weight_bytes,), 0x2A, dtype=torch.uint8, device="cuda")
        self.scratch = torch.empty(max(self.plan.workspace_bytes, 256), dtype=torch.uint8, device="cuda")
        self.stream = torch.cuda.current_stream().cuda_stream

    def pack(self):
        nat.check(self.lib.fdnn_conv2d_pack_weight(ctypes.byref(self.d), self.w.data_ptr(), self.y.data_ptr(), self.packed.data_ptr(),
                                                   self.packed.numel(), self.stream))

    def run(self):
        nat.check(self.lib.fdnn_conv2d_fwd_unpacked(
            ctypes.byref(self.d), self.x.data_ptr(), self.w.data_ptr(), self.packed.data_ptr(), self.packed.numel(), None, None, None,
            nat.ACT_NONE, self.y.data_ptr(), self.scratch.data_ptr(), self.scratch.numel(), self.stream))

    def check(self):
        """16-bit values are moved as they are; fp32 ones lie as two planes whose sum keeps 21 bits or more of the 24."""
        k, c, r, s = self.w.shape
        planes = 2 if self.dtype == torch.float32 else 1
        got = self.packed.view(self.dtype).view(planes, k, r, s, self.plan.c_padded)
        want = self.w.permute(0, 2, 3, 1)
        assert not bool(got[..., c:].any())
        if planes == 1:
            assert torch.equal(got[0, ..., :c], want)
        else:
            torch.testing.assert_close(got[..., :c].sum(0), want, rtol=2.0 ** -21, atol=0)


# taps around the ten that a thread takes
@pytest.mark.parametrize("dtype", list(CODE), ids=["f16", "bf16", "f32"])
@pytest.mark.parametrize("k,c,r,s,strided", [(24, 40, 3, 3, False), (24, 40, 2, 5, False), (24, 40, 1, 11, False), (9, 72, 4, 5, True),
                                             (16, 16, 3, 7, False), (40, 24, 5, 5, True), (8, 8, 1, 101, False), (16, 16, 31, 31, False),
                                             (130, 200, 1, 1, True)])
def test_every_tap_in_its_place(native_lib, k, c, r, s, strided, dtype):
    p = Packing(native_lib, dtype, k, c, r, s, strided)
    p.pack()
    p.check()
    p.packed.fill_(0x2A)
    p.run()       # by the launch that relays x out
    p.check()
    assert device_status() == 0


def test_many_taps_cost_what_few_do(native_lib):
    """The same 490 KB as 31 x 31 taps of 16 x 16 channels and as 3 x 3 of 166 x 164."""
    def microseconds(p):
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph):
            p.stream = torch.cuda.current_stream().cuda_stream
            for _ in range(20):
                p.pack()
        times = []
        for _ in range(7):
            a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            a.record()
            graph.replay()
            b.record()
            b.synchronize()
            times.append(a.elapsed_time(b) * 50)
        return sorted(times)[3]

    many, few = microseconds(Packing(native_lib, torch.bfloat16, 16, 16, 31, 31)), microseconds(Packing(native_lib, torch.bfloat16, 166, 164, 3, 3))
    assert many < 3 * few, (many, few)
