"""Products on CTA pairs whose second operand lies row-major, [C][K]: it is read in place."""
import ctypes

import pytest
import torch

from flagdnn_b200 import _native as nat, device_status

pytestmark = pytest.mark.gpu

CODE = {torch.float16: nat.F16, torch.bfloat16: nat.BF16}
EPS = {torch.bfloat16: 2.0 ** -8, torch.float16: 2.0 ** -11}

# m, c, k: a pair takes 256 rows x 256 columns, a CTA 128 of the columns as two boxes of 64
PRODUCTS = {
    "aligned": (4096, 2048, 1024),
    "ragged_reduction": (4096, 2056, 1000),      # the last step holds 8 of 64 channels, the last tile 232 columns
    "eight_columns_left": (19000, 1032, 264),    # the second column tile: 8 columns, the partner's boxes lie past the filter
    "second_box": (19000, 1032, 328),            # 72 columns: a box and an eighth of one
    "partner_columns": (19000, 1032, 392),       # 136 columns
    "one_column_tile": (9473, 2048, 256),        # 38 tiles on 74 pairs, the last one of a single row
}


def describe(dtype, m, c, k, b, algo=0):
    d = nat.ConvDesc()
    d.dtype, d.n, d.c, d.h, d.w, d.k, d.r, d.s, d.groups = CODE[dtype], 1, c, 1, m, k, 1, 1, 1
    d.stride_h = d.stride_w = d.dil_h = d.dil_w = 1
    d.algo = algo
    for i, (x_s, w_s, y_s) in enumerate(zip((m * c, 1, m * c, c), (b.stride(1), b.stride(0), 1, 1), (m * k, 1, m * k, k))):
        d.x_strides[i], d.w_strides[i], d.y_strides[i] = x_s, w_s, y_s
    return d


def operands(dtype, m, c, k, pitch):
    g = torch.Generator().manual_seed(m + c + k)
    a = torch.randn(m, c, generator=g).to(dtype).cuda()
    # what lies between the rows of b must not be read as part of it
    b = torch.full((c, pitch), float("nan"), dtype=dtype, device="cuda")[:, :k]
    b.copy_((torch.randn(c, k, generator=g) * c ** -0.5).to(dtype))
    return a, b


def check(y, a, b):
    """One rounding to the type; the fp32 sums of two thousand products are far below it."""
    want = a.double() @ b.double()
    eps = EPS[y.dtype]
    torch.testing.assert_close(y.double(), want, rtol=eps, atol=eps * want.abs().max().item())


@pytest.mark.parametrize("gap", [0, 72], ids=["dense", "pitched"])
@pytest.mark.parametrize("dtype", list(EPS), ids=["bf16", "f16"])
@pytest.mark.parametrize("name", PRODUCTS)
def test_second_operand_in_place(native_lib, name, dtype, gap):
    """Against fp64, and bit for bit against the same kernel on a transposed copy, which has the same order of sums."""
    m, c, k = PRODUCTS[name]
    a, b = operands(dtype, m, c, k, k + gap)
    y = torch.empty(m, k, dtype=dtype, device="cuda")
    stream = torch.cuda.current_stream().cuda_stream

    def run(algo):
        d, plan = describe(dtype, m, c, k, b, algo), nat.ConvPlan()
        nat.check(native_lib.fdnn_conv2d_query(ctypes.byref(d), a.data_ptr(), b.data_ptr(), y.data_ptr(), ctypes.byref(plan)))
        packed = None
        if plan.w_packed:
            packed = torch.empty(plan.packed_weight_bytes, dtype=torch.uint8, device="cuda")
            nat.check(native_lib.fdnn_conv2d_pack_weight(ctypes.byref(d), b.data_ptr(), y.data_ptr(), packed.data_ptr(),
                                                         packed.numel(), stream))
        y.fill_(-7.0)
        nat.check(native_lib.fdnn_conv2d_fwd(ctypes.byref(d), a.data_ptr(), b.data_ptr(), None if packed is None else packed.data_ptr(),
                                             None, None, nat.ACT_NONE, y.data_ptr(), None, 0, stream))
        assert device_status() == 0
        return plan, y.clone()

    plan, in_place = run(nat.ALGO_AUTO)
    assert (plan.algo, plan.w_packed, plan.x_repacked) == (nat.ALGO_IGEMM_PAIR, 0, 0)
    check(in_place, a, b)
    plan, copied = run(nat.ALGO_IGEMM_PAIR)
    assert (plan.algo, plan.w_packed) == (nat.ALGO_IGEMM_PAIR, 1)
    assert torch.equal(in_place, copied)


@pytest.mark.parametrize("dtype", list(EPS), ids=["bf16", "f16"])
def test_second_operand_in_place_with_split_reductions(native_lib, dtype):
    m, c, k = 6400, 2056, 1000     # 100 tiles on 74 pairs: the first steps of a tile may begin anywhere in the reduction
    a, b = operands(dtype, m, c, k, k)
    y = torch.full((m, k), -7.0, dtype=dtype, device="cuda")
    d, plan = describe(dtype, m, c, k, b, nat.ALGO_FLAG_STREAM_K), nat.ConvPlan()
    nat.check(native_lib.fdnn_conv2d_query(ctypes.byref(d), a.data_ptr(), b.data_ptr(), y.data_ptr(), ctypes.byref(plan)))
    assert (plan.algo, plan.w_packed, plan.stream_k) == (nat.ALGO_IGEMM_PAIR, 0, 1)
    scratch = torch.zeros(plan.streamk_bytes, dtype=torch.uint8, device="cuda")
    nat.check(native_lib.fdnn_conv2d_fwd_ex(ctypes.byref(d), a.data_ptr(), b.data_ptr(), None, None, None, None, nat.ACT_NONE,
                                            y.data_ptr(), None, 0, scratch.data_ptr(), scratch.numel(),
                                            torch.cuda.current_stream().cuda_stream))
    assert device_status() == 0
    assert not bool(scratch[:nat.STREAMK_FLAG_BYTES].any())
    check(y, a, b)
