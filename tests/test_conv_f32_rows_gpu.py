"""fp32 convolutions with more row tiles than the y and z dimensions of a grid hold (65 535 tiles of 128 output positions), in
inference with its epilogue and in the training form, against float64. 8-term products and a three-term epilogue: within 1e-6
in the 2-norm, 1e-5 of the root mean square for single values (about ten roundings of 2^-24 each, on partial sums of at most
ten times the root mean square)."""
import ctypes as C

import pytest
import torch

from sirius_b200 import _lib
from sirius_b200._lib import ConvEpilogue, call

pytestmark = pytest.mark.gpu
P = lambda t: C.c_void_p(t.data_ptr() if t is not None else 0)
F32, RELU, NONE = 0, 1, 0
LIMIT = 65535 * 128


@pytest.mark.parametrize("rows", [LIMIT, LIMIT + 1, LIMIT + 128 * 3 + 77])
@pytest.mark.parametrize("form", ["infer", "infer_bn_add_relu", "fprop_bias", "dgrad"])
def test_rows_beyond_a_grid_dimension(rows, form):
    ci = k = 8
    d = _lib.ConvDesc.make(1, 1, rows, ci, k, 1, 1, 1, 0)
    g = torch.Generator(device="cuda").manual_seed(rows % 1000)
    new = lambda *s: torch.randn(*s, device="cuda", generator=g)
    x, w = new(rows, ci), new(k, ci)
    add, scale, shift = new(rows, k), new(k), new(k)
    y = torch.full((rows, k), float("nan"), device="cuda")
    torch.cuda.synchronize()
    if form == "infer":
        call("srt_conv_fprop_infer", C.byref(d), F32, 0, P(x), P(w), P(y), P(None), P(None), P(None), NONE, None)
        ref = x.double() @ w.double().t()
    elif form == "infer_bn_add_relu":
        call("srt_conv_fprop_infer", C.byref(d), F32, 0, P(x), P(w), P(y), P(scale), P(shift), P(add), RELU, None)
        ref = (x.double() @ w.double().t() * scale.double() + shift.double() + add.double()).clamp_min(0)
    elif form == "fprop_bias":
        ep = ConvEpilogue(shift.data_ptr(), add.data_ptr(), None)
        call("srt_conv_fprop", C.byref(d), F32, 0, P(x), P(w), P(y), C.byref(ep), None)
        ref = x.double() @ w.double().t() + shift.double() + add.double()
    else:
        call("srt_conv_dgrad", C.byref(d), F32, 0, P(x), P(w), P(y), None, None)   # w here is the transposed filter [C][K]
        ref = x.double() @ w.double().t()
    torch.cuda.synchronize()
    diff = (y.double() - ref).abs()
    assert float((y.double() - ref).norm() / ref.norm()) < 1e-6
    assert float(diff.max() / ref.pow(2).mean().sqrt()) < 1e-5
