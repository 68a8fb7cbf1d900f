"""Convolutions with the epilogue of inference against float64: the cluster-split and persistent tcgen05 kernels (bf16) and
the large-tile CUDA-core kernel (fp32), whole and split.

Bounds: bf16 outputs are rounded once (relative 2^-9 in the largest case, half that in the 2-norm); fp32 sums of up to
4608 products in any order stay within 2e-6 in the 2-norm."""
import ctypes as C

import pytest
import torch

from sirius_b200 import _lib, ops
from sirius_b200._lib import call

pytestmark = pytest.mark.gpu
P = lambda t: C.c_void_p(t.data_ptr() if t is not None else 0)
F32, BF16 = 0, 1

# N, H, W, C, K, R, stride, pad: one tile and one k-block; ragged rows and columns; plain and im2col operands; every cluster
# size; strided; a stem whose channels are gathered; more tiles than SMs
SHAPES = [(1, 1, 1, 64, 8, 1, 1, 0), (1, 1, 128, 768, 768, 1, 1, 0), (1, 14, 14, 256, 256, 3, 1, 1), (3, 7, 7, 512, 512, 3, 1, 1),
          (1, 28, 28, 256, 512, 1, 2, 0), (5, 9, 11, 128, 72, 3, 2, 1), (1, 1, 77, 3072, 200, 1, 1, 0), (1, 30, 30, 8, 64, 7, 2, 3),
          (2, 56, 56, 64, 256, 1, 1, 0), (1, 1, 1000, 200, 1000, 1, 1, 0)]


@pytest.mark.parametrize("shape", SHAPES)
@pytest.mark.parametrize("dtype", [BF16, F32])
@pytest.mark.parametrize("form", ["plain", "bn_add_relu", "bias_gelu"])
def test_conv_infer(shape, dtype, form):
    N, H, W, Ci, K, R, stride, pad = shape
    if form == "bias_gelu" and dtype == F32:
        return
    d = _lib.ConvDesc.make(N, H, W, Ci, K, R, R, stride, pad)
    g = torch.Generator(device="cuda").manual_seed(Ci + K)
    new = lambda *s: torch.randn(*s, device="cuda", generator=g)
    t = torch.bfloat16 if dtype == BF16 else torch.float32
    x, w = new(N, H, W, Ci).to(t), (new(K, R, R, Ci) * (R * R * Ci) ** -0.5).to(t)
    add = new(N, d.P, d.Q, K).to(t) if form == "bn_add_relu" else None
    scale = new(K) if form == "bn_add_relu" else None
    shift = new(K) if form != "plain" else None
    y = torch.full((N, d.P, d.Q, K), float("nan"), device="cuda", dtype=t)
    torch.cuda.synchronize()
    call("srt_conv_fprop_infer", C.byref(d), dtype, 0, P(x), P(w), P(y), P(scale), P(shift), P(add),
         {"plain": 0, "bn_add_relu": 1, "bias_gelu": 2}[form], None)
    torch.cuda.synchronize()
    assert ops.tc_status() == 0
    ref = torch.nn.functional.conv2d(x.double().permute(0, 3, 1, 2), w.double().permute(0, 3, 1, 2), stride=stride, padding=pad)
    ref = ref.permute(0, 2, 3, 1)
    if scale is not None:
        ref = ref * scale.double()
    if shift is not None:
        ref = ref + shift.double()
    if add is not None:
        ref = (ref + add.double()).clamp_min(0)
    if form == "bias_gelu":
        ref = torch.nn.functional.gelu(ref)
    err = float((y.double() - ref).norm() / ref.norm())
    assert err < (4e-3 if dtype == BF16 else 2e-6), err
