"""Further forms of the data gradient on the filter itself, against the one on its transposed copy, to the last bit: an addend
under mask bits (whole words of the mask and single bytes), and the first operand gathered by threads instead of by TMA."""
import ctypes as C

import pytest
import torch

from sirius_b200 import _lib, ops
from sirius_b200._lib import ConvEpilogue, call

pytestmark = pytest.mark.gpu
P = lambda t: C.c_void_p(t.data_ptr() if t is not None else 0)
BF16 = 1


# N, H, W, C, K, R, pad: C a multiple of 64 (the mask is read by words) and not; 3x3 and 1x1; ragged rows
@pytest.mark.parametrize("shape", [(2, 14, 14, 256, 64, 1, 0), (3, 9, 7, 72, 128, 1, 0), (2, 9, 11, 64, 64, 3, 1), (1, 13, 13, 200, 128, 3, 1),
                                   (4, 14, 14, 1024, 2048, 1, 0)])
@pytest.mark.parametrize("gather", [0, 1])
@pytest.mark.parametrize("bits", [False, True])
def test_direct_equals_transposed(shape, gather, bits):
    N, H, W, Ci, K, R, pad = shape
    d = _lib.ConvDesc.make(N, H, W, Ci, K, R, R, 1, pad)
    g = torch.Generator(device="cuda").manual_seed(Ci + K + R)
    new = lambda *s: torch.randn(*s, device="cuda", generator=g).bfloat16()
    dy, w, add = new(N, d.P, d.Q, K), new(K, R, R, Ci), new(N, H, W, Ci)
    mask = torch.randint(0, 256, (N * H * W * Ci // 8,), device="cuda", generator=g, dtype=torch.uint8) if bits else None
    wt = torch.empty(Ci, R, R, K, device="cuda", dtype=torch.bfloat16)
    a, b = (torch.full((N, H, W, Ci), float("nan"), device="cuda", dtype=torch.bfloat16) for _ in range(2))
    ep = ConvEpilogue(None, add.data_ptr(), mask.data_ptr() if bits else None)
    torch.cuda.synchronize()
    call("srt_conv_plan_override", gather, 0, -1)
    try:
        call("srt_conv_filter_transpose", C.byref(d), BF16, P(w), P(wt), None)
        call("srt_conv_dgrad", C.byref(d), BF16, 0, P(dy), P(wt), P(a), C.byref(ep), None)
        call("srt_conv_dgrad_direct", C.byref(d), BF16, 0, P(dy), P(w), P(b), C.byref(ep), None)
        torch.cuda.synchronize()
    finally:
        call("srt_conv_plan_override", 0, 0, -1)
    assert ops.tc_status() == 0
    assert torch.isfinite(a.float()).all() and torch.equal(a, b)
    if bits:                                            # the mask does what it says
        keep = ((mask.view(-1, 1).int() >> torch.arange(8, device="cuda")) & 1).view(N, H, W, Ci).bool()
        ref = torch.nn.functional.conv_transpose2d(dy.double().permute(0, 3, 1, 2), w.double().permute(0, 3, 1, 2), padding=pad)
        ref = ref.permute(0, 2, 3, 1) + torch.where(keep, add.double(), 0.0)
        assert float((b.double() - ref).norm() / ref.norm()) < 4e-3      # one rounding to bf16
