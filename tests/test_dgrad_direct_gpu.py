"""Data gradient on the filter itself (MN-major operand) against the one on its transposed copy, to the last bit: both add the
same products in the same order."""
import ctypes as C

import pytest
import torch

from sirius_b200 import _lib, ops
from sirius_b200._lib import ConvEpilogue, call

pytestmark = pytest.mark.gpu
P = lambda t: C.c_void_p(t.data_ptr() if t is not None else 0)
BF16 = 1


# N, H, W, C, K, R, pad: ragged columns, rows and reduction; every tile width; filters wider than 1x1; CTA pairs (32 k-blocks)
@pytest.mark.parametrize("shape", [(1, 1, 5, 8, 8, 1, 0), (1, 1, 300, 72, 200, 1, 0), (2, 14, 14, 64, 256, 1, 0), (2, 9, 7, 64, 64, 3, 1),
                                   (3, 14, 14, 256, 128, 3, 1), (1, 1, 520, 200, 2048, 1, 0), (1, 1, 2000, 768, 3072, 1, 0),
                                   (1, 1, 640, 896, 4808, 1, 0), (4, 28, 28, 128, 512, 1, 0)])
@pytest.mark.parametrize("with_addend", [False, True])
def test_direct_equals_transposed(shape, with_addend):
    N, H, W, Ci, K, R, pad = shape
    d = _lib.ConvDesc.make(N, H, W, Ci, K, R, R, 1, pad)
    g = torch.Generator(device="cuda").manual_seed(Ci + K)
    new = lambda *s: torch.randn(*s, device="cuda", generator=g).bfloat16()
    dy, w = new(N, d.P, d.Q, K), new(K, R, R, Ci)
    add = new(N, H, W, Ci) if with_addend else None
    wt = torch.empty(Ci, R, R, K, device="cuda", dtype=torch.bfloat16)
    a, b = (torch.full((N, H, W, Ci), float("nan"), device="cuda", dtype=torch.bfloat16) for _ in range(2))
    ep = ConvEpilogue(None, add.data_ptr() if with_addend else None, None)
    torch.cuda.synchronize()
    call("srt_conv_filter_transpose", C.byref(d), BF16, P(w), P(wt), None)
    call("srt_conv_dgrad", C.byref(d), BF16, 0, P(dy), P(wt), P(a), C.byref(ep), None)
    call("srt_conv_dgrad_direct", C.byref(d), BF16, 0, P(dy), P(w), P(b), C.byref(ep), None)
    torch.cuda.synchronize()
    assert ops.tc_status() == 0
    assert torch.isfinite(a.float()).all() and torch.equal(a, b)
