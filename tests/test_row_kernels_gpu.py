"""LayerNorm and AdamW kernels at the edges of their variants, against float64.

Bounds: LayerNorm writes bf16 (relative 2^-9 of every output, 2^-8 of the gradient's largest terms, which cancel); its
parameter gradients and AdamW are fp32 sums and products of a few dozen roundings (1e-5)."""
import ctypes as C

import pytest
import torch

from sirius_b200 import gpt2_step  # noqa: F401  (registers the signatures)
from sirius_b200._lib import call, lib

pytestmark = pytest.mark.gpu
P = lambda t: C.c_void_p(t.data_ptr())
rel = lambda a, b: float((a.double() - b).norm() / b.norm().clamp_min(1e-30))


# columns: below, at and above a lane's vector counts (1, 2, 3, 4, 8) and beyond the register form; rows: one, a partly
# filled block, more than the two-warp blocks serve; shifted parameters are not 16-byte aligned
@pytest.mark.parametrize("cols", [8, 256, 264, 768, 1024, 1032, 2048, 2056])
@pytest.mark.parametrize("rows,shift", [(1, 0), (13, 1), (1300, 0)])
def test_layernorm_variants(rows, cols, shift):
    g = torch.Generator(device="cuda").manual_seed(rows + cols)
    new = lambda *s: torch.randn(*s, device="cuda", generator=g)
    x, dy, add = (new(rows, cols).bfloat16() for _ in range(3))
    gamma, beta = (new(cols + shift)[shift:] for _ in range(2))
    y, dx = torch.empty_like(x), torch.empty_like(x)
    mean, rstd, dg, db = (torch.empty(n, device="cuda") for n in (rows, rows, cols, cols))
    lib().srt_layernorm_bwd_scratch_bytes.restype = C.c_size_t
    n = lib().srt_layernorm_bwd_scratch_bytes(cols)
    scratch = torch.empty(n, dtype=torch.uint8, device="cuda")
    torch.cuda.synchronize()
    call("srt_layernorm_fwd", P(x), P(gamma), P(beta), P(y), P(mean), P(rstd), rows, cols, 1e-5, None)
    call("srt_layernorm_bwd", P(dy), P(x), P(gamma), P(mean), P(rstd), P(add), P(dx), P(dg), P(db), rows, cols, P(scratch), n, None)
    torch.cuda.synchronize()
    xd, gd, bd = (t.double().detach().requires_grad_(True) for t in (x, gamma, beta))
    ref = torch.nn.functional.layer_norm(xd, (cols,), gd, bd, 1e-5)
    ref.backward(dy.double())
    assert rel(y, ref.detach()) < 4e-3
    assert rel(dx, xd.grad + add.double()) < 8e-3
    assert rel(dg, gd.grad) < 1e-5 and rel(db, bd.grad) < 1e-5


@pytest.mark.parametrize("n", [1, 4, 7, 4099, 3_000_001])
@pytest.mark.parametrize("shift", [0, 1])
def test_adamw_tails_and_alignment(n, shift):
    g = torch.Generator(device="cuda").manual_seed(n)
    new = lambda: torch.randn(n + shift, device="cuda", generator=g)[shift:]
    p, gr, m, v = new(), new(), new(), new().abs()
    pb = torch.empty(n + shift, device="cuda", dtype=torch.bfloat16)[shift:]
    lr, b1, b2, eps, wd, step = 0.1, 0.9, 0.999, 1e-8, 0.01, 3
    pd, gd, md, vd = (t.double() for t in (p, gr, m, v))
    torch.cuda.synchronize()
    call("srt_adamw", P(p), P(gr), P(m), P(v), P(pb), n, lr, b1, b2, eps, wd, step, None)
    torch.cuda.synchronize()
    md = b1 * md + (1 - b1) * gd
    vd = b2 * vd + (1 - b2) * gd * gd
    want = pd * (1 - lr * wd) - lr / (1 - b1 ** step) * md / (vd.sqrt() / (1 - b2 ** step) ** 0.5 + eps)
    assert rel(m, md) < 1e-5 and rel(v, vd) < 1e-5 and rel(p, want) < 1e-4   # 1 - b2^3 in fp32 keeps five digits
    assert torch.equal(pb, p.bfloat16())
