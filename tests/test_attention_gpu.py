"""Fused attention against plain attention in float64 on the same bf16 inputs, and against the score-matrix path (batched
GEMM, softmax pass, transposes, batched GEMM) to the last bit.

Bounds against float64: the output, the scores, and the probabilities before the second product are rounded to bf16
(relative 2^-9 each; scores of a few units turn theirs into 2^-8 of a probability), averaging over the keys: 1e-2. A
gradient passes one more such rounding (dP) on terms that partly cancel in dP - dot: 2e-2."""
import ctypes as C

import pytest
import torch

from sirius_b200 import ops
from sirius_b200._lib import call
from sirius_b200.gpt2_step import AttentionShapeC, BgemmDescC

pytestmark = pytest.mark.gpu
P = lambda t, off=0: C.c_void_p(t.data_ptr() + 2 * off)
rel = lambda a, b: float((a.double() - b).norm() / b.norm())
D = 64


def by_score_matrix(qkv, do, B, S, H, scale):
    """out, dq, dk, dv through srt_bgemm, srt_causal_softmax_* and srt_batched_transpose, one KV head per query head."""
    c, ld, SS = H * D, 3 * H * D, S * S
    new = lambda *s: torch.zeros(*s, device="cuda", dtype=torch.bfloat16)
    prob, dp, big, t = new(B * H, S, S), new(B * H, S, S), new(B * H, S, S), new(B * H, D, S)
    out, dqkv = new(B * S, c), new(B * S, ld)
    gemm = lambda d, a, b, o: call("srt_bgemm", C.byref(BgemmDescC(*d)), a, b, o, None)
    heads = (S, H * S)
    scores = (S, S, D, H, B, ld, D, S * ld, ld, D, S * ld, S, SS, H * SS, scale, 1, 0)
    gemm(scores, P(qkv), P(qkv, c), P(prob))
    call("srt_causal_softmax_fwd", P(prob), B * H, S, None)
    turn = lambda src, off, l: call("srt_batched_transpose", P(src, off), P(t), S, D, l, D, S * l, H, B, None)
    product = lambda l, alpha, kc: (S, D, S, H, B, S, SS, H * SS, S, D * S, H * D * S, l, D, S * l, alpha, 0, kc)
    turn(qkv, 2 * c, ld)
    gemm(product(c, 1.0, 1), P(prob), P(t), P(out))
    gemm((S, S, D, H, B, c, D, S * c, ld, D, S * ld, S, SS, H * SS, 1.0, 1, 0), P(do), P(qkv, 2 * c), P(dp))
    turn(do, 0, c)
    call("srt_batched_transpose", P(prob), P(big), S, S, S, SS, H * SS, H, B, None)
    gemm(product(ld, 1.0, 2), P(big), P(t), P(dqkv, 2 * c))
    call("srt_causal_softmax_bwd", P(prob), P(dp), B * H, S, None)
    turn(qkv, c, ld)
    gemm(product(ld, scale, 1), P(dp), P(t), P(dqkv))
    turn(qkv, 0, ld)
    call("srt_batched_transpose", P(dp), P(big), S, S, S, SS, H * SS, H, B, None)
    gemm(product(ld, scale, 2), P(big), P(t), P(dqkv, c))
    return out, dqkv


# eight positions (the shortest length there is), a tile's edges and remainders, several tiles with a ragged last one; grouped and plain heads
@pytest.mark.parametrize("B,S,H,Hkv,gain", [(1, 8, 1, 1, 1.0), (2, 72, 3, 3, 1.0), (1, 128, 2, 1, 1.0), (2, 136, 4, 2, 1.0),
                                            (1, 328, 7, 1, 1.0), (2, 640, 2, 2, 4.0), (1, 1024, 3, 3, 1.0)])
@pytest.mark.parametrize("causal", [1, 0])
def test_attention_forward_backward(B, S, H, Hkv, gain, causal):
    T, scale = B * S, 0.125
    ld = (H + 2 * Hkv) * D
    g = torch.Generator(device="cuda").manual_seed(S)
    qkv = torch.randn(T, ld, device="cuda", generator=g)
    qkv[:, :H * D] *= gain   # a large gain makes the rows nearly one-hot
    qkv = qkv.to(torch.bfloat16)
    do = torch.randn(T, H * D, device="cuda", generator=g).to(torch.bfloat16)
    x = qkv.double().requires_grad_(True)
    q, k, v = (t.reshape(B, S, n, D).transpose(1, 2) for t, n in zip(x.split([H * D, Hkv * D, Hkv * D], 1), (H, Hkv, Hkv)))
    k, v = k.repeat_interleave(H // Hkv, 1), v.repeat_interleave(H // Hkv, 1)
    s = q @ k.transpose(-1, -2) * scale
    if causal:
        s = s.masked_fill(torch.triu(torch.ones(S, S, device="cuda", dtype=torch.bool), 1), float("-inf"))
    ref = (torch.softmax(s, -1) @ v).transpose(1, 2).reshape(T, H * D)

    shape = AttentionShapeC(B, S, H, Hkv, D)
    sp = (S + 127) // 128 * 128
    o = torch.full((T, H * D), float("nan"), device="cuda", dtype=torch.bfloat16)
    rows = torch.full((3, B * H, sp), float("nan"), device="cuda")
    call("srt_attention_fwd", C.byref(shape), P(qkv), P(qkv, H * D), P(qkv, (H + Hkv) * D), ld, P(o), H * D, P(rows), scale,
         causal, None)
    torch.cuda.synchronize()
    assert ops.tc_status() == 0
    assert rel(o, ref.detach()) < 1e-2 * gain
    if not causal:
        return
    ref.backward(do.double())
    dqkv = torch.full((T, ld), float("nan"), device="cuda", dtype=torch.bfloat16)
    dk, dv = (torch.full((B, H, S, D), float("nan"), device="cuda", dtype=torch.bfloat16) for _ in range(2))
    call("srt_attention_bwd_causal", C.byref(shape), P(qkv), P(qkv, H * D), P(qkv, (H + Hkv) * D), ld, P(do), H * D, P(rows),
         P(dqkv), ld, P(dk), P(dv), D, S * D, H * S * D, scale, None)
    torch.cuda.synchronize()
    assert ops.tc_status() == 0
    group = lambda t: t.float().view(B, Hkv, H // Hkv, S, D).sum(2).transpose(1, 2).reshape(T, Hkv * D)
    gq, gk, gv = x.grad.split([H * D, Hkv * D, Hkv * D], 1)
    for name, got, want in (("dq", dqkv[:, :H * D], gq), ("dk", group(dk), gk), ("dv", group(dv), gv)):
        # a short row has next to no gradient through its softmax: compare against the size of the other gradients
        assert float((got.double() - want).norm()) < 2e-2 * gain * max(float(want.norm()), 0.1 * float(gv.norm())), name
    if H != Hkv:
        return
    out2, dqkv2 = by_score_matrix(qkv, do, B, S, H, scale)
    torch.cuda.synchronize()
    assert ops.tc_status() == 0
    flat = lambda t: t.transpose(1, 2).reshape(T, H * D)
    assert torch.equal(o, out2)
    assert torch.equal(dqkv[:, :H * D], dqkv2[:, :H * D])
    assert torch.equal(flat(dk), dqkv2[:, H * D:2 * H * D])
    assert torch.equal(flat(dv), dqkv2[:, 2 * H * D:])
