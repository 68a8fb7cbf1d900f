"""Shifted-window attention against float64 on the same bf16 inputs. Bounds as for the decoder attention: rounded scores,
probabilities and outputs keep the output within 1e-2 in the 2-norm, and one more rounding (dP) the gradients within 2e-2."""
import ctypes as C

import pytest
import torch

from sirius_b200 import swin_step  # noqa: F401  (registers the signatures)
from sirius_b200._lib import call

pytestmark = pytest.mark.gpu
P = lambda t: C.c_void_p(t.data_ptr())
rel = lambda a, b: float((a.double() - b).norm() / b.norm())
D = 32


# windows of one token, of 49 (padded rows and columns) and of a full tile; shifted maps where all masks occur
@pytest.mark.parametrize("B,Hs,Ws,WS,shift,heads", [(1, 7, 7, 7, 0, 1), (2, 14, 21, 7, 3, 4), (3, 14, 14, 7, 0, 2), (1, 16, 8, 8, 4, 3),
                                                    (2, 3, 3, 1, 0, 2), (1, 12, 12, 4, 1, 5)])
def test_window_attention(B, Hs, Ws, WS, shift, heads):
    L, T, scale = WS * WS, B * Hs * Ws, D ** -0.5
    ld = (L + 7) // 8 * 8
    g = torch.Generator(device="cuda").manual_seed(Hs * heads)
    qkv = torch.randn(T, 3, heads, D, device="cuda", generator=g).bfloat16()
    dout = torch.randn(T, heads, D, device="cuda", generator=g).bfloat16()
    table = torch.randn((2 * WS - 1) ** 2, heads, device="cuda", generator=g)
    out, dqkv = torch.full((T, heads, D), float("nan"), device="cuda", dtype=torch.bfloat16), torch.full_like(qkv, float("nan"))
    nw = (Hs // WS) * (Ws // WS)
    dS = torch.full((B * nw, heads, L, ld), float("nan"), device="cuda", dtype=torch.bfloat16)
    torch.cuda.synchronize()
    call("srt_window_attention_fwd", P(qkv), P(table), P(out), B, Hs, Ws, WS, shift, heads, D, scale, None)
    call("srt_window_attention_bwd", P(qkv), P(table), P(dout), P(dqkv), P(dS), ld, B, Hs, Ws, WS, shift, heads, D, scale, None)
    torch.cuda.synchronize()

    x, tb = qkv.double().requires_grad_(True), table.double().requires_grad_(True)

    def windows(t):   # [T][...] natural -> [B * windows][L][...]
        t = t.reshape(B, Hs, Ws, *t.shape[1:]).roll((-shift, -shift), (1, 2))
        t = t.reshape(B, Hs // WS, WS, Ws // WS, WS, *t.shape[3:]).transpose(2, 3)
        return t.reshape(B * nw, L, *t.shape[5:])

    q, k, v = (windows(x[:, i]).transpose(1, 2) for i in range(3))   # [W][heads][L][D]
    iy, ix = torch.arange(L, device="cuda") // WS, torch.arange(L, device="cuda") % WS
    index = (iy[:, None] - iy + WS - 1) * (2 * WS - 1) + ix[:, None] - ix + WS - 1
    s = q @ k.transpose(-1, -2) * scale + tb[index].permute(2, 0, 1)
    if shift:
        def part(n):
            p = torch.arange(n, device="cuda")
            return torch.where(p < n - WS, 0, torch.where(p < n - shift, 1, 2))
        region = (part(Hs)[:, None] * 3 + part(Ws)).reshape(Hs // WS, WS, Ws // WS, WS).transpose(1, 2).reshape(nw, L)
        s = s + torch.where(region[:, :, None] != region[:, None], -100.0, 0.0).repeat(B, 1, 1)[:, None]
    s.retain_grad()
    ref = (torch.softmax(s, -1) @ v).transpose(1, 2)
    ref.backward(windows(dout.double()))
    assert rel(windows(out), ref.detach()) < 1e-2
    for i in range(3):
        if L > 1 or i == 2:   # a window of one token has no gradient through its softmax
            assert rel(dqkv[:, i], x.grad[:, i]) < 2e-2, "qkv"[i]
    if L > 1:
        assert rel(dS[..., :L], s.grad) < 2e-2
    assert (dS[..., L:] == 0).all() and torch.isfinite(dqkv).all()
