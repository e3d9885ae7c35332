"""Shifted windows whose masked scores decide: queries and keys of different regions score higher than the others by about the mask's 100, so
that what the mask leaves of them is a probability like any other. The bias table's gradient shows it, whose terms are kept in fp32.

Bound: scores meet the mask's 100 * log2(e) = 144 in fp32, one rounding within 2^-17, rms 2^-17 / sqrt(3) of the base-2 score and 3.1e-6 of the
masked probability; the other terms of the gradient's norm leave 1.4e-6 to 2.0e-6 of it. (Products summed at the mask's magnitude, which
rounds every 16 channels and towards zero: 5.2e-6.)"""
import pytest
import torch

pytestmark = pytest.mark.gpu
REL = 2.5e-6


@pytest.mark.parametrize("hd,heads,wh,ww", [(128, 2, 8, 8), (64, 2, 8, 8), (32, 4, 8, 8), (16, 4, 8, 12), (32, 2, 8, 12), (32, 3, 7, 7), (32, 4, 4, 8)])
def test_table_gradient(hd, heads, wh, ww):
    from terra_b200.ops.attention import WindowGeometry, shifted_window_sources, window_attention, window_attention_reference

    gen = torch.Generator(device="cuda").manual_seed(hd + wh)
    B, N, C, scale = 256, wh * ww, hd * heads, hd ** -0.5
    geo = WindowGeometry(B, 1, 1, wh, ww)
    _, token, region = (v.cuda().reshape(-1) for v in shifted_window_sources(geo, True))
    side = 1.0 - 2.0 * (region % 2)                                     # (regions 0 to 3 of the one window)
    apart = (100.0 / scale / hd / 2) ** 0.5                             # q.k across sides is higher by 100 over the scale
    q, k, v = (torch.randn(B, N, heads, hd, generator=gen, device="cuda") for _ in range(3))
    q, k = 0.3 * q - apart * side[:, None, None], 0.3 * k + apart * side[:, None, None]
    qkv = torch.empty(B, N, 3 * C, device="cuda", dtype=torch.bfloat16)
    qkv[:, token] = torch.stack((q, k, v), 2).reshape(B, N, 3 * C).to(torch.bfloat16)
    dout = torch.randn(B * N, C, generator=gen, device="cuda").to(torch.bfloat16)
    table = torch.zeros((2 * wh - 1) * (2 * ww - 1), heads, device="cuda", requires_grad=True)
    window_attention(qkv.view(B * N, 3 * C).requires_grad_(True), geo, heads, True, table, True, scale).backward(dout)
    want = torch.zeros_like(table, dtype=torch.float64, requires_grad=True)
    window_attention_reference(qkv.detach().double().view(B, 1, N, -1), geo, heads, True, want, True, scale).backward(dout.double().view(B, 1, N, C))
    rel = ((table.grad.double() - want.grad).norm() / want.grad.norm()).item()
    assert rel < REL, rel
