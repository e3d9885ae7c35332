"""The shifted-window mask added through the products' accumulators: windows cut by the last row, the last column and both, odd sides, scales
that the mask is divided by (none at all, tiny, negative, large), windows padded to a block, no mask.

Bound: against fp32 the kernel rounds P, dS and the results to bf16 (2^-9 each, independent): 3 * 2^-9 = 0.6 % of the norm; 1 % allowed."""
import pytest
import torch

pytestmark = pytest.mark.gpu
REL = 1e-2


@pytest.mark.parametrize("nWh,nWw,wh,ww,hd,heads", [(2, 2, 8, 8, 32, 2), (3, 1, 8, 12, 16, 2), (1, 4, 7, 7, 32, 1), (2, 3, 4, 8, 64, 2), (2, 2, 5, 13, 16, 2)])
@pytest.mark.parametrize("scale", [0.0, 1e-4, -0.2, 0.25])
@pytest.mark.parametrize("use_mask", [True, False])
def test_scales(nWh, nWw, wh, ww, hd, heads, scale, use_mask):
    from terra_b200.ops.attention import WindowGeometry, window_attention, window_attention_reference

    torch.manual_seed(wh + ww)
    geo, C = WindowGeometry(1, nWh, nWw, wh, ww), hd * heads
    rows = nWh * nWw * geo.N
    qkv = torch.randn(rows, 3 * C, device="cuda").to(torch.bfloat16).requires_grad_(True)
    table = (torch.randn((2 * wh - 1) * (2 * ww - 1), heads, device="cuda") * 0.5).requires_grad_(True)
    dout = torch.randn(rows, C, device="cuda").to(torch.bfloat16)
    out = window_attention(qkv, geo, heads, True, table, use_mask, scale)
    out.backward(dout)
    q32, t32 = (t.detach().float().requires_grad_(True) for t in (qkv, table))
    ref = window_attention_reference(q32.reshape(1, nWh * nWw, geo.N, -1), geo, heads, True, t32, use_mask, scale).reshape(-1, C)
    ref.backward(dout.float())
    for got, want in ((out, ref), (qkv.grad, q32.grad), (table.grad, t32.grad)):
        assert ((got.float() - want).norm() <= REL * want.norm()).item()
