"""Window attention where its tiles change: 32-token blocks, two 16-row tiles per warp (head pairs), padding columns beside the
mask, for every head width. The bound is that of the other small-window tests: P, dS and the results are rounded to bf16
(2^-9 each, independent): 3 * 2^-9 = 0.6 % of the norm against fp32; 1 % is allowed."""
import pytest
import torch

from test_attention_small_windows_gpu import REL, _reference, _rel

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("hd", [16, 32, 64, 128])
@pytest.mark.parametrize("wh,ww", [(1, 1), (2, 2), (3, 5), (4, 8), (8, 4), (2, 16), (3, 11), (5, 8), (7, 7), (7, 8), (8, 8), (5, 13), (8, 12)])
def test_window_sizes(wh, ww, hd):
    from terra_b200.ops.attention import WindowGeometry, window_attention

    for heads, shifted, grid in ((2, True, (3, 4)), (3, False, (1, 2)), (4, True, (1, 1))):
        if hd * heads > 384:
            continue
        torch.manual_seed(wh * ww + hd)
        geo, C = WindowGeometry(1, *grid, wh, ww), hd * heads
        rows = grid[0] * grid[1] * geo.N
        qkv = torch.randn(rows, 3 * C, device="cuda").to(torch.bfloat16).requires_grad_(True)
        table = (torch.randn((2 * wh - 1) * (2 * ww - 1), heads, device="cuda") * 0.5).requires_grad_(True)
        dout = torch.randn(rows, C, device="cuda").to(torch.bfloat16)
        out = window_attention(qkv, geo, heads, shifted, table, True, hd ** -0.5)
        out.backward(dout)
        ref, dq, dt = _reference(qkv, table, dout, geo, heads, shifted, hd ** -0.5)
        assert _rel(out, ref) < REL, (heads, shifted)
        assert _rel(qkv.grad, dq) < REL
        # (a window whose tokens are all apart has no score that matters: its gradient is zero)
        assert (table.grad - dt).norm() <= REL * dt.norm() + 1e-6
