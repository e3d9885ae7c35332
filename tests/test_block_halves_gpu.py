"""The native attention half against the same launches made one by one from Python: outputs and input gradients bit for bit,
parameter gradients to the order of their fp32 atomics (1e-5 of the norm); with and without a bias table, several samples,
widths with partial tiles, rows given as a pitched weight-gradient operand."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _rel(a, b):
    return ((a - b).norm() / b.norm().clamp_min(1e-20)).item()


@pytest.mark.parametrize("B,nWh,nWw,window,dim,heads,shifted,table", [
    (1, 2, 4, (8, 8), 96, 3, True, True), (2, 3, 2, (7, 7), 64, 2, True, False), (1, 2, 3, (8, 12), 192, 12, False, True),
    (1, 9, 11, (8, 8), 384, 6, True, True),
])
def test_attention_half(monkeypatch, B, nWh, nWw, window, dim, heads, shifted, table):
    from terra_b200.models.layers import SwinAttentionHalf
    from terra_b200.ops import blocks
    from terra_b200.ops.attention import WindowGeometry
    from terra_b200.ops.gemm import check_status
    from terra_b200.utils.flat_params import ParamArena

    torch.manual_seed(0)
    mod = SwinAttentionHalf(int(shifted), dim, window, heads, use_relative_position_bias=table).cuda()
    arena = ParamArena(mod)
    geo = WindowGeometry(B, nWh, nWw, *window)
    x = torch.randn(geo.rows_local, dim, device="cuda").to(torch.bfloat16)
    dy = torch.randn_like(x)
    got = []
    for native in (True, False):
        if not native:
            monkeypatch.setattr(blocks, "_native_half", lambda *a: False)
        arena.zero_grad()
        t = x.clone().requires_grad_(True)
        y = blocks.attention_half(t, mod, geo, shifted)
        y.backward(dy)
        check_status("cuda")
        got.append((y.detach(), t.grad, arena.grad.clone()))
    assert torch.equal(got[0][0], got[1][0]) and torch.equal(got[0][1], got[1][1])
    assert _rel(got[0][2], got[1][2]) < 1e-5


def test_weight_gradient_of_pitched_rows():
    from terra_b200.ops.blocks import wgrad_accumulate

    torch.manual_seed(1)
    wide = torch.randn(777, 512, device="cuda").to(torch.bfloat16)
    dy, x = wide[:, :200], wide[:, 256:352]
    gw, gb = torch.zeros(200, 96, device="cuda"), torch.zeros(200, device="cuda")
    wgrad_accumulate(dy, x, gw, gb)
    ref = dy.float().t() @ x.float()
    assert _rel(gw, ref) < 1e-5 and _rel(gb, dy.float().sum(0)) < 1e-5


@pytest.mark.parametrize("M,N,K", [(10, 64, 0), (10, 0, 64), (0, 64, 64)])
def test_weight_gradient_refuses_empty_operands(M, N, K):
    """The plan of the tiles divides by their number; an empty operand is an error that Python sees."""
    from terra_b200.ops.blocks import wgrad_accumulate

    dy, x = torch.zeros(M, N, device="cuda", dtype=torch.bfloat16), torch.zeros(M, K, device="cuda", dtype=torch.bfloat16)
    with pytest.raises(RuntimeError):
        wgrad_accumulate(dy, x, torch.zeros(N, K, device="cuda"), torch.zeros(N, device="cuda"))
