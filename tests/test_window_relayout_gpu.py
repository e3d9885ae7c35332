"""Windows of an image and back by one copy kernel: against the tensor operators, bit for bit, and its gradient; what it does not take."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("B,nWh,nWw,wh,ww,C", [(1, 1, 2, 2, 1, 8), (2, 3, 5, 4, 8, 96), (1, 7, 3, 7, 7, 64), (1, 12, 15, 8, 12, 192), (3, 2, 9, 5, 13, 8)])
def test_there_and_back(B, nWh, nWw, wh, ww, C):
    from terra_b200.parallel.context import _swap_middle

    gen = torch.Generator(device="cuda").manual_seed(C + nWw)
    x = torch.randn(B, nWh * wh, nWw * ww, C, generator=gen, device="cuda").to(torch.bfloat16).requires_grad_(True)
    rows = _swap_middle(x, B * nWh, wh, nWw, (B * nWh * wh * nWw * ww, C))
    want = x.detach().view(B, nWh, wh, nWw, ww, C).permute(0, 1, 3, 2, 4, 5).reshape(-1, C)
    assert torch.equal(rows, want)
    back = _swap_middle(rows, B * nWh, nWw, wh, tuple(x.shape))
    assert torch.equal(back, x)
    g = torch.randn(rows.shape, generator=gen, device="cuda").to(torch.bfloat16)
    rows.backward(g)
    assert torch.equal(x.grad.view(B, nWh, wh, nWw, ww, C).permute(0, 1, 3, 2, 4, 5).reshape(-1, C), g)
    once, = torch.autograd.grad(_swap_middle(x, B * nWh, wh, nWw, rows.shape).square().sum(), x, create_graph=True)
    twice, = torch.autograd.grad(once.sum(), x)                                                   # the gradient has a gradient too
    assert torch.equal(twice, torch.full_like(x, 2))


def test_what_the_tensor_operators_do():
    from terra_b200.parallel.context import _swap_middle

    assert _swap_middle(torch.zeros(1, 8, 1, 16, device="cuda", dtype=torch.bfloat16), 1, 8, 1, (8, 16)) is None   # nothing to move
    x = torch.zeros(1, 8, 6, 10, device="cuda", dtype=torch.bfloat16)
    assert _swap_middle(x, 1, 8, 6, (48, 10)) is None                                             # 20 bytes inside
    assert _swap_middle(x.float(), 1, 8, 6, (48, 10)) is None
    assert _swap_middle(x.cpu(), 1, 8, 6, (48, 10)) is None
    assert _swap_middle(torch.zeros(16, 16, 8, device="cuda", dtype=torch.bfloat16).transpose(0, 1), 1, 16, 16, (256, 8)) is None
