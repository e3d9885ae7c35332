"""Weight gradients of convolutions with all taps as one product: tiles that run on across taps (channels that are no multiple of a box of
64), the bias gradient as a row of ones with and without a tile to spare, stacked tiles and CTA pairs, splits with few k-blocks, strides.

Bound: bf16 operands are exact and sums fp32 in another order: 1e-5 of the norm."""
import pytest
import torch

pytestmark = pytest.mark.gpu

# {columns, CTAs, row blocks, split}; None: the rule's
PLANS = [None, (128, 1, 1, 1), (192, 1, 2, 3), (256, 2, 1, 2), (384, 2, 1, 1), (384, 2, 1, 5)]


def _rand(gen, *shape):
    return torch.randn(*shape, generator=gen, device="cuda").to(torch.bfloat16)


def _close(got, want):
    return ((got.double() - want).norm() / want.norm()).item() < 1e-5


@pytest.mark.parametrize("plan", PLANS)
@pytest.mark.parametrize("B,H,W,Cin,Cout,stride", [(1, 1, 2, 8, 8, 1), (2, 9, 130, 96, 200, 1), (1, 12, 65, 384, 384, 1), (1, 7, 64, 256, 264, 1),
                                                   (2, 11, 140, 192, 192, 2), (1, 30, 90, 128, 520, 2)])
def test_conv3x3(plan, B, H, W, Cin, Cout, stride):
    from terra_b200 import _ext
    from terra_b200.ops.gemm import check_status, status_word

    ext, gen = _ext.load(), torch.Generator(device="cuda").manual_seed(H + W)
    x, dy = _rand(gen, B, H, W, Cin), _rand(gen, B, -(-H // stride), W // stride, Cout)
    dw, db, gw = torch.zeros(9, Cin, Cout, device="cuda"), torch.ones(Cout, device="cuda"), torch.ones(Cout, Cin, 3, 3, device="cuda")
    ext.conv3x3_wgrad_taps(x, dy, dw, stride, status_word("cuda"), db, True, 1, None if plan is None else list(plan))
    ext.fold_taps(dw, gw)
    check_status("cuda")
    w = torch.zeros(Cout, Cin, 3, 3, device="cuda", dtype=torch.float64, requires_grad=True)
    torch.nn.functional.conv2d(x.double().permute(0, 3, 1, 2), w, padding=1, stride=stride).backward(dy.double().permute(0, 3, 1, 2))
    assert _close(gw - 1, w.grad) and _close(db - 1, dy.double().sum((0, 1, 2))) and not dw.any()


@pytest.mark.parametrize("plan", [p for p in PLANS if p is None or p[0] != 256])
@pytest.mark.parametrize("B,H,W,Cin,Cout", [(1, 1, 1, 8, 8), (2, 3, 70, 96, 72), (1, 5, 64, 384, 384), (3, 4, 65, 200, 264)])
def test_conv_transpose2x2(plan, B, H, W, Cin, Cout):
    from terra_b200 import _ext
    from terra_b200.ops.gemm import check_status, status_word

    ext, gen = _ext.load(), torch.Generator(device="cuda").manual_seed(H + W)
    x, dy = _rand(gen, B, H, W, Cin), _rand(gen, B, 2 * H, 2 * W, Cout)
    dw, db, gw = torch.zeros(4, Cout, Cin, device="cuda"), torch.ones(Cout, device="cuda"), torch.ones(Cin, Cout, 2, 2, device="cuda")
    ext.convt2x2_wgrad_taps(x, dy, dw, status_word("cuda"), db, True, 1, None if plan is None else list(plan))
    ext.fold_taps(dw, gw)
    check_status("cuda")
    taps = dy.double().view(B, H, 2, W, 2, Cout).permute(2, 4, 5, 0, 1, 3).reshape(4, Cout, -1) @ x.double().view(-1, Cin)
    assert _close(gw - 1, taps.permute(2, 1, 0).reshape(Cin, Cout, 2, 2)) and _close(db - 1, dy.double().sum((0, 1, 2)))


@pytest.mark.parametrize("Cin,Cout,stride", [(96, 128, 1), (384, 384, 2)])
def test_without_the_fused_bias_gradient(Cin, Cout, stride):
    from terra_b200 import _ext
    from terra_b200.ops.gemm import check_status, status_word

    ext, gen = _ext.load(), torch.Generator(device="cuda").manual_seed(5)
    x, dy = _rand(gen, 1, 10, 68, Cin), _rand(gen, 1, 10 // stride, 68 // stride, Cout)
    fused, apart = (torch.zeros(9, Cin, Cout, device="cuda") for _ in range(2))
    db = torch.zeros(2, Cout, device="cuda")
    ext.conv3x3_wgrad_taps(x, dy, fused, stride, status_word("cuda"), db[0], True)
    ext.conv3x3_wgrad_taps(x, dy, apart, stride, status_word("cuda"), db[1], False)
    check_status("cuda")
    assert _close(fused, apart.double()) and _close(db[0], dy.double().sum((0, 1, 2))) and _close(db[1], dy.double().sum((0, 1, 2)))


def test_rule_on_the_sizes_it_is_for():
    from terra_b200 import _ext

    plan = _ext.load().tap_wgrad_plan
    assert plan(9, 384, 384, 9216, True, False)[:2] == [384, 2]      # 27 blocks, and the row of ones fills the last pair
    assert plan(9, 192, 192, 288, True, False)[1] == 1               # a half of 192 columns is no whole box
    assert plan(9, 384, 384, 2, True, False)[3] <= 2                 # never more splits than k-blocks
    for kb in (100, 2304, 9216):      # sums over no more of the contraction at a time than asked for
        for least in (1, 7, 18):
            assert -(-kb // plan(4, 384, 384, kb, False, True, least)[3]) <= max(24, -(-kb // least))
