"""The transposed convolution's weight and bias gradients from one product (dy displaced, its column sums shared out over the column
tiles of a tap): partial tiles and chunks, stacked row blocks, splits. fp32 sums in another order: 1e-5 of the norm."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("B,H,W,Cin,Cout", [(1, 1, 1, 8, 8), (2, 3, 70, 96, 72), (1, 5, 64, 384, 384), (3, 4, 65, 200, 264), (1, 40, 130, 64, 512)])
@pytest.mark.parametrize("stack,split", [(1, 1), (1, 5), (2, 3)])
def test_one_product(B, H, W, Cin, Cout, stack, split):
    from terra_b200 import _ext
    from terra_b200.ops.gemm import check_status, status_word

    gen = torch.Generator(device="cuda").manual_seed(H)
    x = torch.randn(B, H, W, Cin, generator=gen, device="cuda").to(torch.bfloat16)
    dy = torch.randn(B, 2 * H, 2 * W, Cout, generator=gen, device="cuda").to(torch.bfloat16)
    dw, db = torch.zeros(4, Cout, Cin, device="cuda"), torch.ones(Cout, device="cuda")
    _ext.load().convt2x2_wgrad(x, dy, dw, split, status_word("cuda"), stack, db)
    check_status("cuda")
    taps = dy.double().view(B, H, 2, W, 2, Cout).permute(2, 4, 5, 0, 1, 3).reshape(4, Cout, -1)
    want = taps @ x.double().view(-1, Cin)
    assert (dw.double() - want).norm() <= 1e-5 * want.norm()
    sums = 1 + dy.double().sum((0, 1, 2))
    assert (db.double() - sums).norm() <= 1e-5 * sums.norm()
