"""Weight gradients over the tile plans: two row blocks per tile with an odd last block and partial blocks, column sums shared
out over the column tiles (also where a split has fewer k-blocks than there are tiles), tile widths 128, 192 and 256, sizes
on both sides of the rules.

Bound: bf16 operands are exact and sums fp32 in another order: 1e-5 of the norm (1e-4 for gradients summed over 1e5 rows)."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _rand(*shape, scale=1.0):
    return (torch.randn(*shape, device="cuda") * scale).to(torch.bfloat16)


def _rel(got, ref):
    return ((got - ref).norm() / ref.norm()).item()


@pytest.mark.parametrize("M,N,K", [(1, 8, 8), (65, 96, 96), (1000, 288, 96), (9000, 384, 1536), (40000, 384, 384), (40001, 1152, 384),
                                   (30000, 200, 2976), (30000, 1528, 200), (20000, 1024, 1024), (70000, 128, 64), (120000, 640, 192)])
@pytest.mark.parametrize("sums", [True, False])
def test_linear(M, N, K, sums):
    from terra_b200.ops.blocks import wgrad_accumulate
    from terra_b200.ops.gemm import check_status

    torch.manual_seed(M)
    dy, x = _rand(M, N), _rand(M, K)
    gw, gb = torch.ones(N, K, device="cuda"), torch.ones(N, device="cuda")
    wgrad_accumulate(dy, x, gw, gb if sums else None)
    check_status("cuda")
    assert _rel(gw - 1, (dy.double().t() @ x.double()).float()) < 1e-4
    if sums:
        assert _rel(gb - 1, dy.double().sum(0).float()) < 1e-4


@pytest.mark.parametrize("stack,split", [(1, 1), (1, 7), (2, 1), (2, 5), (2, 64)])
@pytest.mark.parametrize("Cin,Cout", [(128, 256), (192, 384), (384, 200), (96, 130 // 8 * 8 + 8)])
def test_convolution(stack, split, Cin, Cout):
    from terra_b200 import _ext
    from terra_b200.ops.gemm import check_status, status_word

    torch.manual_seed(stack + split)
    B, H, W = 2, 9, 130
    x, dy = _rand(B, H, W, Cin), _rand(B, H, W, Cout)
    dw, db = torch.zeros(9, Cout, Cin, device="cuda"), torch.zeros(Cout, device="cuda")
    _ext.load().conv3x3_wgrad(x, dy, dw, 1, split, status_word("cuda"), None, None, bias_grad=db, stack=stack)
    check_status("cuda")
    w = torch.zeros(Cout, Cin, 3, 3, device="cuda", dtype=torch.float64, requires_grad=True)
    torch.nn.functional.conv2d(x.double().permute(0, 3, 1, 2), w, padding=1).backward(dy.double().permute(0, 3, 1, 2))
    assert _rel(dw.view(3, 3, Cout, Cin).permute(2, 3, 0, 1), w.grad.float()) < 1e-5
    assert _rel(db, dy.double().sum((0, 1, 2)).float()) < 1e-5
