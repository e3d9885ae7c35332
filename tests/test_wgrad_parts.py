"""Weight gradients: how long the parts of the contraction are over which the tensor core sums in fp32, whose error grows with their length (about
2^-24 of the norm per k-block of 64). Lengths are those of plans of 128 and 256 rows that fill the GPU once."""
import pytest

# rows, outputs N x K, with the bias gradient, longest part
LINEAR = [(17280, 1024, 1024, False, 30), (156672, 768, 192, False, 50), (557056, 192, 192, False, 59), (557056, 192, 192, True, 59),
          (20638, 2048, 512, False, 36), (132361, 512, 2048, True, 230), (47463, 2976, 192, True, 62), (187968, 1024, 96, False, 80),
          (91855, 512, 512, False, 39), (13253, 2304, 768, False, 42), (18279, 256, 1024, False, 16), (36228, 256, 256, False, 15)]


@pytest.mark.parametrize("M,N,K,sums,longest", LINEAR)
def test_linear_layers(M, N, K, sums, longest):
    from terra_b200 import _ext

    k_blocks = -(-M // 64)
    assert -(-k_blocks // _ext.load().wgrad_plan(N, K, M, sums)[2]) <= longest


@pytest.mark.parametrize("B,H,W,stride,C", [(2, 40, 30, 2, 384), (1, 31, 248, 2, 384), (1, 16, 166, 1, 384), (2, 12, 21, 1, 1024), (1, 512, 1088, 1, 384)])
def test_convolutions_keep_the_least_number_of_parts_down_to_15_k_blocks(B, H, W, stride, C):
    from terra_b200 import _ext
    from terra_b200.ops.conv import _wgrad_split

    k_blocks, parts = B * -(-H // stride) * -(-(W // stride) // 64), _wgrad_split(B, H, W, stride, C, C)[0]
    split = _ext.load().tap_wgrad_plan(9, C, C, k_blocks, True, False, parts)[3]
    assert -(-k_blocks // split) <= max(15, -(-k_blocks // parts))


@pytest.mark.gpu
@pytest.mark.parametrize("M,N,K,sums,longest", LINEAR[:4])
def test_error(M, N, K, sums, longest):
    """1.25 * 2^-24 a k-block, and 2e-7 for the sum of the parts."""
    import torch
    from terra_b200.ops.blocks import wgrad_accumulate
    from terra_b200.ops.gemm import check_status

    gen = torch.Generator(device="cuda").manual_seed(M)
    x, dy = (torch.randn(M, c, generator=gen, device="cuda", dtype=torch.bfloat16) for c in (K, N))
    gw, gb = torch.zeros(N, K, device="cuda"), torch.zeros(N, device="cuda")
    wgrad_accumulate(dy, x, gw, gb if sums else None)
    check_status("cuda")
    want = torch.zeros(N, K, device="cuda", dtype=torch.float64)
    for r in range(0, M, 1 << 17):
        want += dy[r:r + (1 << 17)].double().t() @ x[r:r + (1 << 17)].double()
    assert ((gw.double() - want).norm() <= (1.25 * 2.0 ** -24 * longest + 2e-7) * want.norm()).item()
