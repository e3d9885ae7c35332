"""Bias gradients that are rows of ones of a weight gradient's product, over parts as long as layers have (hundreds of k-blocks): 3x3
convolutions and the transposed weight gradient of a patch embedding, outputs with and without a tensor map, infinities.

Bound: a row of ones takes every 32nd k-block and the tensor core's fp32 sums lose at most 2^-24 of the result per k-block: 870 / 32 * 2^-24 =
1.6e-6 for terms of one sign; random signs keep under a third of it (5e-7; one row over all k-blocks is at 2.6e-6)."""
import pytest
import torch

pytestmark = pytest.mark.gpu
REL = 5e-7


def _rel(got, want):
    return ((got.double() - want).norm() / want.norm()).item()


def _field(gen, *shape):
    return torch.randn(*shape, generator=gen, device="cuda", dtype=torch.bfloat16)


def _conv_sums(dy, C, stride, plan):
    from terra_b200 import _ext
    from terra_b200.ops.gemm import check_status, status_word

    B, H, W, N = dy.shape
    x = torch.zeros(B, H * stride, W * stride, C, device="cuda", dtype=torch.bfloat16)
    dw, db = torch.zeros(9, C, N, device="cuda"), torch.zeros(N, device="cuda")
    _ext.load().conv3x3_wgrad_taps(x, dy, dw, stride, status_word("cuda"), db, True, 1, plan)
    check_status("cuda")
    return db


@pytest.mark.parametrize("plan", [None, [384, 2, 1, 1], [384, 2, 1, 10], [256, 2, 1, 2], [192, 1, 2, 1], [128, 1, 1, 1]])
@pytest.mark.parametrize("H,W,C,N,stride", [(435, 128, 64, 384, 1), (870, 50, 72, 264, 1), (290, 192, 8, 384, 2)])
def test_convolution_over_long_parts(H, W, C, N, stride, plan):
    dy = _field(torch.Generator(device="cuda").manual_seed(H), 1, H, W, N)
    assert _rel(_conv_sums(dy, C, stride, plan), dy.double().sum((0, 1, 2))) < REL


@pytest.mark.parametrize("k_blocks", [1, 2, 31, 32, 33, 65])
def test_every_k_block_is_counted_once(k_blocks):
    dy = torch.ones(1, k_blocks, 64, 136, device="cuda", dtype=torch.bfloat16)
    for plan in ([192, 1, 2, 1], [128, 1, 1, 3]):
        assert (_conv_sums(dy, 8, 1, plan) == 64 * k_blocks).all()


@pytest.mark.parametrize("plan", [[384, 2, 1, 1], [128, 1, 1, 4]])
def test_infinities_stay_infinities(plan):
    dy = torch.zeros(1, 40, 64, 384, device="cuda", dtype=torch.bfloat16)
    dy[0, 3, 5, 7], dy[0, 39, 63, 200], dy[0, 20, 0, 300] = float("inf"), float("-inf"), float("nan")
    db = _conv_sums(dy, 64, 1, plan)
    assert db[7] == float("inf") and db[200] == float("-inf") and db[300].isnan()
    assert torch.isfinite(db).sum() == 381


@pytest.mark.parametrize("M,N,K,pad", [(139264, 384, 2976, 0), (557056, 384, 2976, 0), (60001, 376, 2208, 8)])
def test_transposed_weight_gradient(M, N, K, pad):
    from terra_b200 import _ext
    from terra_b200.ops.blocks import wgrad_accumulate
    from terra_b200.ops.gemm import check_status

    assert _ext.load().wgrad_swapped(N, K, M, True)
    gen = torch.Generator(device="cuda").manual_seed(M)
    dy, x = _field(gen, M, N), torch.zeros(M, K, device="cuda", dtype=torch.bfloat16)
    gw, gb = torch.zeros(N, K + pad, device="cuda")[:, :K], torch.zeros(N, device="cuda")
    wgrad_accumulate(dy, x, gw, gb)
    check_status("cuda")
    assert _rel(gb, dy.double().sum(0)) < REL and not gw.any()


@pytest.mark.parametrize("M,N,K", [(557056, 2976, 384), (156672, 3072, 1024), (60000, 384, 384), (60001, 288, 96)])
def test_weight_gradient_with_its_column_sums(M, N, K):
    """The sums that are an MMA against a tile of ones: each of a k-block's four MMAs has a column of its own."""
    from terra_b200.ops.blocks import wgrad_accumulate
    from terra_b200.ops.gemm import check_status

    gen = torch.Generator(device="cuda").manual_seed(N)
    dy, x = _field(gen, M, N), torch.zeros(M, K, device="cuda", dtype=torch.bfloat16)
    gw, gb = torch.zeros(N, K, device="cuda"), torch.zeros(N, device="cuda")
    wgrad_accumulate(dy, x, gw, gb)
    check_status("cuda")
    want = torch.stack([dy[:, c:c + 384].double().sum(0) for c in range(0, N, 384)]).reshape(-1) if N % 384 == 0 else dy.double().sum(0)
    assert _rel(gb, want) < REL and not gw.any()
    dy[5, 3], dy[M - 1, 7], dy[M // 2, 9] = float("inf"), float("-inf"), float("nan")
    gb.zero_()
    wgrad_accumulate(dy, x[:, :K], gw, gb)
    assert gb[3] == float("inf") and gb[7] == float("-inf") and gb[9].isnan() and torch.isfinite(gb).sum() == N - 3
