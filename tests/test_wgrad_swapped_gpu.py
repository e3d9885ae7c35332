"""Weight gradients computed as their transpose (few outputs of a wide layer and many rows): ragged rows, pitched gradients, with and
without the bias sums. bf16 operands are exact and sums fp32 in another order: 1e-4 of the norm over 1e5 rows and more."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("M,N,K,sums", [(450001, 384, 2304, True), (150001, 384, 2304, False), (200000, 376, 2296, False)])
def test_linear(M, N, K, sums):
    from terra_b200 import _ext
    from terra_b200.ops.blocks import wgrad_accumulate
    from terra_b200.ops.gemm import check_status

    if N == 384:
        assert _ext.load().wgrad_plan(N, K, M, sums)[0] == 1384
    gen = torch.Generator(device="cuda").manual_seed(M)
    dy, x = (torch.randn(M, c, generator=gen, device="cuda", dtype=torch.bfloat16) for c in (N, K))
    wide, gb = torch.ones(N, K + 24, device="cuda"), torch.ones(N, device="cuda")
    wgrad_accumulate(dy, x, wide[:, 8:8 + K], gb if sums else None)
    check_status("cuda")
    want = sum(dy[i:i + 65536].double().t() @ x[i:i + 65536].double() for i in range(0, M, 65536))
    assert ((wide[:, 8:8 + K] - 1).double() - want).norm() <= 1e-4 * want.norm()
    assert (wide[:, :8] == 1).all() and (wide[:, 8 + K:] == 1).all()
    if sums:
        total = dy.double().sum(0)
        assert ((gb - 1).double() - total).norm() <= 1e-4 * total.norm()


@pytest.mark.parametrize("M,N,K,sums", [(450001, 384, 2304, True), (150001, 384, 2304, False), (200000, 376, 2296, False)])
def test_the_sizes_above_take_the_transpose(M, N, K, sums):
    """(An untransposed product of tiles 384 wide has the same width in its plan.)"""
    from terra_b200 import _ext

    assert _ext.load().wgrad_swapped(N, K, M, sums)


@pytest.mark.parametrize("bn", [64, 128, 192, 256, 1128, 1256, 1384])
@pytest.mark.parametrize("M,N,K,split", [(64, 8, 8, 1), (200, 40, 264, 3), (1000, 72, 128, 5), (777, 384, 392, 7), (5000, 376, 1000, 11)])
def test_the_transposed_store(bn, M, N, K, split):
    """One and several row blocks, partial chunks of 32 columns, every tile, splits; sums of 1e3 values in another order."""
    from terra_b200 import _ext
    from terra_b200.ops import _flags as F
    from terra_b200.ops.gemm import check_status, status_word

    gen = torch.Generator(device="cuda").manual_seed(M)
    dy, x = (torch.randn(M, c, generator=gen, device="cuda").to(torch.bfloat16) for c in (N, K))
    wide = torch.ones(N + 2, K + 24, device="cuda")
    out = wide[1:1 + N, 8:8 + K]
    _ext.load().gemm(x, True, dy, True, out, F.EPI_OUT_F32 | F.EPI_ATOMIC | F.EPI_TRANSPOSE, None, None, None, None, 1.0, split, bn,
                     status_word("cuda"), 0, [], 0, [], 0, 0, 0, 1, 1)
    check_status("cuda")
    want = dy.double().t() @ x.double()
    assert ((out - 1).double() - want).norm() <= 1e-5 * want.norm()
    out.fill_(1.0)
    assert (wide == 1).all()
