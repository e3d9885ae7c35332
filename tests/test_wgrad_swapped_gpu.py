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
