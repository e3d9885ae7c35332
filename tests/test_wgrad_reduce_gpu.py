"""Accumulated fp32 outputs: as TMA reductions of 32 x 32 units where the output's base and pitch are whole 16-byte vectors, by the lanes
elsewhere. Partial units on both edges, outputs next to other data, a factor, every tile form; also the transposed store.

Bound: bf16 operands are exact and sums fp32 in another order: 1e-5 of the norm (what lies beside the output is untouched)."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("bn", [64, 128, 192, 256, 1128, 1256, 1384])
@pytest.mark.parametrize("M,N,K,split", [(64, 8, 8, 1), (200, 40, 264, 3), (1000, 136, 72, 5), (2100, 384, 392, 7)])
@pytest.mark.parametrize("offset,extra", [(0, 0), (8, 12), (1, 7)])      # the last: no tensor map
@pytest.mark.parametrize("turned", [False, True])
def test_forms(bn, M, N, K, split, offset, extra, turned):
    from terra_b200 import _ext
    from terra_b200.ops import _flags as F
    from terra_b200.ops.gemm import check_status, status_word

    gen = torch.Generator(device="cuda").manual_seed(M + bn)
    dy, x = (torch.randn(M, c, generator=gen, device="cuda").to(torch.bfloat16) for c in (N, K))
    wide = torch.ones(N, K + offset + extra, device="cuda")
    out = wide[:, offset:offset + K]
    a, b = (x, dy) if turned else (dy, x)
    flags = F.EPI_OUT_F32 | F.EPI_ATOMIC | (F.EPI_TRANSPOSE if turned else 0)
    _ext.load().gemm(a, True, b, True, out, flags, None, None, None, None, 0.5, split, bn, status_word("cuda"), 0, [], 0, [], 0, 0, 0, 1, 1)
    check_status("cuda")
    want = 0.5 * dy.double().t() @ x.double()
    assert ((out - 1).double() - want).norm() <= 1e-5 * want.norm()
    assert (wide[:, :offset] == 1).all() and (wide[:, offset + K:] == 1).all()


@pytest.mark.parametrize("M,N,K", [(60001, 384, 2976), (40000, 376, 2208), (50000, 264, 1096), (450001, 384, 2304)])      # the last: no room behind 36 boxes
@pytest.mark.parametrize("offset", [0, 2])      # 2: a gradient without a tensor map
def test_bias_sums_as_a_row_of_ones(M, N, K, offset):
    """Transposed weight gradients with the bias gradient in the rows that the last pair has to spare, or apart. Sums of 1e4 values: 1e-4."""
    from terra_b200 import _ext
    from terra_b200.ops.blocks import wgrad_accumulate
    from terra_b200.ops.gemm import check_status

    assert _ext.load().wgrad_swapped(N, K, M, True)
    gen = torch.Generator(device="cuda").manual_seed(M)
    dy, x = (torch.randn(M, c, generator=gen, device="cuda", dtype=torch.bfloat16) for c in (N, K))
    wide, gb = torch.ones(N, K + 8, device="cuda"), torch.ones(N, device="cuda")
    wgrad_accumulate(dy, x, wide[:, offset:offset + K], gb)
    check_status("cuda")
    want, sums = dy.double().t() @ x.double(), dy.double().sum(0)
    assert ((wide[:, offset:offset + K] - 1).double() - want).norm() <= 1e-4 * want.norm() and (gb - 1 - sums).norm() <= 1e-4 * sums.norm()
    assert (wide[:, :offset] == 1).all() and (wide[:, offset + K:] == 1).all()
