"""The tile rule of plain products (host code): where CTA pairs may be taken at all."""
import pytest


@pytest.mark.parametrize("sms,pairs", [(1, False), (2, True), (148, True)])
def test_a_pair_needs_two_multiprocessors(sms, pairs):
    from terra_b200 import _ext

    bn, ctas = _ext.load().gemm_tile(128 * 1088, 1152, 384, sms=sms)
    assert bn in (128, 192, 256) and (ctas == 2) == pairs


@pytest.mark.parametrize("N,K", [(96, 96), (288, 96), (384, 1536), (384, 2976), (1000, 1000), (192, 2208)])
@pytest.mark.parametrize("rows", [64, 512, 2048])
def test_few_rows_keep_the_bias_sums_in_the_weight_gradient(N, K, rows):
    """Tiles 256 wide leave the column sums to two launches of their own, which cost more than the product of so few rows."""
    from terra_b200 import _ext

    ext = _ext.load()
    bn, stack, split = ext.wgrad_plan(N, K, rows, True)
    assert bn in (128, 192) and stack in (1, 2) and 1 <= split <= -(-rows // 64)
    with pytest.raises(RuntimeError):
        ext.wgrad_plan(N, 0, rows, True)
