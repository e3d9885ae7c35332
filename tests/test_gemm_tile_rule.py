"""The tile rule of plain products (host code): where CTA pairs may be taken at all."""
import pytest


@pytest.mark.parametrize("sms,pairs", [(1, False), (2, True), (148, True)])
def test_a_pair_needs_two_multiprocessors(sms, pairs):
    from terra_b200 import _ext

    bn, ctas = _ext.load().gemm_tile(128 * 1088, 1152, 384, sms=sms)
    assert bn in (128, 192, 256) and (ctas == 2) == pairs
