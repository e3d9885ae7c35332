"""Inference of a model on fields, settings and weights in every form that training takes them: what the patch layers on the image itself do
not take goes to the copies.

Bound: the two builds round the sum with the input once or twice (2^-9): 2 % of the norm for a whole model."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _model(build=None, **more):
    from terra_b200.models.hierarchical_swin import SequentialHierarchicalSwin

    torch.manual_seed(4)
    return (build or SequentialHierarchicalSwin)(2, num_channels=10, patch_size=4, window_size=4, height=64, width=96, embedding_dim=64, num_heads=2,
                                                 num_layers=2, **more).cuda()


def _field(offset=0):
    flat = torch.randn(64 * 96 * 10 + 8, generator=torch.Generator(device="cuda").manual_seed(1), device="cuda").to(torch.bfloat16)
    return flat[offset:offset + 64 * 96 * 10].view(1, 64, 96, 10)


def _close(a, b):
    return ((a.double() - b.double()).norm() <= 2e-2 * b.double().norm()).item()


@pytest.mark.parametrize("offset", [0, 1, 2, 4, 8])
def test_a_field_at_any_address(offset):
    from terra_b200.ops.gemm import check_status
    from terra_b200.ops.patch import direct_patches_apply

    m, x = _model(), _field(offset)
    assert x.is_contiguous() and x.data_ptr() % 16 == 2 * offset % 16
    kept = m(x)
    with torch.no_grad():
        assert direct_patches_apply(x, 4, 0, 0, 64) == (offset % 8 == 0)
        free = m(x)
    check_status("cuda")
    assert _close(free, kept)
