"""Padding + patch rearrangement kernels against the tensor operators: bit for bit, every vector width (16, 8, 4 and 2 bytes),
with and without padding, forward and backward; fields that the kernels do not take keep the operators."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _plain(x, core, p, pad, raw):
    from terra_b200.models.hierarchical_swin import patchify, unpatchify

    left, right, top, bottom = pad
    y = unpatchify(core(patchify(torch.nn.functional.pad(x, (0, 0, left, right, top, bottom)), p)), p)
    return y[:, top:top + raw[0], left:left + raw[1]] + x


@pytest.mark.parametrize("B,H,W,C,p,pad", [
    (1, 16, 32, 64, 4, (0, 0, 0, 0)), (2, 24, 40, 8, 4, (0, 0, 8, 0)),
    (1, 21, 30, 8, 4, (1, 1, 1, 2)),       # 16-byte vectors, odd padding
    (1, 24, 40, 138, 4, (0, 0, 4, 4)),     # rows of 16-byte multiples, pixels of 276 bytes
    (1, 24, 38, 6, 4, (1, 1, 0, 0)),       # 4-byte vectors
    (1, 23, 41, 5, 4, (2, 1, 1, 0)),       # 2-byte vectors
    (1, 26, 44, 3, 2, (0, 0, 1, 1)), (1, 6, 1200, 96, 2, (4, 4, 0, 0)),
])
def test_matches_the_tensor_operators(B, H, W, C, p, pad):
    from terra_b200.ops.patch import pad_patchify, unpatchify_add

    torch.manual_seed(0)
    left, right, top, bottom = pad
    shape = (H + top + bottom, W + left + right)
    x = torch.randn(B, H, W, C, device="cuda").to(torch.bfloat16)
    g = torch.randn_like(x)
    core = lambda t: t * 2
    a, b = x.clone().requires_grad_(True), x.clone().requires_grad_(True)
    ya = unpatchify_add(core(pad_patchify(a, p, shape, top, left)), a, p, top, left)
    yb = _plain(b, core, p, pad, (H, W))
    assert torch.equal(ya, yb)
    ya.backward(g)
    yb.backward(g)
    assert torch.equal(a.grad, b.grad)


def test_model_takes_fields_in_other_layouts():
    """A non-contiguous or fp32 field gives the same forecast as its contiguous bf16 copy."""
    from terra_b200.models.hierarchical_swin import SequentialSwinReference

    torch.manual_seed(0)
    model = SequentialSwinReference(1, num_channels=6, patch_size=4, window_size=8, height=60, width=64, embedding_dim=64,
                                    num_heads=[2], depths=[1]).cuda()
    x = torch.randn(1, 60, 64, 6, device="cuda").to(torch.bfloat16)
    with torch.no_grad():
        y = model(x)
        assert torch.equal(model(x.transpose(1, 2).contiguous().transpose(1, 2)), y)
        assert torch.equal(model(x.float()), y)
