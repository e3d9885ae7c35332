"""Packed operands of the implicit GEMMs: index arithmetic against the tensor operators that define the layouts (CPU), and the
packing kernel against it (GPU), for channel counts with and without padding."""
import pytest
import torch

from terra_b200.ops import conv


def _pad(taps):
    n, t, c = taps.shape
    out = torch.zeros(n, t, (c + 63) // 64 * 64, dtype=torch.bfloat16)
    out[:, :, :c] = taps
    return out.reshape(n, -1)


def _weights(cout, cin, k):
    torch.manual_seed(cout + cin)
    return torch.randn(cout, cin, k, k).to(torch.bfloat16)


SHAPES = [(64, 64), (40, 72), (8, 200), (129, 8), (384, 96)]


@pytest.mark.parametrize("cout,cin", SHAPES)
def test_layouts(cout, cin):
    w = _weights(cout, cin, 3)
    assert torch.equal(conv.pack_conv3x3_weight(w), _pad(w.permute(0, 2, 3, 1).reshape(cout, 9, cin)))
    assert torch.equal(conv.pack_conv3x3_weight_dgrad(w), _pad(w.flip(2, 3).permute(1, 2, 3, 0).reshape(cin, 9, cout)))
    order = [(0, 0), (0, 2), (2, 0), (2, 2), (1, 0), (1, 2), (0, 1), (2, 1), (1, 1)]
    taps = torch.stack([w[:, :, y, x].t() for y, x in order], 1)
    assert torch.equal(conv.pack_conv3x3_weight_s2_dgrad(w), _pad(taps))


@pytest.mark.gpu
@pytest.mark.parametrize("cout,cin", SHAPES)
def test_kernel(cout, cin):
    w = _weights(cout, cin, 3)
    for pack in (conv.pack_conv3x3_weight, conv.pack_conv3x3_weight_dgrad, conv.pack_conv3x3_weight_s2_dgrad):
        assert torch.equal(pack(w.cuda()).cpu(), pack(w))
    v = _weights(cin, cout, 2)             # transposed convolution: (Cin, Cout, 2, 2)
    for args in ((4, 1, cout, 4, cin, 4 * cout, (0,)), (4, 1, cout, 4, cin, 4 * cout, (0,), cout + 56), (1, 0, cin, 4 * cout, cout, 4, range(4))):
        assert torch.equal(conv._pack_taps(v.cuda(), *args).cpu(), conv._pack_taps(v, *args))


def test_transposed_convolution_takes_wide_images_and_small_ones_gathered():
    """The rule between the gathered transposed convolution and the general path (the kernel's tiles are 128 pixels of a row)."""
    from terra_b200.ops import conv

    tiled = lambda *a: bool(conv._convt_tiled(*a))
    assert tiled(1, 5000, 32, 96, 96) and tiled(1, 4, 4, 96, 96) and tiled(1, 148, 31, 96, 96) and tiled(1, 256, 544, 384, 384)
    assert not tiled(1, 149, 31, 96, 96) and not tiled(2, 75, 8, 96, 96)
    assert not tiled(1, 64, 64, 60, 96) and not tiled(1, 64, 64, 96, 60) and not tiled(1, 64, 64, 96, 2056)
