"""Convolutions whose tiles are 64 pixels of two rows or 32 of four: images that such tiles cover in fewer of them, with rows and columns left over, several
samples (a tile must not run on into the next), all gathered forms, and the patch embedding.

Bound: fp32 sums, one rounding to bf16 (2^-9): 3e-3 of the norm."""
import pytest
import torch
import torch.nn.functional as TF

pytestmark = pytest.mark.gpu


def _rand(*shape, scale=1.0):
    return (torch.randn(*shape, device="cuda") * scale).to(torch.bfloat16)


def _close(got, want):
    got = got.permute(0, 3, 1, 2).double()
    return ((got - want).norm() <= 3e-3 * want.norm()).item()


# tiles of 128 x 1 / 64 x 2 / 32 x 4
@pytest.mark.parametrize("B,H,W", [(1, 151, 40), (2, 77, 180), (3, 53, 30), (1, 201, 65), (5, 31, 96), (2, 76, 131)])
@pytest.mark.parametrize("C", [64, 136])
def test_stride_1(B, H, W, C):
    from terra_b200 import _ext
    from terra_b200.ops import conv
    from terra_b200.ops.gemm import check_status, status_word

    torch.manual_seed(H)
    ext, S = _ext.load(), status_word("cuda")
    x, w, b = _rand(B, H, W, C), _rand(C, C, 3, 3, scale=0.04), _rand(C)
    y = torch.full_like(x, float("nan"))
    ext.conv3x3_fwd(x, conv.pack_conv3x3_weight(w), y, 1, 1, b, None, S, None, None)
    check_status("cuda")
    xr = x.double().permute(0, 3, 1, 2)
    assert _close(y, TF.conv2d(xr, w.double(), b.double(), padding=1))
    wt = _rand(C, C, 2, 2, scale=0.1)
    o = torch.full((B, 2 * H, 2 * W, C), float("nan"), device="cuda", dtype=torch.bfloat16)
    ext.convt2x2(0, x, conv._pack_convt(wt), conv._pack_convt_bias(b), o, S)
    check_status("cuda")
    assert _close(o, TF.conv_transpose2d(xr, wt.double(), b.double(), stride=2))
    dx = torch.full((B, 2 * H, 2 * W, C), float("nan"), device="cuda", dtype=torch.bfloat16)
    ext.conv3x3_s2_dgrad(x, conv.pack_conv3x3_weight_s2_dgrad(w), dx, S)
    check_status("cuda")
    assert _close(dx, TF.conv_transpose2d(xr, w.double(), stride=2, padding=1, output_padding=1))


@pytest.mark.parametrize("B,rows,cols,top,left", [(1, 160, 40, 0, 0), (2, 90, 70, 3, 2)])
def test_patch_embedding_and_recovery(B, rows, cols, top, left):
    from terra_b200.models.hierarchical_swin import patchify, unpatchify
    from terra_b200.ops.gemm import check_status
    from terra_b200.ops.patch import embed_image, recover_image
    from terra_b200.utils.flat_params import ParamArena

    torch.manual_seed(rows)
    p, C, D = 4, 6, 64
    H, W = (rows - top - 1) * p, (cols - left) * p
    embed, recover = torch.nn.Linear(p * p * C, D).cuda(), torch.nn.Linear(D, p * p * C).cuda()
    ParamArena(embed), ParamArena(recover)
    x, t = _rand(B, H, W, C), _rand(B, rows, cols, D)
    with torch.no_grad():
        y = embed_image(x, embed, p, (rows * p, cols * p), top * p, left * p)
        out = recover_image(t, recover, x, p, top * p, left * p)
        check_status("cuda")
        padded = TF.pad(x.double(), (0, 0, left * p, 0, top * p, p))
        want = TF.linear(patchify(padded, p), embed.weight.bf16.double(), embed.bias.bf16.double())
        assert (y.double() - want).norm() <= 3e-3 * want.norm()
        want = unpatchify(TF.linear(t.double(), recover.weight.bf16.double(), recover.bias.bf16.double()), p)[:, top * p:top * p + H, left * p:left * p + W]
        assert (out.double() - want - x.double()).norm() <= 3e-3 * (want + x.double()).norm()
