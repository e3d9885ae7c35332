"""Patch embedding and recovery on the image itself (inference): padding on all sides, rows of patches around a tile of 128, runs that are no
whole box of 64, several samples, channels of the tokens that are no whole box; which fields take the copies instead; a whole model.

Bounds: one rounding to bf16 (2^-9) after fp32 sums: 3e-3 of the norm; two builds of a model that round elsewhere: 2 %."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _linear(fin, fout, gen):
    from terra_b200.utils.flat_params import ParamArena

    lin = torch.nn.Linear(fin, fout).cuda()
    with torch.no_grad():
        for q in lin.parameters():
            q.copy_((torch.randn(q.shape, generator=gen, device="cuda") * fin ** -0.5).to(torch.bfloat16).float())
    ParamArena(lin)
    return lin


@pytest.mark.parametrize("B,H,W,C,p,pads,dim", [
    (1, 4, 4, 2, 4, (0, 0, 0, 0), 8), (2, 12, 20, 8, 2, (2, 4, 0, 6), 72), (1, 64, 520, 138, 4, (8, 8, 4, 12), 192),
    (3, 32, 516, 20, 4, (0, 32, 8, 0), 96), (1, 9, 387, 8, 3, (3, 0, 0, 6), 200), (1, 16, 16, 64, 1, (1, 2, 3, 4), 64)])
def test_layers(B, H, W, C, p, pads, dim):
    from terra_b200.models.hierarchical_swin import patchify, unpatchify
    from terra_b200.ops.gemm import check_status
    from terra_b200.ops.patch import direct_patches_apply, embed_image, recover_image

    gen = torch.Generator(device="cuda").manual_seed(H + W)
    x = torch.randn(B, H, W, C, generator=gen, device="cuda").to(torch.bfloat16)
    top, bottom, left, right = pads
    shape = (H + top + bottom, W + left + right)
    embed, recover = _linear(p * p * C, dim, gen), _linear(dim, p * p * C, gen)
    t = torch.randn(B, shape[0] // p, shape[1] // p, dim, generator=gen, device="cuda").to(torch.bfloat16)
    with torch.no_grad():
        assert direct_patches_apply(x, p, top, left, dim)
        y = embed_image(x, embed, p, shape, top, left)
        out = recover_image(t, recover, x, p, top, left)
        check_status("cuda")
        padded = torch.nn.functional.pad(x.double(), (0, 0, left, right, top, bottom))
        want = torch.nn.functional.linear(patchify(padded, p), embed.weight.double(), embed.bias.double())
        assert (y.double() - want).norm() <= 3e-3 * want.norm()
        want = unpatchify(torch.nn.functional.linear(t.double(), recover.weight.double(), recover.bias.double()), p)
        want = want[:, top:top + H, left:left + W] + x.double()
        assert (out.double() - want).norm() <= 3e-3 * want.norm()


@pytest.mark.parametrize("H,W,C,p,top,left,dim", [(10, 16, 8, 4, 0, 0, 64), (16, 18, 8, 4, 0, 0, 64), (16, 16, 93, 4, 0, 0, 64), (16, 16, 8, 4, 2, 0, 64),
                                                  (16, 16, 8, 4, 0, 1, 64), (16, 16, 8, 8, 0, 0, 64), (16, 16, 8, 4, 0, 0, 60)])
def test_fields_that_take_the_copies(H, W, C, p, top, left, dim):
    from terra_b200.ops.patch import direct_patches_apply

    x = torch.zeros(1, H, W, C, device="cuda", dtype=torch.bfloat16)
    with torch.no_grad():
        assert not direct_patches_apply(x, p, top, left, dim)
    assert not direct_patches_apply(torch.zeros(1, 16, 16, 8, device="cuda", dtype=torch.bfloat16), 4, 0, 0, 64)      # with gradients


@pytest.mark.parametrize("height,width,sampling", [(64, 96, True), (72, 120, True), (48, 40, False)])
def test_a_model_without_gradients(height, width, sampling):
    from terra_b200.models.hierarchical_swin import SequentialHierarchicalSwin, SequentialSwinReference
    from terra_b200.ops.gemm import check_status

    torch.manual_seed(4)
    build = SequentialHierarchicalSwin if sampling else SequentialSwinReference
    m = build(2, num_channels=10, patch_size=4, window_size=4, height=height, width=width, embedding_dim=64, num_heads=2, num_layers=2).cuda()
    x = torch.randn(2, height, width, 10, device="cuda")
    x = x.permute(0, 3, 1, 2) if m.input_nchw else x
    kept = m(x)
    with torch.no_grad():
        for _ in range(2):
            free = m(x)
            check_status("cuda")
            assert free.shape == kept.shape and (free.double() - kept.double()).norm() <= 2e-2 * kept.double().norm()
            next(m.parameters()).data.mul_(1.0)
