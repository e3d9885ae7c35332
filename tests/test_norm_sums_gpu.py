"""GroupNorm's sums without shared-memory atomics, its statistics finished by the last block, and the LayerNorm backward that sums
the shortcut's gradient: partial column rounds, more than 64 vectors a row, more than the default shared memory, one pixel, several
samples, used twice in a row (what a launch leaves behind must be clean)."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("B,HW,C,groups", [(1, 1, 8, 1), (2, 77, 24, 3), (1, 300, 192, 32), (3, 1000, 96, 32), (1, 5000, 520, 5), (2, 64, 2048, 32),
                                           (1, 200, 4096, 32), (150, 20, 64, 8)])
def test_groupnorm_silu_backward_and_statistics(B, HW, C, groups):
    from terra_b200.ops import conv
    from terra_b200.utils.flat_params import ParamArena

    gen = torch.Generator(device="cuda").manual_seed(C)
    r = lambda *s: torch.randn(*s, generator=gen, device="cuda").to(torch.bfloat16)
    gn = torch.nn.GroupNorm(groups, C).cuda()
    with torch.no_grad():
        for p in gn.parameters():
            p.copy_((torch.randn(C, generator=gen, device="cuda") * 0.3 + 1).to(torch.bfloat16).float())
    arena = ParamArena(gn)
    x, dy = (r(B, 1, HW, C) * 2 + 1), r(B, 1, HW, C)
    xr = x.double().requires_grad_(True)
    p64 = [p.detach().double().requires_grad_(True) for p in gn.parameters()]
    want = torch.nn.functional.silu(torch.nn.functional.group_norm(xr.permute(0, 3, 1, 2), groups, *p64, eps=1e-5)).permute(0, 2, 3, 1)
    want.backward(dy.double())
    for _ in range(2):
        arena.zero_grad()
        t = x.clone().requires_grad_(True)
        y = conv.groupnorm_silu(t, gn)
        y.backward(dy)
        # outputs are rounded to bf16 (2^-9), sums are fp32 (1e-5 of the norm; a single pixel's group may be constant)
        rel = lambda a, b: ((a.double() - b).norm() / b.norm().clamp_min(1e-3)).item()
        assert rel(y.detach(), want.detach()) < 5e-3 and rel(t.grad, xr.grad) < 5e-3
        assert rel(gn.weight.grad, p64[0].grad) < 1e-4 and rel(gn.bias.grad, p64[1].grad) < 1e-4


@pytest.mark.parametrize("rows,dim", [(32767, 1024), (32768, 1024), (33000, 512), (33000, 520), (40001, 768), (33000, 1032)])
@pytest.mark.parametrize("half", ["mlp", "attention"])
def test_bias_gradient_beside_the_norm(rows, dim, half):
    """Both sides of the row and width rule; fp32 sums of 3e4 values in another order: 1e-5 of the norm."""
    from terra_b200.models.layers import MlpHalf, SwinAttentionHalf
    from terra_b200.ops import blocks
    from terra_b200.ops.attention import WindowGeometry
    from terra_b200.utils.flat_params import ParamArena

    torch.manual_seed(1)
    if half == "attention":
        if dim not in (512, 768, 1024):
            pytest.skip("head widths are 16 to 128")
        geo = WindowGeometry(1, 2, rows // 128, 8, 8)
        mod = SwinAttentionHalf(0, dim, (8, 8), dim // 32).cuda()
        rows, bias, run = geo.rows_local, mod.attn.proj.bias, lambda t: blocks.attention_half(t, mod, geo, False)
    else:
        mod = MlpHalf(dim, 256).cuda()
        bias, run = mod.fc2.bias, lambda t: blocks.mlp_half(t, mod)
    ParamArena(mod).zero_grad()
    x = torch.randn(rows, dim, device="cuda").to(torch.bfloat16).requires_grad_(True)
    dy = torch.randn(rows, dim, device="cuda").to(torch.bfloat16)
    run(x).backward(dy)
    want = dy.double().sum(0)
    assert (bias.grad.double() - want).norm() <= 1e-5 * want.norm()


def test_inference_skips_the_pre_activation_only():
    from terra_b200.models.layers import MlpHalf
    from terra_b200.ops import blocks
    from terra_b200.utils.flat_params import ParamArena

    torch.manual_seed(2)
    for dim, rows in ((96, 500), (384, 4000)):
        mod = MlpHalf(dim, 4 * dim).cuda()
        ParamArena(mod)
        x = torch.randn(rows, dim, device="cuda").to(torch.bfloat16)
        y = blocks.mlp_half(x.requires_grad_(True), mod)
        with torch.no_grad():
            assert torch.equal(blocks.mlp_half(x, mod), y)
