"""GroupNorm + SiLU with thousands of groups, whose sums take shared memory beside the rows in flight: forward and backward of a layer around and
beyond the 2048 groups that fit into 48 KB.

Bound: outputs and input gradients are rounded to bf16 (2^-9 of each element, 5e-3 of the norm with the roundings before it)."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("C,groups", [(2048, 2048), (2056, 2056), (4112, 2056), (4096, 4096), (6144, 3072), (6144, 6144)])
def test_forward_and_backward(C, groups):
    from terra_b200.ops.conv import groupnorm_silu
    from terra_b200.utils.flat_params import ParamArena

    gen = torch.Generator(device="cuda").manual_seed(groups)
    norm = torch.nn.GroupNorm(groups, C).cuda()
    with torch.no_grad():
        norm.weight.copy_(1 + 0.1 * torch.randn(C, generator=gen, device="cuda"))
        norm.weight.copy_(norm.weight.to(torch.bfloat16))
    arena = ParamArena(norm)
    arena.zero_grad()
    x, dy = (torch.randn(2, 5, 9, C, generator=gen, device="cuda").to(torch.bfloat16) for _ in range(2))
    x.requires_grad_(True)
    y = groupnorm_silu(x, norm)
    y.backward(dy)
    x64 = x.detach().double().permute(0, 3, 1, 2).requires_grad_(True)
    w64, b64 = (p.detach().double().requires_grad_(True) for p in (norm.weight, norm.bias))
    want = torch.nn.functional.silu(torch.nn.functional.group_norm(x64, groups, w64, b64, norm.eps))
    want.backward(dy.double().permute(0, 3, 1, 2))
    for got, ref, tol in ((y, want.detach().permute(0, 2, 3, 1), 5e-3), (x.grad, x64.grad.permute(0, 2, 3, 1), 5e-3),
                          (norm.weight.grad, w64.grad, 1e-4), (norm.bias.grad, b64.grad, 1e-4)):
        assert ((got.double() - ref).norm() <= tol * ref.norm()).item()
