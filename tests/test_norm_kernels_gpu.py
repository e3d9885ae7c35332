"""LayerNorm and GroupNorm+SiLU kernels at the sizes where their layouts change: rows per warp (by the row length and the
number of rows), fewer pixels than a block holds, pixels that do not divide over blocks and threads, channel counts above a
block's width, groups that do not line up with the 16-byte vectors, several samples.

Bound: fp32 arithmetic, one bf16 rounding (2^-9) of each output element; sums over rows in fp32: 0.4 % of the norm."""
import pytest
import torch
import torch.nn.functional as TF

pytestmark = pytest.mark.gpu
REL = 4e-3


def _rand(*shape, scale=1.0):
    return (torch.randn(*shape, device="cuda") * scale).to(torch.bfloat16)


def _rel(got, ref):
    return ((got.float() - ref).norm() / ref.norm()).item()


@pytest.mark.parametrize("C", [32, 40, 64, 96, 128, 192, 384, 640, 768, 1024, 2048])
@pytest.mark.parametrize("rows", [1, 7, 9475, 19001])
@pytest.mark.parametrize("shortcut", [False, True])
def test_layernorm(C, rows, shortcut):
    from terra_b200.ops.blocks import layernorm_bwd_cuda, layernorm_cuda

    torch.manual_seed(C + rows)
    x, dy, dres = _rand(rows, C) + 0.5, _rand(rows, C), _rand(rows, C) if shortcut else None
    w, b = _rand(C) * 0.2 + 1, _rand(C)
    y, mean, rstd = layernorm_cuda(x, w, b)
    gw, gb = torch.ones(C, device="cuda"), torch.ones(C, device="cuda")
    dx = layernorm_bwd_cuda(dy, x, w, mean, rstd, gw, gb, dres=dres)
    xr = x.float().requires_grad_(True)
    wr, br = w.float().requires_grad_(True), b.float().requires_grad_(True)
    ref = TF.layer_norm(xr, (C,), wr, br, 1e-5)
    ref.backward(dy.float())
    assert _rel(y, ref.detach()) < REL and _rel(dx, xr.grad + (dres.float() if shortcut else 0)) < REL
    assert _rel(gw - 1, wr.grad) < REL and _rel(gb - 1, br.grad) < REL          # accumulated on top of what was there


@pytest.mark.parametrize("C", [40, 64, 256, 512, 1536])
def test_layernorm_of_many_rows(C):
    """Row counts that take the larger grids of the backward kernel."""
    test_layernorm(C, 57001, True)


@pytest.mark.parametrize("B,HW,C,groups", [(1, 1, 96, 32), (2, 7, 384, 32), (1, 1000, 64, 32), (3, 20011, 96, 32), (1, 16385, 384, 32),
                                           (2, 333, 1024, 32), (1, 4097, 520, 5)])
@pytest.mark.parametrize("shortcut", [False, True])
def test_groupnorm_silu(B, HW, C, groups, shortcut):
    from terra_b200.ops.conv import groupnorm_silu

    torch.manual_seed(HW + C)
    gn = torch.nn.GroupNorm(groups, C).cuda()
    with torch.no_grad():
        gn.weight.copy_(_rand(C) * 0.2 + 1)
        gn.bias.copy_(_rand(C))
    x, dy, res = (_rand(B, 1, HW, C) + 0.3).requires_grad_(True), _rand(B, 1, HW, C), _rand(B, 1, HW, C)
    y = groupnorm_silu(x, gn, residual=res if shortcut else None)
    y.backward(dy)
    got = (x.grad, gn.weight.grad.clone(), gn.bias.grad.clone())
    gn.zero_grad()
    xr = x.detach().float().requires_grad_(True)
    ref = TF.silu(TF.group_norm(xr.permute(0, 3, 1, 2), groups, gn.weight, gn.bias, 1e-5)).permute(0, 2, 3, 1)
    ref.backward(dy.float())
    # one pixel of a three-channel group: the gradients are differences of nearly equal terms
    rel = 2e-2 if HW == 1 else REL
    assert _rel(y, ref.detach() + (res.float() if shortcut else 0)) < REL
    assert _rel(got[0], xr.grad) < rel and _rel(got[1], gn.weight.grad) < rel and _rel(got[2], gn.bias.grad) < rel


@pytest.mark.parametrize("B,HW", [(0, 16), (2, 0)])
def test_groupnorm_refuses_empty_images(B, HW):
    """The four launchers divide by the sizes; an empty batch or image is an error that Python sees."""
    from terra_b200 import _ext
    from terra_b200.ops.conv import groupnorm_silu

    C, G, ext = 64, 8, _ext.load()
    x, w = torch.empty(B, HW, C, device="cuda", dtype=torch.bfloat16), _rand(C)
    stats, red = torch.zeros(B, G, 2, device="cuda"), torch.zeros(B, C, 2, device="cuda")
    for call in (lambda: ext.groupnorm_stats(x, stats, G),
                 lambda: ext.groupnorm_silu_apply(x, stats, w, w, None, x.clone(), G),
                 lambda: ext.groupnorm_silu_bwd_reduce(x, x, stats, w, w, red, G, None, None),
                 lambda: ext.groupnorm_silu_bwd_apply(x, x, stats, red, w, w, x.clone(), G, 1.0),
                 lambda: groupnorm_silu(x.view(B, 1, HW, C), torch.nn.GroupNorm(G, C).cuda())):
        with pytest.raises(RuntimeError):
            call()
