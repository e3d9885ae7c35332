"""Norm kernels whose loads run ahead through shared memory: fewer pixels or rows than a round, a round's remainder, more column vectors than
lanes, channel counts whose last vector round is partial, gradients that are no whole 16-byte vectors (the scalar ends), an odd group count.

Bound: outputs are rounded to bf16 (2^-9); sums are fp32 in another order (1e-5 of the norm, 1e-4 where a few cancel)."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _rand(gen, *shape):
    return torch.randn(*shape, generator=gen, device="cuda").to(torch.bfloat16)


def _rel(a, b):
    return ((a.double() - b.double()).norm() / b.double().norm().clamp_min(1e-6)).item()


@pytest.mark.parametrize("rows", [1, 3, 5, 17, 1777, 9473])
@pytest.mark.parametrize("C", [8, 72, 96, 192, 384, 520, 1024, 1200, 2048])
@pytest.mark.parametrize("shortcut,offset", [(True, 0), (False, 1)])
def test_layernorm_backward(rows, C, shortcut, offset):
    from terra_b200 import _ext

    gen = torch.Generator(device="cuda").manual_seed(rows + C)
    x, dy, dres = (_rand(gen, rows, C) for _ in range(3))
    w = (1 + 0.1 * torch.randn(C, generator=gen, device="cuda")).to(torch.bfloat16)
    x64 = x.double().requires_grad_(True)
    w64 = w.double().requires_grad_(True)
    b64 = torch.zeros(C, device="cuda", dtype=torch.float64, requires_grad=True)
    torch.nn.functional.layer_norm(x64, (C,), w64, b64, 1e-5).backward(dy.double())
    mean = x.double().mean(1)
    rstd = (x.double().var(1, unbiased=False) + 1e-5).rsqrt()
    dx = torch.empty_like(x)
    gw, gb = (torch.ones(C + offset, device="cuda")[offset:] for _ in range(2))
    _ext.load().layernorm_bwd(dy, x, w, mean.float(), rstd.float(), dx, gw, gb, dres if shortcut else None)
    want = x64.grad + (dres.double() if shortcut else 0)
    assert _rel(dx, want) < 5e-3 and _rel(gw - 1, w64.grad) < 1e-4 and _rel(gb - 1, b64.grad) < 1e-4


@pytest.mark.parametrize("B,HW,C,groups", [(1, 1, 8, 1), (1, 2, 96, 3), (2, 41, 72, 9), (1, 4001, 192, 32), (3, 700, 520, 5), (1, 90001, 384, 32)])
@pytest.mark.parametrize("shortcut,offset", [(True, 0), (False, 1)])
def test_groupnorm(B, HW, C, groups, shortcut, offset):
    from terra_b200 import _ext

    ext, gen = _ext.load(), torch.Generator(device="cuda").manual_seed(HW + C)
    x, dy, res = (_rand(gen, B, HW, C) for _ in range(3))
    g, b = (1 + 0.1 * torch.randn(C, generator=gen, device="cuda")).to(torch.bfloat16), (0.1 * torch.randn(C, generator=gen, device="cuda")).to(torch.bfloat16)
    sums, stats = torch.zeros(B, groups, 2, device="cuda"), torch.empty(B, groups, 2, device="cuda")
    ext.groupnorm_stats(x, sums, groups)
    t = x.double().view(B, HW, groups, C // groups)
    assert _rel(sums[..., 0], t.sum((1, 3))) < 1e-4 and _rel(sums[..., 1], (t * t).sum((1, 3))) < 1e-5
    count = HW * (C // groups)
    ext.groupnorm_finalize(sums, stats, 1.0 / count, 1e-5)
    y, dx, red = torch.empty_like(x), torch.empty_like(x), torch.zeros(B, C, 2, device="cuda")
    ext.groupnorm_silu_apply(x, stats, g, b, res if shortcut else None, y, groups)
    gg, gb = (torch.ones(C + offset, device="cuda")[offset:] for _ in range(2))
    ext.groupnorm_silu_bwd_reduce(dy, x, stats, g, b, red, groups, gg, gb)
    ext.groupnorm_silu_bwd_apply(dy, x, stats, red, g, b, dx, groups, 1.0 / count)
    x64, g64, b64 = (v.double().requires_grad_(True) for v in (x, g, b))
    t = x64.view(B, HW, groups, C // groups)
    mu = t.mean((1, 3), keepdim=True)
    z = ((t - mu) * ((t - mu).square().mean((1, 3), keepdim=True) + 1e-5).rsqrt()).reshape(B, HW, C) * g64 + b64
    want = torch.nn.functional.silu(z)
    want.backward(dy.double())
    assert _rel(y, want.detach() + (res.double() if shortcut else 0)) < 5e-3
    assert _rel(gg - 1, g64.grad) < 2e-4 and _rel(gb - 1, b64.grad) < 1e-4
    if count > 1:
        assert _rel(dx, x64.grad) < 1e-2
