"""LayerNorm where a warp changes from one row to groups of rows (2048 rows forward, 1024 backward): either side of each line, row counts that leave
a group partly empty, for every width that has groups.

Bound: outputs are rounded to bf16 (2^-9 of each element, so of the norm; 1e-4 for fp32 before it); sums are fp32 (1e-4)."""
import pytest
import torch

pytestmark = pytest.mark.gpu
OUT = 2.0 ** -9 + 1e-4


def _rel(a, b):
    return ((a.double() - b).norm() / b.norm()).item()


@pytest.mark.parametrize("C", [32, 64, 96, 128, 192, 384])
@pytest.mark.parametrize("rows", [1023, 1024, 1025, 2047, 2048, 2051, 18943])
def test_either_side_of_the_lines(rows, C):
    from terra_b200 import _ext

    ext, gen = _ext.load(), torch.Generator(device="cuda").manual_seed(rows * C)
    x, dy, dres = (torch.randn(rows, C, generator=gen, device="cuda").to(torch.bfloat16) for _ in range(3))
    w, b = (torch.randn(C, generator=gen, device="cuda").to(torch.bfloat16) for _ in range(2))
    whole = torch.full((rows + 8, C), 3.0, device="cuda", dtype=torch.bfloat16)
    y, mean, rstd = whole[:rows], torch.full((rows + 8,), 3.0, device="cuda"), torch.full((rows + 8,), 3.0, device="cuda")
    ext.layernorm_fwd(x, w, b, y, mean, rstd, 1e-5)
    x64, w64, b64 = (t.double().requires_grad_(True) for t in (x, w, b))
    want = torch.nn.functional.layer_norm(x64, (C,), w64, b64, 1e-5)
    assert _rel(y, want.detach()) < OUT
    assert (whole[rows:] == 3).all() and (mean[rows:] == 3).all() and (rstd[rows:] == 3).all()       # nothing behind the last row
    assert (mean[:rows].double() - x.double().mean(1)).abs().max() < 1e-5
    want.backward(dy.double())
    whole = torch.full((rows + 8, C), 3.0, device="cuda", dtype=torch.bfloat16)
    gw, gb = torch.ones(C, device="cuda"), torch.ones(C, device="cuda")
    ext.layernorm_bwd(dy, x, w, mean[:rows], rstd[:rows], whole[:rows], gw, gb, dres)
    assert _rel(whole[:rows], x64.grad + dres.double()) < OUT and (whole[rows:] == 3).all()
    assert _rel(gw - 1, w64.grad) < 1e-4 and _rel(gb - 1, b64.grad) < 1e-4
