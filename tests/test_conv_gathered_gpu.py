"""The strided forms of the implicit GEMM: input gradient of the stride-2 convolution and the three products of the 2x2
transposed convolution, against fp32 PyTorch, at ragged widths (tiles are 128 pixels wide), odd heights, channel counts with
a padded chunk, sizes that take CTA pairs (there the 3x3 forms as well), and the channel counts that keep the general path.

Bound: bf16 operands are exact, sums fp32, one rounding of the result: 2^-9 = 0.2 % of the norm; the tests allow 0.4 %."""
import pytest
import torch
import torch.nn.functional as TF

pytestmark = pytest.mark.gpu
REL = 4e-3


def _rand(*shape, scale=1.0):
    return (torch.randn(*shape, device="cuda") * scale).to(torch.bfloat16)


def _rel(got, ref):
    return ((got.float() - ref.float()).norm() / ref.float().norm()).item()


@pytest.mark.parametrize("B,H,W,Cin,Cout", [
    (1, 2, 2, 64, 64), (1, 1, 4, 32, 64), (2, 13, 200, 96, 96), (1, 33, 258, 96, 192), (1, 8, 16, 40, 72), (1, 64, 300, 384, 384),
    (1, 512, 512, 192, 64),                # two tiles per image row, many rounds
    (1, 6, 20, 64, 1024),                  # more channels than the tap table holds: columns and gather
])
def test_stride2_input_gradient(B, H, W, Cin, Cout):
    from terra_b200.ops.conv import _conv3x3_s2_dgrad
    from terra_b200.ops.gemm import check_status

    torch.manual_seed(0)
    w, dy = _rand(Cout, Cin, 3, 3, scale=0.05), _rand(B, (H + 1) // 2, W // 2, Cout)
    dx = _conv3x3_s2_dgrad(dy, w, H, W, None)
    check_status("cuda")
    x = torch.zeros(B, Cin, H, W, device="cuda", requires_grad=True)
    TF.conv2d(x, w.float(), stride=2, padding=1).backward(dy.float().permute(0, 3, 1, 2))
    # the general path rounds its columns to bf16 as well
    assert _rel(dx.permute(0, 3, 1, 2), x.grad) < (REL if Cout < 1000 else 2 * REL)


@pytest.mark.parametrize("B,H,W,Cin,Cout", [
    (1, 1, 1, 64, 64), (1, 16, 24, 96, 96), (2, 7, 130, 64, 64), (1, 5, 3, 128, 32), (1, 9, 33, 40, 96), (1, 20, 257, 192, 384),
    (1, 256, 256, 64, 192),                # two tiles per image row, many rounds
    (1, 6, 10, 64, 40),                    # phases that end inside a unit of the epilogue
    (1, 149, 24, 64, 64), (2, 80, 3, 64, 96),            # narrow images: GEMM and permuted copy
    (1, 3, 5, 64, 2056),                   # more channels than the tap table holds: GEMM and permuted copy
])
def test_transposed_convolution(B, H, W, Cin, Cout):
    from terra_b200.ops.conv import conv_transpose2x2
    from terra_b200.ops.gemm import check_status
    from terra_b200.utils.flat_params import ParamArena

    torch.manual_seed(1)
    conv = torch.nn.ConvTranspose2d(Cin, Cout, 2, stride=2).cuda()
    with torch.no_grad():
        for p in conv.parameters():
            p.copy_(p.to(torch.bfloat16).float())
    ref = torch.nn.ConvTranspose2d(Cin, Cout, 2, stride=2).cuda()
    ref.load_state_dict(conv.state_dict())
    plain = torch.nn.ConvTranspose2d(Cin, Cout, 2, stride=2).cuda()        # parameters outside an arena
    plain.load_state_dict(conv.state_dict())
    ParamArena(conv)
    x, dy = _rand(B, H, W, Cin), _rand(B, 2 * H, 2 * W, Cout)
    xr = x.float().permute(0, 3, 1, 2).detach().requires_grad_(True)
    yr = ref(xr)
    yr.backward(dy.float().permute(0, 3, 1, 2))
    for m in (conv, plain):
        xc = x.clone().requires_grad_(True)
        y = conv_transpose2x2(xc, m)
        y.backward(dy)
        check_status("cuda")
        assert _rel(y.permute(0, 3, 1, 2), yr) < REL and _rel(xc.grad.permute(0, 3, 1, 2), xr.grad) < REL
        assert _rel(m.weight.grad, ref.weight.grad) < REL and _rel(m.bias.grad, ref.bias.grad) < REL


def _pairs(row_tiles, N, k_blocks):
    from terra_b200 import _ext

    return _ext.load().gemm_tile(128 * row_tiles, N, 64 * k_blocks, gathered=True)[1] == 2


@pytest.mark.parametrize("B,H,W,stride,halos", [
    (1, 1201, 100, 1, False), (1, 601, 200, 1, True), (3, 401, 100, 1, False),      # 1201, 1202, 1203 row tiles
    (1, 2401, 200, 2, False), (3, 801, 200, 2, True),                                # 1201, 1203
])
def test_3x3_convolutions_on_pairs(B, H, W, stride, halos):
    """Forward with bias, and the input gradient of stride 1 (the same kernel on other weights), on CTA pairs: counts of row tiles
    that leave half a pair over, several samples, rows from a neighbour above and below."""
    from terra_b200 import _ext
    from terra_b200.ops.conv import pack_conv3x3_weight, pack_conv3x3_weight_dgrad
    from terra_b200.ops.gemm import check_status, status_word

    torch.manual_seed(6)
    Cin, Cout, ext = 64, 192, _ext.load()
    Ho, Wo = -(-H // stride), W // stride
    assert _pairs(-(-Wo // 128) * Ho * B, Cout, 9)
    x, w, bias = _rand(B, H, W, Cin), _rand(Cout, Cin, 3, 3, scale=0.04), _rand(Cout)
    lo, hi = (_rand(B, 1, W, Cin), _rand(B, 1, W, Cin)) if halos else (None, None)
    y = torch.empty(B, Ho, Wo, Cout, device="cuda", dtype=torch.bfloat16)
    ext.conv3x3_fwd(x, pack_conv3x3_weight(w), y, stride, 1, bias, None, status_word("cuda"), lo, hi)     # 1: with bias
    check_status("cuda")
    zero = torch.zeros_like(x[:, :1])
    whole = torch.cat([zero if lo is None else lo, x, zero if hi is None else hi], dim=1).float().permute(0, 3, 1, 2)
    ref = TF.conv2d(whole, w.float(), bias.float(), stride=stride, padding=(0, 1))[:, :, :Ho]
    assert _rel(y.permute(0, 3, 1, 2), ref) < REL
    if stride == 1:
        wt = _rand(Cin, Cout, 3, 3, scale=0.04)       # of the convolution whose input has the 192 channels
        dx = torch.empty(B, H, W, Cout, device="cuda", dtype=torch.bfloat16)
        ext.conv3x3_fwd(x, pack_conv3x3_weight_dgrad(wt), dx, 1, 0, None, None, status_word("cuda"), lo, hi)
        check_status("cuda")
        ref = TF.conv_transpose2d(whole, wt.float(), padding=1)[:, :, 1:-1]
        assert _rel(dx.permute(0, 3, 1, 2), ref) < REL


def test_strided_forms_on_pairs():
    """The input gradient of the stride-2 convolution and the transposed convolution with half a pair left over."""
    from terra_b200 import _ext
    from terra_b200.ops import conv
    from terra_b200.ops.gemm import check_status, status_word

    torch.manual_seed(7)
    ext, B, H, W = _ext.load(), 3, 401, 100              # 1203 row tiles
    Cin, Cout = 192, 256
    assert _pairs(4 * B * H, Cin, 9)
    w, dy = _rand(Cout, Cin, 3, 3, scale=0.04), _rand(B, H, W, Cout)
    dx = torch.empty(B, 2 * H, 2 * W, Cin, device="cuda", dtype=torch.bfloat16)
    ext.conv3x3_s2_dgrad(dy, conv.pack_conv3x3_weight_s2_dgrad(w), dx, status_word("cuda"))
    check_status("cuda")
    ref = TF.conv_transpose2d(dy.float().permute(0, 3, 1, 2), w.float(), stride=2, padding=1, output_padding=1)
    assert _rel(dx.permute(0, 3, 1, 2), ref) < REL
    Cin, Cout = 384, 192
    assert _pairs(B * H, 4 * Cout, Cin // 64) and _pairs(B * H, Cin, 4 * Cout // 64)
    x, w, bias = _rand(B, H, W, Cin), _rand(Cin, Cout, 2, 2, scale=0.05), _rand(Cout)
    y = torch.empty(B, 2 * H, 2 * W, Cout, device="cuda", dtype=torch.bfloat16)
    ext.convt2x2(0, x, conv._pack_taps(w, 4, 1, Cout, 4, Cin, 4 * Cout, (0,)), bias.repeat(4), y, status_word("cuda"))
    dx = torch.empty_like(x)
    ext.convt2x2(1, y, conv._pack_taps(w, 1, 0, Cin, 4 * Cout, Cout, 4, range(4)), None, dx, status_word("cuda"))
    check_status("cuda")
    ref = TF.conv_transpose2d(x.float().permute(0, 3, 1, 2), w.float(), bias.float(), stride=2)
    assert _rel(y.permute(0, 3, 1, 2), ref) < REL
    ref = TF.conv2d(y.float().permute(0, 3, 1, 2), w.float(), stride=2)
    assert _rel(dx.permute(0, 3, 1, 2), ref) < REL


_BY_LANE = """
import sys, torch
from terra_b200 import _ext
from terra_b200.ops import conv
ext = _ext.load()
assert not ext.gemm_tma_epilogue()
torch.manual_seed(5)
mods = [torch.nn.Conv2d(96, 72, 3, padding=1), torch.nn.Conv2d(96, 72, 3, stride=2, padding=1), torch.nn.ConvTranspose2d(96, 72, 2, stride=2)]
out = []
for m, op in zip(mods, (conv.conv3x3, lambda x, m: conv.conv3x3(x, m, 2), conv.conv_transpose2x2)):
    m = m.cuda()
    with torch.no_grad():
        for p in m.parameters():
            p.copy_(p.to(torch.bfloat16).float())
    x = torch.randn(2, 18, 140, 96, device="cuda").to(torch.bfloat16).requires_grad_(True)
    y = op(x, m)
    dy = torch.randn(y.shape, device="cuda").to(torch.bfloat16)
    y.backward(dy)
    xr = x.detach().float().permute(0, 3, 1, 2).requires_grad_(True)
    yr = m(xr)
    yr.backward(dy.float().permute(0, 3, 1, 2))
    rel = lambda a, b: ((a.float().permute(0, 3, 1, 2) - b).norm() / b.norm()).item()
    out += [rel(y.detach(), yr.detach()), rel(x.grad, xr.grad)]
print(*out)
"""


def test_convolutions_without_the_tma_epilogue():
    """TERRA_GEMM_TMA_EPILOGUE=0 reaches the convolutions: per-lane stores, or the general path where there are none (columns
    that are rounded to bf16 as well for the stride-2 input gradient)."""
    import os
    import subprocess
    import sys

    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    r = subprocess.run([sys.executable, "-c", _BY_LANE], cwd=root, env=dict(os.environ, TERRA_GEMM_TMA_EPILOGUE="0"),
                       capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stderr
    errors = [float(v) for v in r.stdout.split()]
    assert len(errors) == 6 and max(errors[:3] + errors[4:]) < REL and errors[3] < 2 * REL, errors
