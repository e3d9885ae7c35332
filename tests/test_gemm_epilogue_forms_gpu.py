"""Every form of the GEMM epilogue that goes through TMA, at the sizes where its units, buffers and tiles end."""
import pytest
import torch

from terra_b200.ops.gemm import check_status, gemm

pytestmark = pytest.mark.gpu

# rows: below / at / behind a 128-row block and a 256-row pair; columns: inside a 32- and a 64-column unit, units of two
# tiles; contractions on both sides of the 12 k-blocks that separate one input buffer from two
SIZES = [(1, 8, 8), (127, 72, 64), (128, 192, 384), (257, 328, 392), (300, 200, 768), (300, 384, 776), (1000, 576, 1000)]
FORMS = ["plain", "bias", "bias32", "gelu_pre", "gelu", "residual", "residual_nobias", "dgelu", "alpha"]


def _data(m, n, k, seed=0):
    gen = torch.Generator(device="cuda").manual_seed(seed)
    r = lambda *s: torch.randn(*s, generator=gen, device="cuda").to(torch.bfloat16)
    return r(m, k), r(n, k) * k ** -0.5, r(n), r(m, n) * 3


@pytest.mark.parametrize("bn", [0, 128, 192, 256, 1128, 1192, 1256, 1384])
@pytest.mark.parametrize("form", FORMS)
def test_forms_against_64_bits(form, bn):
    for m, n, k in SIZES:
        a, w, bias, other = _data(m, n, k)
        acc = a.double() @ w.double().t()
        pre_want = None
        kw = dict(bn=bn)
        if form == "plain":
            want = acc
        elif form in ("bias", "bias32"):
            kw["bias"] = bias if form == "bias" else bias.float()
            want = acc + bias.double()
        elif form in ("gelu", "gelu_pre"):
            kw.update(bias=bias, gelu=True, save_pre=form == "gelu_pre")
            pre_want = acc + bias.double()
            want = torch.nn.functional.gelu(pre_want)
        elif form in ("residual", "residual_nobias"):
            kw["residual"] = other
            want = acc + other.double()
            if form == "residual":
                kw["bias"] = bias
                want = want + bias.double()
        elif form == "dgelu":
            kw["dgelu_aux"] = other
            x = other.double()
            want = acc * (0.5 * (1 + torch.erf(x / 2 ** 0.5)) + x * torch.exp(-x * x / 2) / (2 * torch.pi) ** 0.5)
        else:
            kw["alpha"] = 0.5
            want = acc * 0.5
        got = gemm(a, w, **kw)
        if form == "gelu_pre":
            got, pre = got
            assert ((pre.double() - pre_want).abs() <= pre_want.abs() * 2 ** -8 + 1e-5).all(), (m, n, k)
        # half a bf16 step of the result (2^-9, taken twice); fp32 sums of values near 1 (1e-5); the fit of GELU (2.6e-5) and of
        # its derivative (1.2e-4 times the product)
        bound = want.abs() * 2 ** -8 + {"gelu": 5e-5, "gelu_pre": 5e-5}.get(form, 1e-5)
        if form == "dgelu":
            bound = bound + acc.abs() * 1.5e-4
        assert ((got.double() - want).abs() <= bound).all(), (m, n, k, ((got.double() - want).abs() - bound).max().item())
    check_status("cuda")


def test_gelu_derivative_outside_the_fit():
    """Beyond the clamp (|x| > 8, infinities) the derivative is 0 or 1. (The build with the erf form itself gives NaN at infinity, as
    PyTorch does, so it is asked for finite values only.)"""
    from terra_b200 import _ext

    far = 1e30 if _ext.GELU_EXACT else float("inf")
    x = torch.tensor([-1e30, -9.0, -8.0, 8.0, 9.0, 1e30, far, -far], device="cuda").to(torch.bfloat16)
    eye = torch.eye(8, device="cuda").to(torch.bfloat16)
    got = gemm(torch.ones(8, 8, device="cuda").to(torch.bfloat16), eye, dgelu_aux=x.repeat(8, 1)).float()
    want = (x.float() > 0).float().repeat(8, 1)
    assert (got - want).abs().max() < 1e-3


@pytest.mark.parametrize("m,n,k", [(1, 8, 64), (255, 264, 64), (256, 384, 128), (1000, 392, 1000), (20000, 768, 200), (40000, 384, 1160)])
def test_tiles_384_wide_with_the_weight_as_stored(m, n, k):
    """Input gradients: B MN-major, whose halves of 256 and of 128 columns are whole boxes."""
    a, w, _, _ = _data(m, n, k, 1)
    got = gemm(a, w.t().contiguous(), b_mn=True, bn=1384)
    want = a.double() @ w.double().t()
    assert ((got.double() - want).abs() <= want.abs() * 2 ** -8 + 1e-5).all()      # half a bf16 step, fp32 sums of values near 1
    check_status("cuda")


@pytest.mark.parametrize("rows,n,k,split", [(64, 8, 264, 1), (1000, 256, 384, 3), (5000, 400, 392, 7), (30000, 1528, 768, 11)])
@pytest.mark.parametrize("bn,sums", [(1384, True), (1384, False), (1256, False)])
def test_weight_gradients_of_pairs(rows, n, k, split, bn, sums):
    """Both operands MN-major, the column sums from a 32-column MMA over the pair. fp32 sums in another order: 1e-5 of the norm."""
    gen = torch.Generator(device="cuda").manual_seed(rows)
    dy, x = (torch.randn(rows, c, generator=gen, device="cuda").to(torch.bfloat16) for c in (n, k))
    gw, gb = torch.ones(n, k, device="cuda"), torch.ones(n, device="cuda")
    gemm(dy, x, a_mn=True, b_mn=True, out=gw, accumulate=True, split_k=split, bn=bn, colsum=gb if sums else None)
    check_status("cuda")
    rel = lambda got, want: ((got.double() - want).norm() / want.norm()).item()
    assert rel(gw - 1, dy.double().t() @ x.double()) < 1e-5
    if sums:
        assert rel(gb, 1 + dy.double().sum(0)) < 1e-5


@pytest.mark.parametrize("m,n,k", [(104, 64, 64), (1000, 384, 136), (304, 1024, 200)])      # (rows a multiple of 8: a pitch)
@pytest.mark.parametrize("bn", [384, 100])
def test_a_width_that_single_tiles_do_not_have_falls_back_to_the_rule(m, n, k, bn):
    """Only a pair (1384) has tiles of 384 columns; any other width asked for is left to the rule, forward and for weight gradients."""
    a, w, _, _ = _data(m, n, k, 1)
    want = a.double() @ w.double().t()
    assert ((gemm(a, w, bn=bn).double() - want).abs() <= want.abs() * 2 ** -8 + 1e-5).all()      # half a bf16 step, fp32 sums
    gw = gemm(a.t().contiguous(), w.t().contiguous(), a_mn=True, b_mn=True, out_f32=True, accumulate=True, bn=bn)
    assert ((gw.double() - want).norm() / want.norm()).item() < 1e-5
    check_status("cuda")
