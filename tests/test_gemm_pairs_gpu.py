"""CTA pairs of the tcgen05 GEMM with the epilogue through TMA, every epilogue and tile width, at the edges of tiles: rows
that end in the first or the second CTA's half, columns that end inside a chunk's tile, contractions shorter than a k-block;
the single-CTA tiles run the same cases.

Bound: operands are bf16 and exact, sums fp32; the result is rounded once (2^-9), GELU's fit is within 2.6e-5 and its
derivative within 1.2e-4: 0.4 % of the norm is twice the sum."""
import pytest
import torch

pytestmark = pytest.mark.gpu
REL = 4e-3


def _rand(*shape, scale=1.0):
    return (torch.randn(*shape, device="cuda") * scale).to(torch.bfloat16)


def _rel(got, ref):
    return ((got.float() - ref).norm() / ref.norm()).item()


@pytest.mark.parametrize("bn", [1128, 1192, 1256, 128, 192, 256])
@pytest.mark.parametrize("M,N,K", [(1, 64, 8), (128, 192, 64), (129, 200, 72), (300, 384, 200), (511, 1000, 384), (2050, 256, 136)])
@pytest.mark.parametrize("epilogue", ["plain", "bias", "gelu", "residual", "dgelu"])
def test_epilogues(bn, M, N, K, epilogue):
    from terra_b200.ops.gemm import check_status, gemm

    torch.manual_seed(M + N)
    a, w, bias = _rand(M, K), _rand(N, K, scale=K ** -0.5), _rand(N)
    extra = _rand(M, N)
    kw = dict(plain={}, bias=dict(bias=bias), gelu=dict(bias=bias, gelu=True, save_pre=True),
              residual=dict(bias=bias, residual=extra), dgelu=dict(dgelu_aux=extra))[epilogue]
    got = gemm(a, w, bn=bn, **kw)
    check_status("cuda")
    ref = a.float() @ w.float().t()
    if epilogue in ("bias", "gelu", "residual"):
        ref = ref + bias.float()
    if epilogue == "gelu":
        got, pre = got
        assert _rel(pre, ref) < REL
        ref = torch.nn.functional.gelu(ref)
    if epilogue == "residual":
        ref = ref + extra.float()
    if epilogue == "dgelu":
        x = extra.float().requires_grad_(True)
        torch.nn.functional.gelu(x).sum().backward()
        ref = ref * x.grad
    assert _rel(got, ref) < REL


@pytest.mark.parametrize("bn", [1128, 1256, 128, 256])
@pytest.mark.parametrize("M,N,K", [(129, 200, 72), (700, 384, 1152)])
def test_untransposed_weights(bn, M, N, K):
    from terra_b200.ops.gemm import check_status, gemm

    torch.manual_seed(2)
    a, w = _rand(M, K), _rand(K, N, scale=K ** -0.5)
    got = gemm(a, w, b_mn=True, bn=bn)
    check_status("cuda")
    assert _rel(got, a.float() @ w.float()) < REL


@pytest.mark.parametrize("N,K,b_mn", [(1152, 320, False), (384, 320, True), (96, 384, False)])
def test_rule_takes_pairs_for_many_tiles(N, K, b_mn):
    """The smallest product for which the rule takes CTA pairs, the one below it, and one whose last pair holds a single row
    block, each with a ragged last block: the rule's choice and the values."""
    from terra_b200 import _ext
    from terra_b200.ops.gemm import check_status, gemm

    torch.manual_seed(3)
    pairs = lambda blocks: _ext.load().gemm_tile(128 * blocks - 51, N, K, b_mn)[1] == 2
    line = next(b for b in range(1, 2000) if pairs(b))
    odd = next(b for b in range(line | 1, 4000, 2) if pairs(b))
    a = _rand(128 * max(line, odd) - 51, K)
    w = _rand(K, N, scale=K ** -0.5) if b_mn else _rand(N, K, scale=K ** -0.5)
    ref = a.float() @ (w.float() if b_mn else w.float().t())
    for blocks in (line, line - 1, odd):
        assert pairs(blocks) == (blocks != line - 1)
        rows = 128 * blocks - 51
        got = gemm(a[:rows].contiguous(), w, b_mn=b_mn)
        check_status("cuda")
        assert _rel(got, ref[:rows]) < REL


def test_gelu_keeps_its_limits():
    """Large, infinite and NaN pre-activations: x for large x, 0 for small ones, NaN stays NaN; the derivative goes to 1 and 0."""
    from terra_b200.ops.gemm import check_status, gemm

    vals = torch.tensor([0.0, -0.0, 9.0, -9.0, 40.0, -40.0, 3e4, -3e4, float("inf"), float("nan")], device="cuda")
    bias = vals.repeat(32)[:64].to(torch.bfloat16)
    a, w = torch.zeros(128, 64, device="cuda", dtype=torch.bfloat16), torch.zeros(64, 64, device="cuda", dtype=torch.bfloat16)
    act, _ = gemm(a, w, bias=bias, gelu=True, save_pre=True)
    ref = torch.nn.functional.gelu(bias.float())
    ones = torch.eye(64, device="cuda", dtype=torch.bfloat16)
    grad = gemm(torch.ones(128, 64, device="cuda", dtype=torch.bfloat16), ones, dgelu_aux=bias.expand(128, 64).contiguous())
    check_status("cuda")
    assert torch.equal(torch.isnan(act[0]), torch.isnan(ref))
    fine = ~torch.isnan(ref)
    assert torch.allclose(act[0].float()[fine], ref.to(torch.bfloat16).float()[fine], rtol=1e-2, atol=1e-4)
    x = bias.float()
    assert torch.allclose(grad[0].float()[x >= 9], torch.ones_like(x[x >= 9])) and grad[0].float()[x <= -9].abs().max() < 1e-3


@pytest.mark.parametrize("sms", [1, 2, 3])
def test_few_multiprocessors(sms):
    """A product held to a few SMs computes every tile; one SM holds no pair, asked for or not."""
    from terra_b200.ops.gemm import check_status, gemm

    torch.manual_seed(4)
    a, w = _rand(128 * 9 + 1, 64), _rand(384, 64, scale=0.125)
    got = gemm(a, w, sms=sms)
    check_status("cuda")
    assert _rel(got, a.float() @ w.float().t()) < REL
    if sms == 1:
        with pytest.raises(RuntimeError):
            gemm(a, w, sms=1, bn=1128)
