"""The layers as C++ autograd nodes against the Python nodes they stand for: outputs and input gradients bit for bit, parameter
gradients to the order of their fp32 atomics (1e-5 of the norm); and the cases that stay with the Python nodes."""
import pytest
import torch

from terra_b200.ops import blocks, conv
from terra_b200.ops.gemm import check_status
from terra_b200.utils.flat_params import ParamArena

pytestmark = pytest.mark.gpu


def _rel(a, b):
    return ((a - b).norm() / b.norm().clamp_min(1e-20)).item()


def _layer(kind, dim=96):
    torch.manual_seed(3)
    r = lambda *s: torch.randn(*s, device="cuda").to(torch.bfloat16)
    if kind.startswith("linear"):
        m = torch.nn.Linear(dim, 72).cuda()
        x, res = r(333, dim), r(333, 72)
        run = {"linear": lambda t, u: blocks.linear(t, m), "linear_res": lambda t, u: blocks.linear(t, m, residual=u),
               "linear_no_dx": lambda t, u: blocks.linear(t, m, need_dx=False)}[kind]
    elif kind.startswith("conv"):
        stride = 2 if kind == "conv_s2" else 1
        m, x, res = torch.nn.Conv2d(dim, 72, 3, stride=stride, padding=1).cuda(), r(2, 10, 140, dim), None
        run = lambda t, u: conv.conv3x3(t, m, stride)
    elif kind == "up":
        m, x, res = torch.nn.ConvTranspose2d(dim, 72, 2, stride=2).cuda(), r(2, 5, 140, dim), None
        run = lambda t, u: conv.conv_transpose2x2(t, m)
    else:
        m, x = torch.nn.GroupNorm(8, dim).cuda(), r(2, 9, 30, dim)
        res = r(2, 9, 30, dim)
        run = (lambda t, u: conv.groupnorm_silu(t, m, residual=u)) if kind == "gn_res" else (lambda t, u: conv.groupnorm_silu(t, m))
    return m, x, res, run


@pytest.mark.parametrize("fused", [True, False])
@pytest.mark.parametrize("kind", ["linear", "linear_res", "linear_no_dx", "conv", "conv_s2", "up", "gn", "gn_res"])
def test_against_the_python_node(monkeypatch, kind, fused):
    monkeypatch.setattr(blocks, "FUSE_BIAS_GRAD", fused)
    monkeypatch.setattr(conv, "FUSE_BIAS_GRAD", fused)
    m, x, res, run = _layer(kind)
    arena, got = ParamArena(m), []
    for native in (True, False):
        for mod in (blocks, conv):
            monkeypatch.setattr(mod, "native_node", (lambda grads=(): True) if native else (lambda grads=(): False))
        arena.zero_grad()
        t = x.clone().requires_grad_(True)
        u = None if res is None else res.clone().requires_grad_(True)
        y = run(t, u)
        torch.manual_seed(4)
        y.backward(torch.randn_like(y))
        got.append((y.detach(), t.grad, None if u is None else u.grad, arena.grad.clone(), type(y.grad_fn).__name__))
        with torch.no_grad():
            assert _rel(run(x, res).float(), got[-1][0].float()) < 1e-3
    check_status("cuda")
    (y0, dx0, du0, g0, n0), (y1, dx1, du1, g1, n1) = got
    # (GroupNorm's statistics are fp32 atomics too: half a bf16 step where their order moves a rounding)
    same = (lambda a, b: _rel(a.float(), b.float()) < 1e-3) if kind.startswith("gn") else torch.equal
    assert n0 != n1 and same(y0, y1)
    for a, b in ((dx0, dx1), (du0, du1)):
        assert (a is None) == (b is None) and (a is None or same(a, b))
    assert _rel(g0, g1) < 1e-5


@pytest.mark.parametrize("kind", ["linear", "conv", "up", "gn"])
def test_backward_without_an_input_gradient_and_a_freed_graph(kind):
    m, x, _, run = _layer(kind)
    arena = ParamArena(m)
    arena.zero_grad()
    y = run(x, None)
    y.backward(torch.ones_like(y))
    assert arena.grad.abs().sum() > 0
    with pytest.raises(RuntimeError):
        y.backward(torch.ones_like(y))


@pytest.mark.parametrize("kind", ["linear", "conv", "gn"])
def test_transforms_and_forward_mode_are_refused(kind):
    m, x, _, run = _layer(kind)
    ParamArena(m)
    with pytest.raises(RuntimeError):
        torch.func.vmap(lambda t: run(t, None))(x[None])
    with pytest.raises((RuntimeError, NotImplementedError)):
        torch.func.jvp(lambda t: run(t, None), (x,), (torch.ones_like(x),))
    import torch.autograd.forward_ad as fwd

    with pytest.raises((RuntimeError, NotImplementedError)), fwd.dual_level():
        run(fwd.make_dual(x, torch.ones_like(x)), None)


def test_a_trace_is_refused():
    """The weights' working copies are constants to a trace, gradient accumulators among them."""
    m, x, _, run = _layer("linear")
    ParamArena(m)
    with pytest.raises(RuntimeError):
        torch.jit.trace(lambda t: run(t, None), (x,), check_trace=False)


def test_inference_without_gradient_accumulators():
    m, x, _, run = _layer("linear")
    arena = ParamArena(m)
    want = run(x, None).detach()
    for p in arena.params:
        p.grad = None
    with torch.no_grad():
        assert torch.equal(run(x, None), want)


@pytest.mark.parametrize("fused", [True, False])
@pytest.mark.parametrize("change", ["dropped", "one dropped", "bound anew"])
@pytest.mark.parametrize("kind", ["conv", "conv_s2", "up", "gn"])
def test_gradients_go_where_the_parameters_point_in_the_backward_pass(monkeypatch, kind, change, fused):
    """`zero_grad(set_to_none=True)` or another accumulator between the forward and the backward pass."""
    monkeypatch.setattr(conv, "FUSE_BIAS_GRAD", fused)
    m, x, _, run = _layer(kind)
    arena = ParamArena(m)

    def backward(t, between):
        arena.zero_grad()
        y = run(t, None)
        between()
        torch.manual_seed(4)
        y.backward(torch.randn_like(y))
        return [p.grad.clone() for p in m.parameters()]

    def drop():
        for p in list(m.parameters())[:1 if change == "one dropped" else 2]:
            p.grad = None

    def rebind():
        for p in m.parameters():
            p.grad = torch.full_like(p, 2.0)

    want = backward(x.clone().requires_grad_(True), lambda: None)
    got = backward(x.clone().requires_grad_(True), rebind if change == "bound anew" else drop)
    for p, a, b in zip(m.parameters(), got, want):
        assert a.shape == p.shape and _rel(a - (2.0 if change == "bound anew" else 0.0), b) < 1e-5
    if change != "one dropped":
        assert not arena.grad.any()      # what the parameters no longer point to stays as it was
    check_status("cuda")


def test_a_residual_with_the_rows_of_several_samples():
    m, x, res, _ = _layer("linear_res")
    ParamArena(m)
    x, res = x[:330], res[:330]
    want = blocks.linear(x, m, residual=res)
    u = res.view(2, 165, 72).detach().requires_grad_(True)
    y = blocks.linear(x, m, residual=u)
    assert torch.equal(y, want)
    y.backward(torch.ones_like(y))
    assert u.grad.shape == u.shape and (u.grad == 1).all()
    for wrong in (res[:200], res.view(2, 165, 72)[:, :100]):      # (rows that are not there are not read)
        with pytest.raises(RuntimeError):
            blocks.linear(x, m, residual=wrong)
    check_status("cuda")
