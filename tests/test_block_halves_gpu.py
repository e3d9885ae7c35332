"""The native attention half against the same launches made one by one from Python: outputs and input gradients bit for bit,
parameter gradients to the order of their fp32 atomics (1e-5 of the norm); with and without a bias table, several samples,
widths with partial tiles, rows given as a pitched weight-gradient operand. The native MLP half likewise, and against fp32."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _rel(a, b):
    return ((a - b).norm() / b.norm().clamp_min(1e-20)).item()


@pytest.mark.parametrize("B,nWh,nWw,window,dim,heads,shifted,table", [
    (1, 2, 4, (8, 8), 96, 3, True, True), (2, 3, 2, (7, 7), 64, 2, True, False), (1, 2, 3, (8, 12), 192, 12, False, True),
    (1, 9, 11, (8, 8), 384, 6, True, True),
])
def test_attention_half(monkeypatch, B, nWh, nWw, window, dim, heads, shifted, table):
    from terra_b200.models.layers import SwinAttentionHalf
    from terra_b200.ops import blocks
    from terra_b200.ops.attention import WindowGeometry
    from terra_b200.ops.gemm import check_status
    from terra_b200.utils.flat_params import ParamArena

    torch.manual_seed(0)
    mod = SwinAttentionHalf(int(shifted), dim, window, heads, use_relative_position_bias=table).cuda()
    arena = ParamArena(mod)
    geo = WindowGeometry(B, nWh, nWw, *window)
    x = torch.randn(geo.rows_local, dim, device="cuda").to(torch.bfloat16)
    dy = torch.randn_like(x)
    got = []
    for native in (True, False):
        if not native:
            monkeypatch.setattr(blocks, "_native_half", lambda *a: False)
        arena.zero_grad()
        t = x.clone().requires_grad_(True)
        y = blocks.attention_half(t, mod, geo, shifted)
        y.backward(dy)
        check_status("cuda")
        got.append((y.detach(), t.grad, arena.grad.clone()))
    assert torch.equal(got[0][0], got[1][0]) and torch.equal(got[0][1], got[1][1])
    assert _rel(got[0][2], got[1][2]) < 1e-5


@pytest.mark.parametrize("dim,rows", [(96, 512), (64, 1), (72, 333), (192, 4001), (384, 20000)])
def test_mlp_half(monkeypatch, dim, rows):
    from terra_b200.ops import blocks
    from terra_b200.ops.gemm import check_status

    mod, arena, x = _mlp(dim, rows)
    dy = torch.randn_like(x)
    got = []
    for native in (True, False):
        monkeypatch.setattr(blocks, "_LAUNCHES_OBSERVED", not native)
        arena.zero_grad()
        t = x.clone().requires_grad_(True)
        y = blocks.mlp_half(t, mod)
        y.backward(dy)
        check_status("cuda")
        got.append((y.detach(), t.grad, arena.grad.clone()))
    assert torch.equal(got[0][0], got[1][0]) and torch.equal(got[0][1], got[1][1])
    assert _rel(got[0][2], got[1][2]) < 1e-5
    # and against the layer in fp32 (bf16 weights; three roundings of 2^-9 along the way, and the GELU fit's 2.6e-5)
    m = {k: v.to(torch.bfloat16).float().requires_grad_(True) for k, v in mod.state_dict().items()}
    t = x.float().requires_grad_(True)
    xn = torch.nn.functional.layer_norm(t, (dim,), m["norm2.weight"], m["norm2.bias"], 1e-5)
    act = torch.nn.functional.gelu(xn @ m["fc1.weight"].t() + m["fc1.bias"])
    ref = t + act @ m["fc2.weight"].t() + m["fc2.bias"]
    ref.backward(dy.float())
    assert _rel(got[0][0].float(), ref.detach()) < 8e-3 and _rel(got[0][1].float(), t.grad) < 8e-3
    for name, p in mod.named_parameters():
        assert _rel(p.grad, m[name].grad) < 1e-2, name


_OBSERVED = """
import sys, torch
names = []
torch.cuda.nvtx.range_push, torch.cuda.nvtx.range_pop = names.append, lambda: None
from terra_b200.models.layers import MlpHalf, SwinAttentionHalf
from terra_b200.ops import blocks
from terra_b200.ops.attention import WindowGeometry
from terra_b200.utils.flat_params import ParamArena
geo = WindowGeometry(1, 2, 2, 8, 8)
attn, mlp = SwinAttentionHalf(1, 64, (8, 8), 2, use_relative_position_bias=True).cuda(), MlpHalf(64, 256).cuda()
for m, run in ((attn, lambda x: blocks.attention_half(x, attn, geo, True)), (mlp, lambda x: blocks.mlp_half(x, mlp))):
    ParamArena(m)
    x = torch.randn(geo.rows_local, 64, device="cuda").to(torch.bfloat16).requires_grad_(True)
    run(x).backward(torch.ones_like(x))
print(names.count("terra.gemm"), names.count("terra.layernorm"))
"""


def test_launches_can_be_observed():
    """TERRA_TRACE=1 prints a line per product and TERRA_NVTX=1 opens a range per launch, in the halves too: two products
    forward, two input and two weight gradients backward, one LayerNorm, each."""
    import os
    import subprocess
    import sys

    env = dict(os.environ, TERRA_TRACE="1", TERRA_NVTX="1")
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    r = subprocess.run([sys.executable, "-c", _OBSERVED], cwd=root, env=env, capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stderr
    assert r.stdout.split() == ["12", "2"]
    assert r.stderr.count("[terra trace] gemm") == 12


def test_weight_gradient_of_pitched_rows():
    from terra_b200.ops.blocks import wgrad_accumulate

    torch.manual_seed(1)
    wide = torch.randn(777, 512, device="cuda").to(torch.bfloat16)
    dy, x = wide[:, :200], wide[:, 256:352]
    gw, gb = torch.zeros(200, 96, device="cuda"), torch.zeros(200, device="cuda")
    wgrad_accumulate(dy, x, gw, gb)
    ref = dy.float().t() @ x.float()
    assert _rel(gw, ref) < 1e-5 and _rel(gb, dy.float().sum(0)) < 1e-5


@pytest.mark.parametrize("M,N,K", [(10, 64, 0), (10, 0, 64), (0, 64, 64)])
def test_weight_gradient_refuses_empty_operands(M, N, K):
    """The plan of the tiles divides by their number; an empty operand is an error that Python sees."""
    from terra_b200.ops.blocks import wgrad_accumulate

    dy, x = torch.zeros(M, N, device="cuda", dtype=torch.bfloat16), torch.zeros(M, K, device="cuda", dtype=torch.bfloat16)
    with pytest.raises(RuntimeError):
        wgrad_accumulate(dy, x, torch.zeros(N, K, device="cuda"), torch.zeros(N, device="cuda"))


def _mlp(dim, rows):
    from terra_b200.models.layers import MlpHalf
    from terra_b200.utils.flat_params import ParamArena

    torch.manual_seed(2)
    mod = MlpHalf(dim, 4 * dim).cuda()
    return mod, ParamArena(mod), torch.randn(rows, dim, device="cuda").to(torch.bfloat16)


def test_native_halves_refuse_other_operands():
    """Weights and biases are read by raw pointers: types, sizes and strides that do not fit are errors."""
    from terra_b200 import _ext
    from terra_b200.ops.gemm import status_word

    ext, C, H = _ext.load(), 64, 256
    r = lambda *s, dt=torch.bfloat16: torch.randn(*s, device="cuda").to(dt)
    good = dict(x=r(32, C), ln_w=r(C), ln_b=r(C), fc1_w=r(H, C), fc1_b=r(H), fc2_w=r(C, H), fc2_b=r(C))
    run = lambda **kw: ext.mlp_half_fwd(*{**good, **kw}.values(), 1e-5, status_word("cuda"))[0]
    y = run()
    # an fp32 bias is taken by its type
    assert torch.equal(run(fc1_b=good["fc1_b"].float(), fc2_b=good["fc2_b"].float()), y)
    for bad in (dict(fc1_w=r(H, C, dt=torch.float32)), dict(fc1_w=r(C, H).t()), dict(fc2_w=r(C, H).cpu()), dict(fc1_b=r(H - 8)),
                dict(fc2_b=r(2 * C)[::2]), dict(fc2_b=r(C, dt=torch.float16)), dict(x=r(32, 2 * C)[:, :C]), dict(ln_w=r(C).float())):
        with pytest.raises(RuntimeError):
            run(**bad)


@pytest.mark.parametrize("half", ["attention", "mlp"])
@pytest.mark.parametrize("native", [True, False])
def test_saved_tensors_of_another_form(monkeypatch, half, native):
    """Hooks may hand the saved tensors back with another row pitch: products take that, what is read as dense rows is
    refused."""
    from terra_b200.models.layers import SwinAttentionHalf
    from terra_b200.ops import blocks
    from terra_b200.ops.attention import WindowGeometry
    from terra_b200.utils.flat_params import ParamArena

    monkeypatch.setattr(blocks, "_LAUNCHES_OBSERVED", not native)
    if half == "attention":
        torch.manual_seed(2)
        geo = WindowGeometry(1, 2, 2, 8, 8)
        mod = SwinAttentionHalf(1, 64, (8, 8), 2, use_relative_position_bias=True).cuda()
        arena, x = ParamArena(mod), torch.randn(geo.rows_local, 64, device="cuda").to(torch.bfloat16)
        run = lambda t: blocks.attention_half(t, mod, geo, True)
        pitched_ok, dense = (3, 5), (0, 4)          # xn, o / x, qkv in the order of saving
    else:
        mod, arena, x = _mlp(64, 300)
        run = lambda t: blocks.mlp_half(t, mod)
        pitched_ok, dense = (3, 4, 5), (0,)         # xn, pre, act / x
    dy = torch.randn_like(x)

    def grads(pitched):
        seen = []

        def pack(t):
            seen.append(len(seen))
            return len(seen) - 1, t

        def unpack(p):
            i, t = p
            return torch.cat([t, t], dim=1)[:, :t.shape[1]] if i in pitched else t

        arena.zero_grad()
        t = x.clone().requires_grad_(True)
        with torch.autograd.graph.saved_tensors_hooks(pack, unpack):
            y = run(t)
        y.backward(dy)
        return t.grad, arena.grad.clone()

    dx, g = grads(())
    dx2, g2 = grads(pitched_ok)
    assert torch.equal(dx, dx2) and _rel(g2, g) < 1e-5
    for i in dense:
        with pytest.raises(RuntimeError):
            grads((i,))


def test_weight_gradient_into_pitched_rows():
    from terra_b200.ops.blocks import wgrad_accumulate

    torch.manual_seed(3)
    dy, x = torch.randn(500, 136, device="cuda").to(torch.bfloat16), torch.randn(500, 72, device="cuda").to(torch.bfloat16)
    wide = torch.ones(136, 200, device="cuda")
    wgrad_accumulate(dy, x, wide[:, 64:136])
    assert _rel(wide[:, 64:136] - 1, dy.float().t() @ x.float()) < 1e-5
    assert (wide[:, :64] == 1).all() and (wide[:, 136:] == 1).all()
