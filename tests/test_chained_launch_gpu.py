"""Kernels that overlap the tail of their predecessor see its results: chains of dependent launches, with nothing between them,
give the bits that the same launches give when the GPU is idle before each (fp32 atomics: their sums in another order)."""
import os
import subprocess
import sys

import pytest
import torch

pytestmark = pytest.mark.gpu
ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def _chain(rows, dim, sync):
    """LayerNorm, products with every kind of tile start, their gradients and a column sum, each reading what the one before
    wrote; buffers are reused, so that a kernel that starts too early also overwrites what is still read."""
    from terra_b200.ops.blocks import bias_grad_accumulate, layernorm_bwd_cuda, layernorm_cuda, wgrad_accumulate
    from terra_b200.ops.gemm import gemm

    gen = torch.Generator(device="cuda").manual_seed(rows)
    x = torch.randn(rows, dim, generator=gen, device="cuda").to(torch.bfloat16)
    w = (torch.randn(dim, dim, generator=gen, device="cuda") * dim ** -0.5).to(torch.bfloat16)
    one, zero = torch.ones(dim, device="cuda").to(torch.bfloat16), torch.zeros(dim, device="cuda").to(torch.bfloat16)
    a, b = torch.empty_like(x), torch.empty_like(x)
    sums, gw = torch.zeros(dim, device="cuda"), torch.zeros(2, dim, device="cuda")
    weight = torch.zeros(dim, dim, device="cuda")

    def step(f):
        r = f()
        if sync:
            torch.cuda.synchronize()
        return r

    cur = x
    for bn in (0, 128, 1128, 192, 1256):
        y, mean, rstd = step(lambda: layernorm_cuda(cur, one, zero))
        step(lambda: gemm(y, w, bias=zero, residual=cur, out=a, bn=bn))
        step(lambda: gemm(a, w, b_mn=True, out=b))
        dx = step(lambda: layernorm_bwd_cuda(b, cur, one, mean, rstd, gw[0], gw[1], dres=a))
        step(lambda: wgrad_accumulate(dx, y, weight))
        step(lambda: bias_grad_accumulate(dx, sums))
        cur = dx
    return cur, weight, sums, gw


def _same(got, want):
    """The chain's bits; its accumulated gradients to 1e-5 of the norm (fp32 sums of up to 2e5 values in another order)."""
    return torch.equal(got[0], want[0]) and all(((g - w).norm() <= 1e-5 * w.norm()).item() for g, w in zip(got[1:], want[1:]))


@pytest.mark.parametrize("rows,dim", [(64, 64), (512, 96), (5000, 384), (30000, 192)])
def test_a_chain_gives_the_bits_of_single_launches(rows, dim):
    from terra_b200.ops.gemm import check_status

    want = _chain(rows, dim, True)
    for _ in range(10):
        assert _same(_chain(rows, dim, False), want)
    check_status("cuda")


def test_chains_on_two_streams_and_in_a_graph():
    from terra_b200.ops.gemm import check_status

    want = _chain(512, 96, True)
    streams = [torch.cuda.Stream() for _ in range(2)]
    got = []
    for _ in range(4):
        for s in streams:
            s.wait_stream(torch.cuda.current_stream())
            with torch.cuda.stream(s):
                got.append(_chain(512, 96, False))
    for s in streams:
        torch.cuda.current_stream().wait_stream(s)
    assert all(_same(g, want) for g in got)
    from terra_b200.ops.blocks import layernorm_cuda
    from terra_b200.ops.gemm import gemm

    x = torch.randn(512, 96, device="cuda").to(torch.bfloat16)
    w = (torch.randn(96, 96, device="cuda") * 0.1).to(torch.bfloat16)
    one, zero = torch.ones(96, device="cuda").to(torch.bfloat16), torch.zeros(96, device="cuda").to(torch.bfloat16)

    def steps():
        cur = x
        for _ in range(6):
            cur = gemm(layernorm_cuda(cur, one, zero)[0], w, residual=cur)
        return cur

    want = steps()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        out = steps()
    for _ in range(5):
        out.zero_()
        graph.replay()
        torch.cuda.synchronize()
        assert torch.equal(out, want)
    check_status("cuda")


def _model_pass():
    """Two training steps of a small stack, so that every staging, packed weight and optimizer state is used again: padding and patches,
    linear, both convolutions, GroupNorm, transposed convolution, an attention and an MLP half, crop, masked loss, backward, AdamW."""
    from terra_b200.models.layers import MlpHalf, SwinAttentionHalf
    from terra_b200.ops import blocks, conv
    from terra_b200.ops.attention import WindowGeometry
    from terra_b200.ops.gemm import check_status
    from terra_b200.ops.loss import masked_loss
    from terra_b200.ops.patch import pad_patchify, unpatchify_add
    from terra_b200.optim.adamw import FusedAdamW
    from terra_b200.utils.flat_params import ParamArena

    torch.manual_seed(7)
    D, H, W, C = 96, 32, 64, 24
    m = torch.nn.ModuleDict(dict(
        embed=torch.nn.Linear(16 * C, D), down=torch.nn.Conv2d(D, D, 3, stride=2, padding=1), n0=torch.nn.GroupNorm(32, D),
        conv=torch.nn.Conv2d(D, D, 3, padding=1), n1=torch.nn.GroupNorm(32, D), attn=SwinAttentionHalf(0, D, (8, 8), 3), mlp=MlpHalf(D, 4 * D),
        up=torch.nn.ConvTranspose2d(D, D, 2, stride=2), n2=torch.nn.GroupNorm(32, D), out=torch.nn.Linear(D, 16 * C)))
    field, label = torch.randn(2, 1, 4 * H - 5, 4 * W - 6, C).to(torch.bfloat16).cuda()
    m = m.cuda()
    arena = ParamArena(m)
    opt = FusedAdamW(m.parameters(), lr=1e-3, model=m)
    geo = WindowGeometry(1, 2, 4, 8, 8)
    found = []
    for _ in range(2):
        arena.zero_grad()
        x = blocks.linear(pad_patchify(field, 4, (4 * H, 4 * W), 2, 3).view(-1, 16 * C), m["embed"]).view(1, H, W, D)
        t = conv.groupnorm_silu(conv.conv3x3(x, m["down"], 2), m["n0"])
        t = conv.groupnorm_silu(conv.conv3x3(t, m["conv"]), m["n1"], residual=t)
        rows = blocks.mlp_half(blocks.attention_half(t.reshape(-1, D), m["attn"], geo, True), m["mlp"])
        t = conv.groupnorm_silu(conv.conv_transpose2x2(rows.view(1, H // 2, W // 2, D), m["up"]), m["n2"], residual=x)
        y = unpatchify_add(blocks.linear(t.view(-1, D), m["out"]).view(1, H, W, 16 * C), field, 4, 2, 3)
        masked_loss(y, label, None, "MSE", 100.0).backward()
        found += [y.detach().float().cpu(), arena.grad.cpu()]
        opt.step()
        found.append(arena.master.cpu())
    check_status("cuda")
    return found


def test_whole_layers_against_launches_one_by_one(tmp_path):
    """The same two steps in a process that waits for each launch (CUDA_LAUNCH_BLOCKING). Atomics move roundings of bf16 activations
    (2^-9) in one layer and all that follow: 1 % of the norm; AdamW's first steps divide by the gradient's size: 1 % of the values too."""
    path = str(tmp_path / "waited.pt")
    env = dict(os.environ, CUDA_LAUNCH_BLOCKING="1", PYTHONPATH=ROOT)
    subprocess.run([sys.executable, os.path.abspath(__file__), path], env=env, check=True, timeout=300)
    want = torch.load(path)
    for _ in range(5):
        for g, w in zip(_model_pass(), want):
            assert torch.isfinite(g).all() and (g - w).norm() <= 1e-2 * w.norm()


if __name__ == "__main__":
    torch.save(_model_pass(), sys.argv[1])
