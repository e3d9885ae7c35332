"""Kernels that overlap the tail of their predecessor see its results: chains of dependent launches, with nothing between them,
give the bits that the same launches give when the GPU is idle before each."""
import pytest
import torch

pytestmark = pytest.mark.gpu


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
    return cur


@pytest.mark.parametrize("rows,dim", [(64, 64), (512, 96), (5000, 384), (30000, 192)])
def test_a_chain_gives_the_bits_of_single_launches(rows, dim):
    from terra_b200.ops.gemm import check_status

    want = _chain(rows, dim, True)
    for _ in range(10):
        assert torch.equal(_chain(rows, dim, False), want)
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
    assert all(torch.equal(g, want) for g in got)
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
