"""Layers of equal sizes on several streams at once, and in a capture: each call has sums and staging of its own. Outputs against one
stream after the other: bf16 with fp32 sums in another order (GroupNorm's statistics are atomics: half a bf16 step where their order
moves a rounding, 1e-3 of the norm), gradients fp32 (1e-4: they see those roundings)."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _layers(dim, seed):
    from terra_b200.utils.flat_params import ParamArena

    torch.manual_seed(seed)
    m = torch.nn.ModuleDict(dict(conv=torch.nn.Conv2d(dim, dim, 3, padding=1), norm=torch.nn.GroupNorm(dim // 8, dim),
                                 up=torch.nn.ConvTranspose2d(dim, dim, 2, stride=2), last=torch.nn.GroupNorm(dim // 8, dim))).cuda()
    return m, ParamArena(m)


def _pass(m, arena, x):
    from terra_b200.ops import conv

    arena.grad.zero_()
    t = x.detach().requires_grad_(True)
    y = conv.groupnorm_silu(conv.conv_transpose2x2(conv.groupnorm_silu(conv.conv3x3(t, m["conv"]), m["norm"], residual=t), m["up"]), m["last"])
    y.backward(torch.full_like(y, 0.5))
    return y.detach().float(), t.grad.float(), arena.grad.clone()


def _close(got, want):
    for g, w, tol in zip(got, want, (1e-3, 2e-3, 1e-4)):
        assert torch.isfinite(g).all() and ((g - w).norm() / w.norm()).item() < tol


@pytest.mark.parametrize("native", [True, False])
@pytest.mark.parametrize("B,H,W,dim", [(1, 24, 40, 96), (2, 96, 180, 192)])
def test_streams_side_by_side(monkeypatch, native, B, H, W, dim):
    from terra_b200.ops import conv
    from terra_b200.ops.gemm import check_status

    if not native:
        monkeypatch.setattr(conv, "native_node", lambda grads=(): False)
    sets = [_layers(dim, s) for s in range(3)]
    xs = [(torch.randn(B, H, W, dim, device="cuda") * (1 + s)).to(torch.bfloat16) for s in range(3)]
    want = [_pass(m, a, x) for (m, a), x in zip(sets, xs)]
    streams = [torch.cuda.Stream() for _ in sets]
    for s in streams:
        s.wait_stream(torch.cuda.current_stream())
    got = [[] for _ in sets]
    for _ in range(12):
        for i, s in enumerate(streams):
            with torch.cuda.stream(s):
                got[i].append(_pass(*sets[i], xs[i]))
    torch.cuda.synchronize()
    for w, results in zip(want, got):
        for g in results:
            _close(g, w)
    for (m, a), x, w in zip(sets, xs, want):      # and nothing of it stays behind for one stream alone
        _close(_pass(m, a, x), w)
    check_status("cuda")


def test_threads_with_streams_of_their_own():
    """Backward passes run without the interpreter's lock while other threads go forward."""
    import threading

    from terra_b200.ops.gemm import check_status

    sets = [_layers(72, s) for s in range(3)]
    xs = [(torch.randn(1, 33, 40, 72, device="cuda") * (1 + s)).to(torch.bfloat16) for s in range(3)]
    want = [_pass(m, a, x) for (m, a), x in zip(sets, xs)]
    torch.cuda.synchronize()
    got = [None] * 3

    def work(i):
        with torch.cuda.stream(torch.cuda.Stream()):
            got[i] = [_pass(*sets[i], xs[i]) for _ in range(10)]

    threads = [threading.Thread(target=work, args=(i,)) for i in range(3)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    torch.cuda.synchronize()
    for w, results in zip(want, got):
        for g in results:
            _close(g, w)
    check_status("cuda")


def test_first_use_inside_a_capture():
    """Nothing that a capture only records is used by the calls beside it."""
    from terra_b200.ops import conv

    m, arena = _layers(48, 5)
    x = (torch.randn(1, 17, 31, 48, device="cuda") + 1).to(torch.bfloat16)
    gamma, beta = (p.detach().double() for p in m["norm"].parameters())
    want = torch.nn.functional.silu(torch.nn.functional.group_norm(x.double().permute(0, 3, 1, 2), 6, gamma, beta, eps=1e-5)).permute(0, 2, 3, 1)
    rel = lambda y: ((y.double() - want).norm() / want.norm()).item()
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.no_grad():
        with torch.cuda.graph(graph):
            out = conv.groupnorm_silu(x, m["norm"])
        eager = conv.groupnorm_silu(x, m["norm"])
        graph.replay()
        torch.cuda.synchronize()
    assert rel(eager) < 5e-3 and rel(out) < 5e-3      # (outputs are rounded to bf16: 2^-9)


def test_scratch_belongs_to_one_call_and_one_stream():
    from terra_b200 import _ext

    ext = _ext.load()
    like = torch.zeros(1, device="cuda")
    a, b = ext.scratch_take(like, [2, 331]), ext.scratch_take(like, [331, 2])      # two calls at once
    assert a.shape == (2, 331) and a.data_ptr() != b.data_ptr() and not a.any() and not b.any()
    at = a.data_ptr()
    ext.scratch_give(a)
    other = torch.cuda.Stream()
    with torch.cuda.stream(other):
        c = ext.scratch_take(like, [662])
        assert c.data_ptr() != at
    d = ext.scratch_take(like, [662])
    assert d.data_ptr() == at and ext.scratch_take(like, [662]).data_ptr() not in (at, b.data_ptr())
    ext.scratch_give(d)
    graph = torch.cuda.CUDAGraph()
    torch.cuda.synchronize()
    with torch.cuda.graph(graph):      # neither taken from the pool nor kept in it
        e = ext.scratch_take(like, [662])
        assert e.data_ptr() != at
        ext.scratch_give(e)
        f = ext.scratch_take(like, [662])
        assert f.data_ptr() not in (e.data_ptr(), at)
    assert ext.scratch_take(like, [662]).data_ptr() == at


def test_idle_scratch_is_bounded():
    from terra_b200 import _ext

    ext = _ext.load()
    like = torch.zeros(1, device="cuda")
    torch.cuda.synchronize()
    before = torch.cuda.memory_allocated()
    for n in range(200):      # 200 sizes of 4 MB: no more than 256 MB of them stay
        ext.scratch_give(ext.scratch_take(like, [(1 << 20) + 8 * n]))
    assert torch.cuda.memory_allocated() - before <= 260 << 20
    ext.scratch_give(ext.scratch_take(like, [65 << 20]))      # larger than all that may lie idle
    assert torch.cuda.memory_allocated() - before <= 260 << 20
