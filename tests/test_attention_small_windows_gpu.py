"""Window attention of at most 128 tokens (csrc/window_attn.cu) where its variants change: window widths with and without
compile-time bias addressing, windows that pad a 16-row block, every head dim, head counts that the forward kernel cannot
group, few and many windows per thread block, several owners of windows and token shards, non-finite inputs.

Bound: against fp32 the kernel rounds P, dS and the results to bf16 (2^-9 each, independent): 3 * 2^-9 = 0.6 % of the norm;
the tests allow 1 %."""
import pytest
import torch

pytestmark = pytest.mark.gpu
REL = 1e-2


def _rel(got, ref):
    return ((got.float() - ref.float()).norm() / ref.float().norm()).item()


def _reference(qkv, table, dout, geo, heads, shifted, scale):
    from terra_b200.ops.attention import window_attention_reference

    q32 = qkv.detach().float().requires_grad_(True)
    t32 = table.detach().clone().requires_grad_(True)
    ref = window_attention_reference(q32.reshape(geo.B, geo.nWh * geo.nWw, geo.N, -1), geo, heads, shifted, t32, True,
                                     scale).reshape(-1, qkv.shape[1] // 3)
    ref.backward(dout.float())
    return ref.detach(), q32.grad, t32.grad


@pytest.mark.parametrize("B,nWh,nWw,wh,ww,hd,heads,shifted", [
    (1, 1, 1, 8, 8, 32, 2, True),          # one window: every edge of the frame is its own
    (2, 3, 2, 8, 8, 16, 3, True),          # odd head count: one head per block forward
    (1, 2, 3, 8, 8, 128, 1, False),        # one stage, dQ staged outside the stash
    (1, 40, 41, 8, 8, 64, 2, True),        # more windows than blocks
    (1, 2, 3, 8, 12, 16, 4, True),         # 96 tokens, width 12
    (1, 2, 3, 12, 8, 32, 2, True),         # 96 tokens, generic width
    (1, 2, 2, 8, 12, 128, 1, True),        # largest shared memory that is accepted
    (1, 2, 3, 8, 16, 32, 2, False),        # 128 tokens, generic width
    (1, 2, 3, 16, 8, 64, 1, True),         # 128 tokens, width 8
    (1, 3, 2, 7, 7, 32, 2, True),          # 49 tokens: padding inside the last block
    (1, 3, 2, 4, 8, 16, 2, True),          # 32 tokens: two blocks without a token
    (1, 2, 2, 5, 13, 64, 1, True),         # 65 tokens: one row in the fifth block
    (1, 2, 2, 9, 12, 16, 2, True),         # 108 tokens, width 12 with padding
])
def test_forward_backward_and_bias_gradient(B, nWh, nWw, wh, ww, hd, heads, shifted):
    from terra_b200.ops.attention import WindowGeometry, window_attention

    torch.manual_seed(3)
    geo, C = WindowGeometry(B, nWh, nWw, wh, ww), hd * heads
    rows = B * nWh * nWw * geo.N
    qkv = torch.randn(rows, 3 * C, device="cuda").to(torch.bfloat16).requires_grad_(True)
    table = (torch.randn((2 * wh - 1) * (2 * ww - 1), heads, device="cuda") * 0.5).requires_grad_(True)
    dout = torch.randn(rows, C, device="cuda").to(torch.bfloat16)
    out = window_attention(qkv, geo, heads, shifted, table, True, hd ** -0.5)
    out.backward(dout)
    ref, dq, dt = _reference(qkv, table, dout, geo, heads, shifted, hd ** -0.5)
    assert _rel(out, ref) < REL and _rel(qkv.grad, dq) < REL and _rel(table.grad, dt) < REL


@pytest.mark.parametrize("wh,ww,sp", [(8, 8, 1), (8, 8, 2), (7, 7, 2), (8, 12, 3)])
def test_several_owners_of_windows_and_token_shards(wh, ww, sp):
    """The launches of all ranks of a 2-group layout, one after the other on one GPU (a rank's kernel waits for nobody):
    together they write every row once and reproduce the single-rank results."""
    from terra_b200 import _ext
    from terra_b200.ops.attention import WindowGeometry, launch_window_attn_bwd, launch_window_attn_fwd

    torch.manual_seed(5)
    ext, nWh, nWw, hd, heads = _ext.load(), 3, 4, 32, 2
    C, N, nW, split = hd * heads, wh * ww, 12, [0, 5, 12]
    shard = -(-N // sp)
    table = torch.randn((2 * wh - 1) * (2 * ww - 1), heads, device="cuda") * 0.5
    whole = torch.randn(nW, N, 3 * C, device="cuda").to(torch.bfloat16)
    dwhole = torch.randn(nW, N, C, device="cuda").to(torch.bfloat16)

    def shards(t):          # slot (group, shard): [windows of the group, shard tokens, channels], padded rows behind the last
        out = []
        for g in range(2):
            for s in range(sp):
                part = torch.zeros(split[g + 1] - split[g], shard, t.shape[2], device="cuda", dtype=t.dtype)
                piece = t[split[g]:split[g + 1], s * shard:(s + 1) * shard]
                part[:, :piece.shape[1]] = piece
                out.append(part)
        return out

    def join(parts):
        return torch.cat([torch.cat(parts[g * sp:(g + 1) * sp], 1)[:, :N] for g in range(2)])

    qkv, dout = shards(whole), shards(dwhole)
    out = [torch.full_like(t, float("nan")) for t in dout]
    dqkv = [torch.full_like(t, float("nan")) for t in qkv]
    dtable = torch.zeros_like(table)
    ptrs = lambda ts: [t.data_ptr() for t in ts]
    for g in range(2):
        for s in range(sp):
            geo = WindowGeometry(1, nWh, nWw, wh, ww, win_start=list(split), my_wg=g, sp=sp, my_sp=s)
            launch_window_attn_fwd(ext, ptrs(qkv), ptrs(out), table, geo, C, heads, wh // 2, ww // 2, True, hd ** -0.5, "cuda")
            launch_window_attn_bwd(ext, ptrs(qkv), ptrs(dout), ptrs(dqkv), table, dtable, geo, C, heads, wh // 2, ww // 2, True,
                                   hd ** -0.5, "cuda")
    one = WindowGeometry(1, nWh, nWw, wh, ww)
    ref, dq, dt = _reference(whole.reshape(-1, 3 * C), table, dwhole.reshape(-1, C), one, heads, True, hd ** -0.5)
    assert _rel(join(out).reshape(-1, C), ref) < REL
    assert _rel(join(dqkv).reshape(-1, 3 * C), dq) < REL and _rel(dtable, dt) < REL


@pytest.mark.parametrize("wh,ww", [(8, 8), (7, 7)])
def test_non_finite_values_stay_in_their_window(wh, ww):
    """A window with NaN and infinite values spoils its own results only, also where a block's shared-memory rows are used
    for hundreds of windows and some of them are padding."""
    from terra_b200.ops.attention import WindowGeometry, window_attention

    torch.manual_seed(7)
    geo, hd, heads, bad = WindowGeometry(1, 40, 40, wh, ww), 32, 2, 11
    C, N = hd * heads, wh * ww
    clean = torch.randn(geo.nWh * geo.nWw, N, 3 * C, device="cuda").to(torch.bfloat16)
    dirty = clean.clone()
    dirty[bad, 0], dirty[bad, 5] = float("nan"), float("inf")
    dout = torch.randn(geo.nWh * geo.nWw * N, C, device="cuda").to(torch.bfloat16)
    got = []
    for t in (clean, dirty):
        q = t.reshape(-1, 3 * C).clone().requires_grad_(True)
        o = window_attention(q, geo, heads, False, None, True, hd ** -0.5)
        o.backward(dout)
        got.append((o.detach().reshape(-1, N, C), q.grad.reshape(-1, N, 3 * C)))
    others = torch.arange(geo.nWh * geo.nWw, device="cuda") != bad
    assert torch.equal(got[0][0][others], got[1][0][others]) and torch.equal(got[0][1][others], got[1][1][others])
    assert torch.isnan(got[1][0][bad]).any() and torch.isnan(got[1][1][bad]).any()
