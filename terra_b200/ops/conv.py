"""FuXi-style sampling-block operators on NHWC activations.

CUDA: 3x3 convolutions (stride 1 / 2, padding 1) are implicit GEMMs on the tcgen05 kernel - the A operand is
gathered by 5-D TMA boxes with zero fill outside the image, k-blocks enumerate (tap, channel chunk); the input
gradient of the stride-1 convolution is the same kernel with flipped, transposed weights; weight gradients
contract over pixels with one tile group per tap. The 2x2/stride-2 transposed convolution, its input gradient and that of
the stride-2 convolution are the same kernel with other tap tables and outputs stored to every second pixel. GroupNorm+SiLU is a statistics pass plus one fused apply pass (optionally adding
the block's shortcut), its backward a reduce pass plus an apply pass.

With row-stripe domain parallelism (``dom`` given) halo rows come from the neighbours and GroupNorm statistics
are summed over the stripe group, so that the result equals the single-rank one.
CPU: plain PyTorch on the same NHWC tensors (oracle for the tests, gloo ranks for the multi-rank logic).

Reference: models/utils.py:101-180 (``CreditDownBlock`` / ``CreditUpBlock``), credit/domain_parallel/layers.py:18-84,
87-208, 429-483 and halo_exchange.py:18-157 for the row-stripe forms.
"""
from __future__ import annotations

import functools
from typing import Optional

import torch
import torch.nn.functional as TF

from .. import _ext
from . import _flags as F
from .gemm import gemm, status_word
from .packed import PACK_EPOCH, _packed, fp32_values, invalidate_packed_weights  # noqa: F401  (re-exported)
from .blocks import FUSE_BIAS_GRAD, native_node, wgrad_accumulate, bias_grad_accumulate
from ..utils.nvtx import nvtx_range

GN_EPS = 1e-5
_MAX_TAP_CHUNKS = 128       # (tap, 64-channel chunk) entries of the implicit GEMM's table (GEMM_MAX_KTABLE)


# ------------------------------------------------------------------------------------------------ weight packing
def _pack_taps(w, n1, s1, n2, s2, channels, sc, offsets, pad2=None):
    """bf16 ``[n1 * n2, taps * C_pad]`` with ``out[i * n2 + j, t, c] = w.flatten()[i * s1 + j * s2 + c * sc + offsets[t]]``, the
    channels padded to a multiple of 64 with zeros, and the ``n2`` rows of every ``i`` to ``pad2``."""
    valid2, n2 = n2, pad2 or n2
    cpad, taps = (channels + 63) // 64 * 64, len(offsets)
    if w.is_cuda and w.dtype == torch.bfloat16:
        return _ext.load().packed_taps(w, n1, s1, n2, s2, channels, sc, offsets, valid2)
    steps = [(n1, s1), (valid2, s2), (1, 0), (channels, sc)]
    at = sum(torch.arange(n, device=w.device).view([-1 if d == e else 1 for e in range(4)]) * s for d, (n, s) in enumerate(steps))
    at = at + torch.tensor(list(offsets), device=w.device).view(1, 1, -1, 1)
    out = torch.zeros(n1, n2, taps, cpad, device=w.device, dtype=torch.bfloat16)
    out[:, :valid2, :, :channels] = w.reshape(-1)[at.reshape(-1)].view(n1, valid2, taps, channels)
    return out.view(n1 * n2, taps * cpad)


def pack_conv3x3_weight(w: torch.Tensor) -> torch.Tensor:
    """(Cout, Cin, 3, 3) -> bf16 [Cout, 9 * Cin_pad], tap-major, Cin padded to a multiple of 64 with zeros."""
    cout, cin = w.shape[:2]
    return _pack_taps(w, 1, 0, cout, cin * 9, cin, 9, range(9))


# The stride-2 input gradient: taps (ky, kx) by the parity of the input pixel they reach, odd row and column first
_S2_TAPS = (0, 2, 6, 8, 3, 5, 1, 7, 4)


def pack_conv3x3_weight_s2_dgrad(w: torch.Tensor) -> torch.Tensor:
    cout, cin = w.shape[:2]
    return _pack_taps(w, 1, 0, cin, 9, cout, cin * 9, _S2_TAPS)


def pack_conv3x3_weight_dgrad(w: torch.Tensor) -> torch.Tensor:
    """Weights of the stride-1 input-gradient convolution: taps flipped, channels swapped."""
    cout, cin = w.shape[:2]
    return _pack_taps(w, 1, 0, cin, 9, cout, cin * 9, range(8, -1, -1))


def _arena_grad(p):
    """The parameter's fp32 gradient view in the flat arena (accumulated into in place), or None."""
    g = getattr(p, "grad", None)
    if g is not None and g.is_cuda and g.dtype == torch.float32 and g.is_contiguous() and getattr(p, "bf16", None) is not None:
        return g
    return None


class _Conv3x3Fn(torch.autograd.Function):
    @staticmethod
    def forward(ctx, x, weight, bias, stride, dom):
        ext = _ext.load()
        B, H, W, Cin = x.shape
        Cout = weight.shape[0]
        Ho, Wo = (H, W) if stride == 1 else ((H + 1) // 2, W // 2)
        y = torch.empty(B, Ho, Wo, Cout, device=x.device, dtype=torch.bfloat16)
        w16 = weight.bf16 if getattr(weight, "bf16", None) is not None else weight.detach().to(torch.bfloat16)
        b16 = bias.bf16 if getattr(bias, "bf16", None) is not None else bias.detach().to(torch.bfloat16)
        wp = _packed(weight, w16, "fwd", pack_conv3x3_weight)
        multi = dom is not None and dom.world > 1
        lo, hi = dom.exchange_rows(x) if multi else (None, None)
        ext.conv3x3_fwd(x, wp, y, stride, F.EPI_BIAS, b16, None, status_word(x.device), lo, hi)
        ctx.save_for_backward(x)
        ctx.p = (weight, bias, w16, stride, dom, lo, hi)
        return y

    @staticmethod
    def backward(ctx, dy):
        ext = _ext.load()
        (x,) = ctx.saved_tensors
        weight, bias, w16, stride, dom, lo, hi = ctx.p
        multi = dom is not None and dom.world > 1
        dy = dy.contiguous()
        B, H, W, Cin = x.shape
        Cout = weight.shape[0]
        # ---- weight / bias gradients (fp32); the halo rows received in forward serve the boundary taps
        gw, gb = _arena_grad(weight), _arena_grad(bias)
        split, stack = _wgrad_split(B, H, W, stride, Cout, Cin)
        if gw is not None:
            # tap-major staging [9, Cout, Cin] folded into the arena's (Cout, Cin, 3, 3) view
            dw9 = ext.scratch_take(x, [9, Cout, Cin])
            # the bias gradient (column sums of dy) comes out of the same kernel
            ext.conv3x3_wgrad(x, dy, dw9, stride, split, status_word(x.device), lo, hi,
                              bias_grad=gb if FUSE_BIAS_GRAD else None, stack=stack)
            ext.strided_add(dw9, gw, 1, Cin * 9, 9)
            ext.scratch_give(dw9)
            dw = None
        else:
            dw9 = torch.zeros(9, Cout, Cin, device=x.device, dtype=torch.float32)
            ext.conv3x3_wgrad(x, dy, dw9, stride, split, status_word(x.device), lo, hi, stack=stack)
            dw = dw9.view(3, 3, Cout, Cin).permute(2, 3, 0, 1)
        if gb is not None:
            if gw is None or not FUSE_BIAS_GRAD:
                ext.colsum(dy.view(-1, Cout), gb)
            db = None
        else:
            db = torch.zeros(Cout, device=x.device, dtype=torch.float32)
            ext.colsum(dy.view(-1, Cout), db)
        # ---- input gradient
        dx = None
        if ctx.needs_input_grad[0]:
            if stride == 1:
                dx = torch.empty_like(x)
                wf = _packed(weight, w16, "dgrad", pack_conv3x3_weight_dgrad)
                glo, ghi = dom.exchange_rows(dy) if multi else (None, None)
                ext.conv3x3_fwd(dy, wf, dx, 1, 0, None, None, status_word(x.device), glo, ghi)
            else:
                dx = _conv3x3_s2_dgrad(dy, w16, H, W, dom, weight)
        return dx, dw, db, None, None


def balanced_split(tiles: int, kblocks: int, sms: int = 148, limit: int = 64) -> int:
    """Split-K factor for a persistent kernel of ``sms`` CTAs: the one whose ``tiles * split`` work items fill whole
    rounds of CTAs best (time ~ ceil(tiles * split / sms) / split), the smaller factor on near ties (every split adds
    one pass of fp32 atomics over the output)."""
    best, best_cost = 1, float("inf")
    for s in range(1, max(1, min(kblocks, limit)) + 1):
        cost = -(-tiles * s // sms) / s + 0.002 * s
        if cost < best_cost - 1e-9:
            best, best_cost = s, cost
    return best


def _stream_cost(heavy, light, bn, split, sms=148):
    """KB through the most loaded CTA's shared-memory port (operand fill and tensor-core reads) per k-block of the whole
    contraction, when ``heavy`` tiles of two row blocks are handed out before ``light`` ones of a single block."""
    one = 2 * (16 + bn // 8)
    two = 32 + bn // 8 + one
    return (-(-heavy * split // sms) * (two - one) + -(-(heavy + light) * split // sms) * one) / split


@functools.lru_cache(maxsize=256)
def _wgrad_plan(taps, M, N, kblocks):
    """(split-K factor, row blocks per tile) of a convolution's weight gradient: ``taps`` products of ``M`` x ``N`` outputs.
    Two row blocks share a tile of the other operand (15 % less traffic per output) where that also comes out ahead with the
    single block an odd count leaves over and with whole rounds of CTAs; every split adds 0.2 % for its pass of atomics. The
    native nodes of one rank run all taps as one product, with a plan of their own (``gemm_host.cu::model_tap_wgrad``), and take
    this split as the least number of parts: the sums of a part are as long as here at most, and so is their error."""
    bn = 192 if N % 192 == 0 else 128            # the tile width the kernel picks
    blocks, n = (M + 127) // 128, taps * ((N + bn - 1) // bn)
    best = balanced_split(blocks * n, kblocks)
    plan, cost = (best, 1), _stream_cost(0, blocks * n, bn, best) * (1 + 0.002 * best)
    if N > 64 and blocks >= 2 and (blocks + 1) // 2 * n * kblocks >= 148 * 8:
        for s in range(1, max(1, min(kblocks, 64)) + 1):
            c = _stream_cost(blocks // 2 * n, blocks % 2 * n, bn, s) * (1 + 0.002 * s)
            if c < cost * 0.99:
                plan, cost = (s, 2), c
    return plan


def _wgrad_split(B, H, W, stride, Cout, Cin):
    Ho, Wo = (H, W) if stride == 1 else ((H + 1) // 2, W // 2)
    return _wgrad_plan(9, Cout, Cin, B * Ho * ((Wo + 63) // 64))


def _conv3x3_s2_dgrad(dy, w16, H, W, dom, weight=None):
    """Input gradient of the stride-2 convolution. One launch: the four parities of the input pixel are four tile groups
    of the implicit GEMM, with the 1, 2, 2 or 4 taps that reach them. With halo rows to give back (multi-rank stripes),
    more channels than the tap table holds, or without the TMA epilogue: dcol = dy @ W (tap-major columns) on the GEMM, then one gather kernel over the
    taps that reach each input pixel. (Images of fewer than about 50 columns of ``dy`` would be faster by columns - 32768
    pixels of 384 channels, us, one launch / columns: 2048 x 16 472 / 161, 682 x 48 166 / 159, 512 x 64 128 / 162 - but the
    columns round every tap's share to bf16 where the one launch sums them in fp32.)"""
    B, Ho, Wo, Cout = dy.shape
    Cin = w16.shape[1]
    if not (dom is not None and dom.world > 1) and 9 * ((Cout + 63) // 64) <= _MAX_TAP_CHUNKS and _ext.load().gemm_tma_epilogue():
        wp = _packed(weight, w16, "s2dgrad_taps", pack_conv3x3_weight_s2_dgrad) if weight is not None else \
            pack_conv3x3_weight_s2_dgrad(w16)
        out = torch.empty(B, H, W, Cin, device=dy.device, dtype=torch.bfloat16)
        _ext.load().conv3x3_s2_dgrad(dy, wp, out, status_word(dy.device))
        return out
    build = lambda w: w.permute(0, 2, 3, 1).reshape(Cout, 9 * Cin).contiguous()          # [Cout, (tap, ci)]
    wk = _packed(weight, w16, "s2dgrad", build) if weight is not None else build(w16)
    dcol = gemm(dy.view(-1, Cout), wk, b_mn=True).view(B, Ho, Wo, 9, Cin)     # dcol[p, tap, ci]
    ext = _ext.load()
    if dom is not None and dom.world > 1:
        # the rows above / below the stripe (padded rows 0 and H + 1) receive gradient too: it goes back to the
        # neighbours, so the padded rows are produced (fp32, as the halo fold accumulates)
        dxp = torch.zeros(B, H + 2, W + 2, Cin, device=dy.device, dtype=torch.float32)
        inner = torch.empty(B, H + 2, W, Cin, device=dy.device, dtype=torch.float32)
        ext.conv_s2_col2im(dcol.contiguous(), inner, W, 0)
        dxp[:, :, 1:W + 1] = inner
        return dom.fold_halo_grad(dxp, H, W).to(torch.bfloat16).contiguous()
    out = torch.empty(B, H, W, Cin, device=dy.device, dtype=torch.bfloat16)
    ext.conv_s2_col2im(dcol.contiguous(), out, W, 1)
    return out


def _native_layer(a, b) -> bool:
    """Whether a native node may stand for the layer of two parameters (it reads their gradients again when it runs backward)."""
    return native_node() and _arena_grad(a) is not None and _arena_grad(b) is not None


def _conv3x3_node(x, weight, bias, stride, dom):
    """The convolution of one rank as a native autograd node; None where it is not one."""
    if (dom is not None and dom.world > 1) or x.dim() != 4 or not _native_layer(weight, bias):
        return None
    ext = _ext.load()
    (B, H, W, Cin), Cout, w16 = x.shape, weight.shape[0], weight.bf16
    if stride != 1 and not (9 * ((Cout + 63) // 64) <= _MAX_TAP_CHUNKS and ext.gemm_tma_epilogue()):
        return None
    wd = None
    if x.requires_grad and torch.is_grad_enabled():
        wd = _packed(weight, w16, "dgrad", pack_conv3x3_weight_dgrad) if stride == 1 else \
            _packed(weight, w16, "s2dgrad_taps", pack_conv3x3_weight_s2_dgrad)
    return ext.nodes.conv3x3(x, weight, bias, _packed(weight, w16, "fwd", pack_conv3x3_weight), wd, bias.bf16,
                             stride, _wgrad_split(B, H, W, stride, Cout, Cin)[0], FUSE_BIAS_GRAD, status_word(x.device))


@nvtx_range("terra.conv3x3")
def conv3x3(x, conv: torch.nn.Conv2d, stride: int = 1, dom=None):
    """x NHWC -> NHWC. ``conv`` holds a (Cout, Cin, 3, 3) weight and a bias."""
    if x.is_cuda:
        y = _conv3x3_node(x, conv.weight, conv.bias, stride, dom)
        return _Conv3x3Fn.apply(x, conv.weight, conv.bias, stride, dom) if y is None else y
    xin = x.permute(0, 3, 1, 2)
    if dom is not None and dom.world > 1:
        xin = dom.halo_exchange_cpu(xin, 1)
        y = TF.conv2d(xin, conv.weight, conv.bias, stride=stride, padding=(0, 1))
        if stride == 2 and y.shape[2] > (x.shape[1] + 1) // 2:
            y = y[:, :, :(x.shape[1] + 1) // 2]
    else:
        y = TF.conv2d(xin, conv.weight, conv.bias, stride=stride, padding=1)
    return y.permute(0, 2, 3, 1)


# ------------------------------------------------------------------------------------------------ transposed conv 2x2 / s2
def _convt_tiled(B, H, W, Cin, Cout):
    """The gathered forms: the (tap, channel chunk) tables must hold the layer, and their outputs leave through TMA. Otherwise
    a plain GEMM and permuted copies, as for images of fewer than 32 columns whose rows make more than one round of tiles: a
    tile is 128 pixels of one row, so below a quarter of it the padding costs more than the copies. Forward + backward at
    32768 pixels of 384 channels (us, gathered / general): 2048 x 16 658 / 440, 1365 x 24 466 / 442, 1024 x 32 368 / 441, 512 x 64
    232 / 440; at 512 pixels, in one round, 32 x 16 53 / 77 (both forms round once: the sums are fp32)."""
    if W < 32 and B * H > 148:
        return False
    return _ext.load().gemm_tma_epilogue() and Cout % 8 == 0 and Cin % 8 == 0 and max(4 * ((Cout + 63) // 64), (Cin + 63) // 64) <= _MAX_TAP_CHUNKS


class _ConvT2x2Fn(torch.autograd.Function):
    @staticmethod
    def forward(ctx, x, weight, bias):
        ext = _ext.load()
        B, H, W, Cin = x.shape
        Cout = weight.shape[1]
        w16 = weight.bf16 if getattr(weight, "bf16", None) is not None else weight.detach().to(torch.bfloat16)
        b16 = bias.bf16 if getattr(bias, "bf16", None) is not None else bias.detach().to(torch.bfloat16)
        y = torch.empty(B, 2 * H, 2 * W, Cout, device=x.device, dtype=torch.bfloat16)
        if _convt_tiled(B, H, W, Cin, Cout):
            wt = _packed(weight, w16, "convT", _pack_convt)
            b4 = _packed(bias, b16, "convT_bias", _pack_convt_bias)
            ext.convt2x2(0, x.contiguous(), wt, b4, y, status_word(x.device))
        else:
            b4 = _packed(bias, b16, "convT_bias_flat", lambda b: b.repeat(4))
            flat = gemm(x.reshape(-1, Cin), _convt_flat_weight(weight, w16), bias=b4)
            y.view(B, H, 2, W, 2, Cout).copy_(flat.view(B, H, W, 2, 2, Cout).transpose(2, 3))
        ctx.save_for_backward(x)
        ctx.p = (w16, Cout, weight, bias)
        return y

    @staticmethod
    def backward(ctx, dy):
        ext = _ext.load()
        (x,) = ctx.saved_tensors
        w16, Cout, weight, bias = ctx.p
        B, H, W, Cin = x.shape
        tiled = _convt_tiled(B, H, W, Cin, Cout)
        dy = dy.contiguous()
        gw, gb = _arena_grad(weight), _arena_grad(bias)
        # [tap, co, ci] staging -> (Cin, Cout, 2, 2)
        shape, layout = (4, Cout, Cin), (1, 4, Cout * 4)
        fused = tiled and gb is not None and FUSE_BIAS_GRAD
        if tiled:
            split, stack = _wgrad_plan(4, Cout, Cin, B * H * ((W + 63) // 64))
            wgrad = lambda dwt: ext.convt2x2_wgrad(x.contiguous(), dy, dwt, split, status_word(x.device), stack, gb if fused else None)
        else:
            # un-shuffle dy to [pixels, (dy, dx, co)] once; both products read it
            dyu = dy.view(B, H, 2, W, 2, Cout).permute(0, 1, 3, 2, 4, 5).reshape(B * H * W, 4 * Cout)
            wgrad = lambda dwt: wgrad_accumulate(dyu, x.reshape(-1, Cin), dwt.view(4 * Cout, Cin))
        if gw is not None:
            dwt = ext.scratch_take(x, shape)
            wgrad(dwt)
            ext.strided_add(dwt, gw, *layout)
            ext.scratch_give(dwt)
            dw = None
        else:
            dwt = torch.zeros(*shape, device=x.device, dtype=torch.float32)
            wgrad(dwt)
            dw = dwt.view(2, 2, *shape[1:]).permute(3, 2, 0, 1)
        if gb is not None:
            if not fused:
                ext.colsum(dy.view(-1, Cout), gb)
            db = None
        else:
            db = torch.zeros(Cout, device=x.device, dtype=torch.float32)
            ext.colsum(dy.view(-1, Cout), db)
        dx = None
        if ctx.needs_input_grad[0]:
            if tiled:
                dx = torch.empty(B, H, W, Cin, device=x.device, dtype=torch.bfloat16)
                wd = _packed(weight, w16, "convT_dgrad", _pack_convt_dgrad)
                ext.convt2x2(1, dy, wd, None, dx, status_word(x.device))
            else:
                dx = gemm(dyu, _convt_flat_weight(weight, w16), b_mn=True).view(B, H, W, Cin)
        return dx, dw, db


def _pack_convt(w):
    """Rows (dy, dx, co), every phase padded to whole units of the epilogue, which stores it to its pixels."""
    cin, cout = w.shape[:2]
    return _pack_taps(w, 4, 1, cout, 4, cin, 4 * cout, (0,), (cout + 63) // 64 * 64)


def _pack_convt_bias(b):
    return TF.pad(b, (0, -b.shape[0] % 64)).repeat(4)


def _pack_convt_dgrad(w):
    cin, cout = w.shape[:2]
    return _pack_taps(w, 1, 0, cin, 4 * cout, cout, 4, range(4))


def _conv_transpose2x2_node(x, weight, bias):
    """The transposed convolution as a native autograd node (the gathered forms); None where it is not one."""
    if x.dim() != 4 or not _native_layer(weight, bias):
        return None
    (B, H, W, Cin), Cout, w16 = x.shape, weight.shape[1], weight.bf16
    if not _convt_tiled(B, H, W, Cin, Cout):
        return None
    wd = _packed(weight, w16, "convT_dgrad", _pack_convt_dgrad) if x.requires_grad and torch.is_grad_enabled() else None
    return _ext.load().nodes.conv_transpose2x2(
        x, weight, bias, _packed(weight, w16, "convT", _pack_convt), wd, _packed(bias, bias.bf16, "convT_bias", _pack_convt_bias),
        _wgrad_plan(4, Cout, Cin, B * H * ((W + 63) // 64))[0], FUSE_BIAS_GRAD, status_word(x.device))


def _convt_flat_weight(weight, w16):
    """(Cin, Cout, 2, 2) -> [(dy, dx, co), ci]"""
    cin, cout = w16.shape[:2]
    return _packed(weight, w16, "convT_flat", lambda w: w.permute(2, 3, 1, 0).reshape(4 * cout, cin).contiguous())


def conv_transpose2x2(x, convt: torch.nn.ConvTranspose2d):
    if x.is_cuda:
        y = _conv_transpose2x2_node(x, convt.weight, convt.bias)
        return _ConvT2x2Fn.apply(x, convt.weight, convt.bias) if y is None else y
    return TF.conv_transpose2d(x.permute(0, 3, 1, 2), convt.weight, convt.bias, stride=2).permute(0, 2, 3, 1)


# ------------------------------------------------------------------------------------------------ GroupNorm + SiLU
class _GroupNormSiluFn(torch.autograd.Function):
    @staticmethod
    def forward(ctx, x, gamma, beta, residual, groups, dom):
        ext = _ext.load()
        B, H, W, C = x.shape
        x3 = x.view(B, H * W, C)
        multi = dom is not None and dom.world > 1
        count = float(H * W * (C // groups)) * (dom.world if multi else 1)
        stats = torch.empty(B, groups, 2, device=x.device, dtype=torch.float32)
        if multi:
            sums = torch.zeros(B, groups, 2, device=x.device, dtype=torch.float32)
            ext.groupnorm_stats(x3, sums, groups)
            ext.groupnorm_finalize(dom.all_reduce_small(sums), stats, 1.0 / count, GN_EPS)
        else:
            sums = ext.scratch_take(x, [B, groups, 2])
            ext.groupnorm_stats(x3, sums, groups)
            ext.groupnorm_finalize(sums, stats, 1.0 / count, GN_EPS)
            ext.scratch_give(sums)
        g16 = gamma.bf16 if getattr(gamma, "bf16", None) is not None else gamma.detach().to(torch.bfloat16)
        b16 = beta.bf16 if getattr(beta, "bf16", None) is not None else beta.detach().to(torch.bfloat16)
        y = torch.empty_like(x)
        ext.groupnorm_silu_apply(x3, stats, g16, b16, None if residual is None else residual.view(B, H * W, C),
                                 y.view(B, H * W, C), groups)
        ctx.save_for_backward(x, stats, g16, b16)
        ctx.p = (groups, dom, count, residual is not None, gamma, beta)
        return y

    @staticmethod
    def backward(ctx, dy):
        ext = _ext.load()
        x, stats, g16, b16 = ctx.saved_tensors
        groups, dom, count, has_res, gamma, beta = ctx.p
        B, H, W, C = x.shape
        dy = dy.contiguous()
        x3, dy3 = x.view(B, H * W, C), dy.view(B, H * W, C)
        red = torch.zeros(B, C, 2, device=x.device, dtype=torch.float32)
        gg, gbt = _arena_grad(gamma), _arena_grad(beta)
        if gg is not None and gbt is not None:
            # the affine parameters' gradients are accumulated by the reduce kernel itself
            ext.groupnorm_silu_bwd_reduce(dy3, x3, stats, g16, b16, red, groups, gg, gbt)
            dgamma = dbeta = None
        else:
            ext.groupnorm_silu_bwd_reduce(dy3, x3, stats, g16, b16, red, groups)
            dgamma, dbeta = red[..., 1].sum(0), red[..., 0].sum(0)
        if dom is not None and dom.world > 1:
            red = dom.all_reduce_small(red)
        dx = torch.empty_like(x)
        ext.groupnorm_silu_bwd_apply(dy3, x3, stats, red, g16, b16, dx.view(B, H * W, C), groups, 1.0 / count)
        return dx, dgamma, dbeta, (dy if has_res else None), None, None


def groupnorm_silu(x, gn: torch.nn.GroupNorm, residual=None, dom=None):
    """silu(group_norm(x)) [+ residual] on NHWC; statistics span the whole (global) image."""
    if x.is_cuda:
        if not (dom is not None and dom.world > 1) and x.dim() == 4 and _native_layer(gn.weight, gn.bias):
            return _ext.load().nodes.groupnorm_silu(x, gn.weight, gn.bias, residual, gn.weight.bf16, gn.bias.bf16, gn.num_groups, GN_EPS)
        return _GroupNormSiluFn.apply(x, gn.weight, gn.bias, residual, gn.num_groups, dom)
    xc = x.permute(0, 3, 1, 2)
    if dom is not None and dom.world > 1:
        y = dom.group_norm_cpu(xc, gn.num_groups, gn.weight, gn.bias, GN_EPS)
    else:
        y = TF.group_norm(xc, gn.num_groups, gn.weight, gn.bias, GN_EPS)
    y = TF.silu(y).permute(0, 2, 3, 1)
    return y if residual is None else y + residual
