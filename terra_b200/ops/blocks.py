"""Fused transformer-block operators.

On CUDA each Swin half-block is one autograd node built from the sm_100a kernels:

  attention half:  LN -> [q|k|v] GEMM (one [3C, C] operand) -> window attention -> proj GEMM (+bias +shortcut)
  MLP half:        LN -> fc1 GEMM (+bias, GELU, pre-activation kept) -> fc2 GEMM (+bias +shortcut)

Backward runs the transposed products on the same tcgen05 kernel (weights read MN-major for input gradients,
both operands MN-major with split-K fp32 atomics for weight gradients, accumulated straight into the flat
gradient arena), fuses GELU' into the fc2 input-gradient epilogue and the shortcut gradient into the LayerNorm
backward. On CPU the same math is plain PyTorch (autograd does the rest); that path is the oracle of the tests.

What these nodes compute is the reference's block halves: models/transformer.py:71-160 (``SequentialSwinTransformer``),
:963-1036 (window-parallel forward), models/attention.py:874-910 (window attention), models/mlp.py:138-175, 375-412 (MLP).
"""
from __future__ import annotations

import os

from typing import Optional

import torch
import torch.nn.functional as TF

from .. import _ext
from .attention import (MAX_KERNEL_WINDOW_TOKENS, WindowGeometry, attn_backward_impl, attn_forward_impl,
                        launch_window_attn_bwd, launch_window_attn_fwd, window_attention)
from . import _flags as F
from .gemm import TRACE, gemm, status_word, trace_product
from .packed import fp32_values
from ..utils import nvtx
from ..utils.nvtx import nvtx_range

LN_EPS = 1e-5


# Bias gradients come out of the weight-gradient GEMM itself (3 ms of an 88 ms step against the separate column-sum
# kernel, measured back to back on one GPU); TERRA_FUSED_BIAS_GRAD=0 restores the separate kernel.
FUSE_BIAS_GRAD = os.environ.get("TERRA_FUSED_BIAS_GRAD", "1") == "1"


# TERRA_TRACE=1 / TERRA_NVTX=1 report single launches, so the halves are then launched one by one from Python
_LAUNCHES_OBSERVED = TRACE or nvtx.ENABLED


@nvtx_range("terra.gemm")
def wgrad_accumulate(dy: torch.Tensor, x: torch.Tensor, grad_w: torch.Tensor, grad_b: torch.Tensor = None) -> None:
    """grad_w[N, K] (fp32) += dy[M, N]^T @ x[M, K]; with ``grad_b``: grad_b[N] (fp32) += column sums of dy, from the
    same kernel (a 16-column MMA of the dy tiles against ones), which saves the separate pass over dy."""
    ext = _ext.load()
    if TRACE:
        sizes = (grad_w.shape[0], grad_w.shape[1], dy.shape[0], grad_b is not None and FUSE_BIAS_GRAD)
        bn, _, split = ext.wgrad_plan(*sizes)
        if ext.wgrad_swapped(*sizes):
            trace_product(x, True, dy, True, grad_w, F.EPI_OUT_F32 | F.EPI_ATOMIC | F.EPI_TRANSPOSE, split, bn)
        else:
            trace_product(dy, True, x, True, grad_w, F.EPI_OUT_F32 | F.EPI_ATOMIC, split, bn)
    ext.wgrad(dy, x, grad_w, grad_b, FUSE_BIAS_GRAD, status_word(dy.device))


def bias_grad_accumulate(dy: torch.Tensor, grad_b: torch.Tensor) -> None:
    _ext.load().colsum(dy, grad_b)


@nvtx_range("terra.layernorm")
def layernorm_cuda(x, w16, b16):
    ext = _ext.load()
    y = torch.empty_like(x)
    mean = torch.empty(x.shape[0], dtype=torch.float32, device=x.device)
    rstd = torch.empty_like(mean)
    ext.layernorm_fwd(x, w16, b16, y, mean, rstd, LN_EPS)
    return y, mean, rstd


def layernorm_bwd_cuda(dy, x, w16, mean, rstd, grad_w, grad_b, dres=None):
    ext = _ext.load()
    dx = torch.empty_like(x)
    ext.layernorm_bwd(dy, x, w16, mean, rstd, dx, grad_w, grad_b, dres)
    return dx


class ParamPack:
    """bf16 value + fp32 gradient-accumulator views of the parameters one fused block needs."""

    def __init__(self, **kw):
        self.__dict__.update(kw)


def _views(p: torch.nn.Parameter):
    if getattr(p, "bf16", None) is None:
        raise RuntimeError("CUDA path needs flattened parameters: call terra_b200.utils.flat_params.ParamArena(model)")
    return p.bf16, p.grad


def native_node(grads=()) -> bool:
    """Whether a layer may be a node in C++: not while a trace is recorded or a function transform is active (the Python nodes
    are recorded by the first and refuse the second), when single launches are to be observed, or without gradient
    accumulators (which only a backward pass asks for)."""
    for g in grads:
        if g is None:
            return False
    return not _LAUNCHES_OBSERVED and torch._C._get_tracing_state() is None and not torch._C._are_functorch_transforms_active()


def _native_half(comm, geo: WindowGeometry, impl: str) -> bool:
    """One native call runs the half when this rank owns every window and token and the small-window kernels are the
    selected ones (not in the bounds-checked build, whose reports go through the Python launches, nor when single launches
    are to be observed)."""
    return not _LAUNCHES_OBSERVED and comm is None and impl == "mma" and geo.sp == 1 and geo.tp == 1 and geo.n_wg == 1 and not _ext.DEBUG_BOUNDS


def _native_geometry(geo: WindowGeometry, num_heads, shifted, use_mask):
    return [geo.B, geo.nWh, geo.nWw, geo.wh, geo.ww, num_heads, *geo.shift(shifted), int(bool(use_mask and shifted))]


class _AttnHalfFn(torch.autograd.Function):
    @staticmethod
    def forward(ctx, x, anchor, pk: ParamPack, geo: WindowGeometry, num_heads, shifted, use_mask, scale, comm):
        ext = _ext.load()
        C = x.shape[1]
        ctx.pk, ctx.geo, ctx.args, ctx.comm = pk, geo, (num_heads, shifted, use_mask, scale), comm
        if _native_half(comm, geo, attn_forward_impl(geo.N)):
            y, mean, rstd, xn, qkv, o = ext.attn_half_fwd(
                x, pk.ln_w, pk.ln_b, pk.qkv_w, pk.qkv_b, pk.proj_w, pk.proj_b, pk.bias_table,
                _native_geometry(geo, num_heads, shifted, use_mask), scale, LN_EPS, status_word(x.device))
            ctx.save_for_backward(x, mean, rstd, xn, qkv, o)
            return y
        xn, mean, rstd = layernorm_cuda(x, pk.ln_w, pk.ln_b)
        if comm is not None:
            qkv = comm.alloc_qkv(x.shape[0], 3 * C)
            gemm(xn, pk.qkv_w, bias=pk.qkv_b, out=qkv)
            o, qkv_ptrs, out_ptrs = comm.attn_forward_buffers(qkv, C, shifted)
        else:
            qkv = gemm(xn, pk.qkv_w, bias=pk.qkv_b)
            o = torch.empty(x.shape[0], C, dtype=torch.bfloat16, device=x.device)
            qkv_ptrs, out_ptrs = [qkv.data_ptr()], [o.data_ptr()]
        sh, sw = geo.shift(shifted)
        launch_window_attn_fwd(ext, qkv_ptrs, out_ptrs, pk.bias_table, geo, C, num_heads, sh, sw, use_mask and shifted,
                               scale, x.device)
        if comm is not None:
            o, qkv = comm.attn_forward_done(o, qkv, shifted)
        y = gemm(o, pk.proj_w, bias=pk.proj_b, residual=x)
        ctx.save_for_backward(x, mean, rstd, xn, qkv, o)
        return y

    @staticmethod
    def backward(ctx, dy):
        ext = _ext.load()
        x, mean, rstd, xn, qkv, o = ctx.saved_tensors
        pk, geo, comm = ctx.pk, ctx.geo, ctx.comm
        num_heads, shifted, use_mask, scale = ctx.args
        C = x.shape[1]
        dy = dy.contiguous()
        if _native_half(comm, geo, attn_backward_impl(geo.N, C // num_heads)):
            dx = ext.attn_half_bwd(dy, x, mean, rstd, xn, qkv, o, pk.ln_w, pk.qkv_w, pk.proj_w, pk.bias_table, pk.ln_wg, pk.ln_bg,
                                   pk.qkv_wg, pk.qkv_bg, pk.proj_wg, pk.proj_bg, pk.bias_table_g,
                                   _native_geometry(geo, num_heads, shifted, use_mask), scale, FUSE_BIAS_GRAD,
                                   status_word(x.device))
            return dx, None, None, None, None, None, None, None, None
        wgrad_accumulate(dy, o, pk.proj_wg, pk.proj_bg)
        if comm is not None:
            do = comm.alloc_dout(x.shape[0], C)
            gemm(dy, pk.proj_w, b_mn=True, out=do)
            dqkv, qkv_ptrs, dout_ptrs, dqkv_ptrs = comm.attn_backward_buffers(qkv, do, shifted)
        else:
            if not qkv.is_contiguous():      # (saved-tensor hooks may hand it back in another form)
                raise RuntimeError("attention half: qkv must be contiguous [rows, 3 C]")
            do = gemm(dy, pk.proj_w, b_mn=True)
            dqkv = torch.empty_like(qkv)
            qkv_ptrs, dout_ptrs, dqkv_ptrs = [qkv.data_ptr()], [do.data_ptr()], [dqkv.data_ptr()]
        sh, sw = geo.shift(shifted)
        launch_window_attn_bwd(ext, qkv_ptrs, dout_ptrs, dqkv_ptrs, pk.bias_table, pk.bias_table_g, geo, C, num_heads, sh, sw,
                               use_mask and shifted, scale, x.device)
        if comm is not None:
            dqkv = comm.attn_backward_done(dqkv, shifted)
        wgrad_accumulate(dqkv, xn, pk.qkv_wg, pk.qkv_bg)
        dxn = gemm(dqkv, pk.qkv_w, b_mn=True)
        dx = layernorm_bwd_cuda(dxn, x, pk.ln_w, mean, rstd, pk.ln_wg, pk.ln_bg, dres=dy)
        return dx, None, None, None, None, None, None, None, None


class _MlpHalfFn(torch.autograd.Function):
    @staticmethod
    def forward(ctx, x, anchor, pk: ParamPack):
        if _LAUNCHES_OBSERVED:
            xn, mean, rstd = layernorm_cuda(x, pk.ln_w, pk.ln_b)
            act, pre = gemm(xn, pk.fc1_w, bias=pk.fc1_b, gelu=True, save_pre=True)
            y = gemm(act, pk.fc2_w, bias=pk.fc2_b, residual=x)
        else:
            y, mean, rstd, xn, pre, act = _ext.load().mlp_half_fwd(x, pk.ln_w, pk.ln_b, pk.fc1_w, pk.fc1_b, pk.fc2_w, pk.fc2_b,
                                                                   LN_EPS, status_word(x.device))
        ctx.save_for_backward(x, mean, rstd, xn, pre, act)
        ctx.pk = pk
        return y

    @staticmethod
    def backward(ctx, dy):
        x, mean, rstd, xn, pre, act = ctx.saved_tensors
        pk = ctx.pk
        dy = dy.contiguous()
        if _LAUNCHES_OBSERVED:
            wgrad_accumulate(dy, act, pk.fc2_wg, pk.fc2_bg)
            dpre = gemm(dy, pk.fc2_w, b_mn=True, dgelu_aux=pre)
            wgrad_accumulate(dpre, xn, pk.fc1_wg, pk.fc1_bg)
            dxn = gemm(dpre, pk.fc1_w, b_mn=True)
            return layernorm_bwd_cuda(dxn, x, pk.ln_w, mean, rstd, pk.ln_wg, pk.ln_bg, dres=dy), None, None
        dx = _ext.load().mlp_half_bwd(dy, x, mean, rstd, xn, pre, act, pk.ln_w, pk.fc1_w, pk.fc2_w, pk.ln_wg, pk.ln_bg, pk.fc1_wg,
                                      pk.fc1_bg, pk.fc2_wg, pk.fc2_bg, FUSE_BIAS_GRAD, status_word(x.device))
        return dx, None, None


class _LinearFn(torch.autograd.Function):
    """y = x @ W^T + b (+ residual). ``anchor`` is any parameter: it makes autograd call backward even when the
    activation input carries no gradient (first layer)."""

    @staticmethod
    def forward(ctx, x, anchor, w16, b16, wg, bg, residual, need_dx):
        y = gemm(x, w16, bias=b16, residual=residual)
        ctx.save_for_backward(x)
        ctx.p = (w16, wg, bg, residual is not None, need_dx)
        return y

    @staticmethod
    def backward(ctx, dy):
        (x,) = ctx.saved_tensors
        w16, wg, bg, has_res, need_dx = ctx.p
        dy = dy.contiguous()
        wgrad_accumulate(dy, x, wg, bg)
        dx = gemm(dy, w16, b_mn=True) if need_dx else None
        return dx, None, None, None, None, None, (dy if has_res else None), None


class LayerNormFn(torch.autograd.Function):
    """Standalone LayerNorm on the CUDA kernels (where the norm is not fused into a block half: in front of a
    collective, or for windows too large for the fused attention half). ``weight`` / ``bias`` are arena parameters;
    their gradients are accumulated in place."""

    @staticmethod
    def forward(ctx, x, weight, bias):
        y, mean, rstd = layernorm_cuda(x, weight.bf16, bias.bf16)
        ctx.save_for_backward(x, mean, rstd)
        ctx.p = (weight, bias)
        return y

    @staticmethod
    def backward(ctx, dy):
        x, mean, rstd = ctx.saved_tensors
        weight, bias = ctx.p
        dx = layernorm_bwd_cuda(dy.contiguous(), x, weight.bf16, mean, rstd, weight.grad, bias.grad)
        return dx, None, None


# ------------------------------------------------------------------------------------------------ public entry points
@nvtx_range("terra.attention_half")
def attention_half(x, mod, geo: WindowGeometry, shifted: bool, comm=None):
    """x + proj(window_attention(qkv(norm1(x)))) for a ``SwinAttentionHalf`` module ``mod``."""
    if x.is_cuda and geo.N > MAX_KERNEL_WINDOW_TOKENS:
        # large windows: the fused half needs the shared-memory kernel; compose the half from its parts instead
        a = mod.attn
        xn = LayerNormFn.apply(x.contiguous(), mod.norm1.weight, mod.norm1.bias)
        qkv = torch.cat([linear(xn, a.q_linear), linear(xn, a.k_linear), linear(xn, a.v_linear)], dim=-1)
        o = window_attention(qkv, geo, a.num_heads, shifted, a.bias_table(), mod.use_attn_mask, a.scale, comm)
        return linear(o.to(x.dtype).contiguous(), a.proj, residual=x)
    if x.is_cuda:
        fused = getattr(mod.attn, "fused", None)
        if fused is None:
            raise RuntimeError("CUDA path needs flattened parameters (ParamArena)")
        attn, ln_w, ln_b = mod.attn, mod.norm1.weight, mod.norm1.bias
        proj_w, proj_b = attn.proj.weight, attn.proj.bias
        qkv_w, qkv_b = fused["qkv_weight"], fused["qkv_bias"]
        table = attn.relative_position_bias_table if attn.use_relative_position_bias else None
        grads = [ln_w.grad, ln_b.grad, qkv_w.grad, qkv_b.grad, proj_w.grad, proj_b.grad]
        if (_native_half(comm, geo, attn_forward_impl(geo.N)) and native_node(grads)
                and attn_backward_impl(geo.N, x.shape[1] // attn.num_heads) == "mma"):
            return _ext.load().nodes.attn_half(
                x, ln_w, [ln_w.bf16, ln_b.bf16, qkv_w.bf16, qkv_b.bf16, proj_w.bf16, proj_b.bf16], grads,
                None if table is None else fp32_values(table), None if table is None else table.grad,
                _native_geometry(geo, attn.num_heads, shifted, mod.use_attn_mask), attn.scale, LN_EPS, FUSE_BIAS_GRAD,
                status_word(x.device))
        pk = ParamPack(
            ln_w=ln_w.bf16, ln_b=ln_b.bf16, ln_wg=ln_w.grad, ln_bg=ln_b.grad,
            qkv_w=qkv_w.bf16, qkv_b=qkv_b.bf16, qkv_wg=qkv_w.grad, qkv_bg=qkv_b.grad,
            proj_w=proj_w.bf16, proj_b=proj_b.bf16, proj_wg=proj_w.grad, proj_bg=proj_b.grad,
            bias_table=fp32_values(table) if table is not None else None,
            bias_table_g=table.grad if table is not None else None)
        return _AttnHalfFn.apply(x, ln_w, pk, geo, attn.num_heads, shifted, mod.use_attn_mask, attn.scale, comm)
    a = mod.attn
    xn = TF.layer_norm(x, (x.shape[-1],), mod.norm1.weight, mod.norm1.bias, LN_EPS)
    qkv = torch.cat([a.q_linear(xn), a.k_linear(xn), a.v_linear(xn)], dim=-1)
    o = window_attention(qkv, geo, a.num_heads, shifted, a.bias_table(), mod.use_attn_mask, a.scale, comm)
    return x + a.proj(o)


@nvtx_range("terra.mlp_half")
def mlp_half(x, mod):
    """x + fc2(gelu(fc1(norm2(x))))."""
    if x.is_cuda:
        ln_w, ln_b, fc1, fc2 = mod.norm2.weight, mod.norm2.bias, mod.fc1, mod.fc2
        w1, b1, w2, b2 = fc1.weight, fc1.bias, fc2.weight, fc2.bias
        grads = [ln_w.grad, ln_b.grad, w1.grad, b1.grad, w2.grad, b2.grad]
        if native_node(grads):
            return _ext.load().nodes.mlp_half(x, ln_w, [ln_w.bf16, ln_b.bf16, w1.bf16, b1.bf16, w2.bf16, b2.bf16], grads, LN_EPS,
                                              FUSE_BIAS_GRAD, status_word(x.device))
        pk = ParamPack(
            ln_w=ln_w.bf16, ln_b=ln_b.bf16, ln_wg=ln_w.grad, ln_bg=ln_b.grad,
            fc1_w=w1.bf16, fc1_b=b1.bf16, fc1_wg=w1.grad, fc1_bg=b1.grad,
            fc2_w=w2.bf16, fc2_b=b2.bf16, fc2_wg=w2.grad, fc2_bg=b2.grad)
        return _MlpHalfFn.apply(x, ln_w, pk)
    xn = TF.layer_norm(x, (x.shape[-1],), mod.norm2.weight, mod.norm2.bias, LN_EPS)
    return x + mod.fc2(TF.gelu(mod.fc1(xn)))


def linear(x, lin: torch.nn.Linear, residual=None, need_dx=True):
    """2-D ``x``; on CUDA runs the tcgen05 GEMM with the bias (and residual) fused."""
    if x.is_cuda:
        w16, wg = _views(lin.weight)
        b16, bg = _views(lin.bias) if lin.bias is not None else (None, None)
        if native_node((wg,)):
            if residual is not None and residual.dim() != 2:
                residual = residual.reshape(-1, w16.shape[0])
            return _ext.load().nodes.linear(x, lin.weight, w16, b16, wg, bg, residual, need_dx, FUSE_BIAS_GRAD, status_word(x.device))
        return _LinearFn.apply(x, lin.weight, w16, b16, wg, bg, residual, need_dx)
    y = TF.linear(x, lin.weight, lin.bias)
    return y if residual is None else y + residual
