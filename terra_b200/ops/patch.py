"""Padding and patch rearrangement of the sequential builds on CUDA: image [B, H, W, C] to patches [B, h, w, p*p*C] (feature
order p1, p2, c) and back, one copy kernel each way where ``pad`` + ``permute`` + ``reshape`` (+ crop + add) took four passes
over the field; in inference, where whole patches lie inside the image, the patch layers read and write it themselves. The
reference pads and rearranges with tensor operators (models/reference_model/sequential_hierarchical_swin.py:25-449)."""
from __future__ import annotations

import torch

from .. import _ext
from . import blocks
from .conv import _pack_taps
from .gemm import status_word
from .packed import _packed

MAX_ROWS = 65535        # batch x padded rows of one launch


def patch_kernels_apply(x: torch.Tensor, padded_shape) -> bool:
    """Whether the kernels take the field ``x`` (an NHWC CUDA tensor): bf16, contiguous, rows within a launch's grid."""
    return (x.is_cuda and x.dtype == torch.bfloat16 and x.is_contiguous() and x.numel() > 0
            and x.shape[0] * padded_shape[0] <= MAX_ROWS and padded_shape[1] * x.shape[3] <= 1 << 30)


def _to_patches(image, p, padded_shape, top, left):
    B, _, _, C = image.shape
    out = torch.empty(B, padded_shape[0] // p, padded_shape[1] // p, p * p * C, device=image.device, dtype=torch.bfloat16)
    _ext.load().pad_patchify(image, out, p, top, left)
    return out


def _to_image(patches, add, shape, p, top, left):
    out = torch.empty(shape, device=patches.device, dtype=torch.bfloat16)
    _ext.load().unpatchify_crop(patches, add, out, p, top, left)
    return out


class _PadPatchifyFn(torch.autograd.Function):
    @staticmethod
    def forward(ctx, x, p, padded_shape, top, left):
        ctx.p = (x.shape, p, top, left)
        return _to_patches(x, p, padded_shape, top, left)

    @staticmethod
    def backward(ctx, g):
        shape, p, top, left = ctx.p
        return _to_image(g.contiguous(), None, shape, p, top, left), None, None, None, None


class _UnpatchifyAddFn(torch.autograd.Function):
    @staticmethod
    def forward(ctx, patches, x, p, top, left):
        ctx.p = (p, (patches.shape[1] * p, patches.shape[2] * p), top, left)
        return _to_image(patches, x, x.shape, p, top, left)

    @staticmethod
    def backward(ctx, g):
        g = g.contiguous()
        return (_to_patches(g, *ctx.p) if ctx.needs_input_grad[0] else None), (g if ctx.needs_input_grad[1] else None), None, None, None


def pad_patchify(x, p, padded_shape, top, left):
    """Zero-padded ``x`` (``top`` rows above, ``left`` columns left, up to ``padded_shape``) as patches."""
    return _PadPatchifyFn.apply(x, p, tuple(padded_shape), top, left)


def unpatchify_add(patches, x, p, top, left):
    """The image inside ``patches``, plus ``x``."""
    return _UnpatchifyAddFn.apply(patches.contiguous(), x, p, top, left)


# ------------------------------------------------------------------------------------------------ without the copies (inference)
def direct_patches_apply(x: torch.Tensor, p, top, left, dim) -> bool:
    """Whether the patch layers may read and write the field ``x`` itself, in a call that keeps nothing for a backward pass: whole patches
    inside the image and outside it, runs of whole 16-byte vectors from an address of such (tensor maps need one; the copies take any), the
    product's tables and phases."""
    _, H, W, C = x.shape
    return (x.data_ptr() % 16 == 0 and not torch.is_grad_enabled() and torch.autograd.forward_ad._current_level < 0 and blocks.native_node()
            and 1 <= p <= 4 and H % p == W % p == top % p == left % p == 0 and p * C % 8 == 0 and dim % 8 == 0
            and p * ((p * C + 63) // 64) <= 128 and (dim + 63) // 64 <= 128 and _ext.load().gemm_tma_epilogue())


def _pack_embed(w, p):
    run = w.shape[1] // p
    return _pack_taps(w, 1, 0, w.shape[0], w.shape[1], run, 1, [r * run for r in range(p)])


def _pack_recover(w, p):
    run, dim = w.shape[0] // p, w.shape[1]
    return _pack_taps(w, p, run * dim, run, dim, dim, 1, (0,), (run + 63) // 64 * 64)


def _pack_recover_bias(b, p):
    run = b.shape[0] // p
    return torch.nn.functional.pad(b.view(p, run), (0, -run % 64)).reshape(-1)


class ImageField:
    """A field whose patches and their layers are taken from the image itself, in the place of its patches (``direct_patches_apply``)."""

    def __init__(self, image, p, padded_shape, top, left):
        self.image, self.p, self.padded_shape, self.top, self.left = image, p, padded_shape, top, left

    @property
    def shape(self):
        return (self.image.shape[0], self.padded_shape[0] // self.p, self.padded_shape[1] // self.p, self.p * self.p * self.image.shape[3])

    def embed(self, lin):
        return embed_image(self.image, lin, self.p, self.padded_shape, self.top, self.left)

    def recover(self, t, lin):
        return recover_image(t, lin, self.image, self.p, self.top, self.left)


def _operand(param, kind, build):
    """The packed form of a parameter; of a graph's capture, packed by the graph, whose replays read the parameters of their time."""
    if torch.cuda.is_current_stream_capturing():
        return build(param.bf16)
    return _packed(param, param.bf16, kind, build)


def embed_image(x, lin, p, padded_shape, top, left):
    """``linear(pad_patchify(x))`` for ``direct_patches_apply`` fields: ``[B, rows, cols, N]``."""
    y = torch.empty(x.shape[0], padded_shape[0] // p, padded_shape[1] // p, lin.weight.shape[0], device=x.device, dtype=x.dtype)
    _ext.load().embed_image(x, _operand(lin.weight, f"embed{p}", lambda w: _pack_embed(w, p)), lin.bias.bf16, y, p, top // p, left // p,
                            status_word(x.device))
    return y


def recover_image(t, lin, x, p, top, left):
    """``unpatchify_add(linear(t), x)`` for ``direct_patches_apply`` fields; the sum is rounded once."""
    out = torch.empty_like(x)
    w = _operand(lin.weight, f"recover{p}", lambda v: _pack_recover(v, p))
    b = _operand(lin.bias, f"recover{p}", lambda v: _pack_recover_bias(v, p))
    _ext.load().recover_image(t.contiguous(), w, b, x, out, p, top // p, left // p, status_word(x.device))
    return out
