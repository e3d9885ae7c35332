"""Padding and patch rearrangement of the sequential builds on CUDA: image [B, H, W, C] to patches [B, h, w, p*p*C] (feature
order p1, p2, c) and back, one copy kernel each way where ``pad`` + ``permute`` + ``reshape`` (+ crop + add) took four passes
over the field. The reference pads and rearranges with tensor operators (models/reference_model/
sequential_hierarchical_swin.py:25-449)."""
from __future__ import annotations

import torch

from .. import _ext

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
