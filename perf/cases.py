"""The work this framework is used for, as cases that can be timed and checked: the layers of the forecast models through
their public entry points, forward and backward, and two whole calls of a model.

Sizes are those of the shipped configurations: the high-resolution model (2048 x 4320 grid, 186 channels, patch 4, width
384, windows 8 x 8), the medium one (720 x 1440, 138 channels, width 192, windows 8 x 12), the 0.1 b pretraining
configuration (2304 x 4352 padded, width 1024, 8 heads) and the small correctness grid (128 x 256, 64 channels, width 96).
Activations are bf16, the master weights and their gradients fp32, as in every configuration.

Inputs are standard normal fields; weights have the scale of a trained layer (1 / sqrt(fan in)), so that attention scores
spread over a few units. Master weights are rounded to bf16, so that the working copy and the masters agree and a 64-bit
evaluation of the same layer has the same weights.
"""
from __future__ import annotations

import math

import torch
import torch.nn.functional as TF

DEV = "cuda"
BF16 = torch.bfloat16
LN_EPS = GN_EPS = 1e-5


def listed():
    return [
        # one attention half of the correctness grid: 8 windows, every launch counts
        dict(name="attn_tiny", kind="attn", batch=1, nwh=2, nww=4, wh=8, ww=8, dim=96, heads=3, shifted=True),
        # the medium model's wide stage: 96-token windows, 16-channel heads, shifted
        dict(name="attn_medium", kind="attn", batch=1, nwh=12, nww=15, wh=8, ww=12, dim=192, heads=12, shifted=True),
        # the high-resolution model's most frequent layer: 2176 shifted windows, 12 heads of 32 channels
        dict(name="attn_high", kind="attn", batch=1, nwh=32, nww=68, wh=8, ww=8, dim=384, heads=12, shifted=True),
        # the 0.1 b pretraining configuration: 8 heads of 128 channels, a layer without shift
        dict(name="attn_pretrain", kind="attn", batch=1, nwh=36, nww=68, wh=8, ww=8, dim=1024, heads=8, shifted=False),
        # the MLP half of the high-resolution model
        dict(name="mlp_high", kind="mlp", rows=139264, dim=384),
        # a residual convolution of the medium model's down block (width not a multiple of a tile)
        dict(name="conv_medium", kind="conv", batch=1, h=96, w=180, dim=192),
        # a residual convolution of the high-resolution model's up block, at full token resolution
        dict(name="conv_high", kind="conv", batch=1, h=512, w=1088, dim=384),
        # entry of the high-resolution model: patch embedding and the stride-2 convolution
        dict(name="stem_high", kind="stem", batch=1, h=512, w=1088, dim=384, patch=4, channels=186),
        # transposed convolution of the high-resolution model's up block
        dict(name="up_high", kind="up", batch=1, h=256, w=544, dim=384),
        # exit of the high-resolution model: patch recovery with the input added, and the masked loss
        dict(name="head_high", kind="head", rows=557056, dim=384, patch=4, channels=186),
        # one forecast step of the medium model (inference: no gradients kept)
        dict(name="forecast_medium", kind="forecast", height=720, width=1440, channels=138, dim=192, depths="2,6,2",
             heads="6,12,6", wh=8, ww=12),
        # one training step of a small model: forward, loss, backward, optimizer
        dict(name="step_small", kind="step", height=128, width=256, channels=64, dim=96, depths="1,1", heads="3,6", wh=8,
             ww=8),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


WINDOWS = ((8, 8), (8, 12), (7, 7), (4, 8), (8, 8))


def _heads_for(rng, dim):
    return dim // rng.choice([hd for hd in (16, 32, 64, 128) if dim % hd == 0])


def draw(rng):
    kind = rng.choice(["attn", "attn", "attn", "mlp", "mlp", "conv", "conv", "stem", "up", "head", "forecast", "step"])
    if kind == "attn":
        wh, ww = rng.choice(WINDOWS)
        dim = rng.choice([96, 128, 192, 256, 384, 512, 768, 1024])
        windows = _log_int(rng, 4, min(2448, 156000 * 1024 // (dim * wh * ww)))
        nwh = rng.randint(2, max(2, int(math.sqrt(windows))))
        return dict(kind="attn", batch=1, nwh=nwh, nww=max(2, windows // nwh), wh=wh, ww=ww, dim=dim,
                    heads=_heads_for(rng, dim), shifted=rng.random() < 0.6)
    if kind == "mlp":
        dim = rng.choice([96, 128, 192, 256, 384, 768, 1024])
        return dict(kind="mlp", rows=_log_int(rng, 200, min(139264, 139264 * 384 * 384 // (dim * dim))), dim=dim)
    if kind == "conv":
        return dict(kind="conv", batch=rng.choice([1, 1, 2]), h=_log_int(rng, 16, 360), w=_log_int(rng, 24, 720),
                    dim=rng.choice([96, 128, 192, 256, 384]))
    if kind == "stem":
        return dict(kind="stem", batch=1, h=2 * _log_int(rng, 16, 180), w=2 * _log_int(rng, 16, 360),
                    dim=rng.choice([96, 192, 384]), patch=4, channels=rng.choice([64, 93, 138, 186]))
    if kind == "up":
        return dict(kind="up", batch=rng.choice([1, 1, 2]), h=_log_int(rng, 16, 180), w=_log_int(rng, 24, 360),
                    dim=rng.choice([96, 128, 192, 384]))
    if kind == "head":
        return dict(kind="head", rows=_log_int(rng, 2000, 300000), dim=rng.choice([96, 192, 384]), patch=4,
                    channels=rng.choice([64, 93, 138, 186]))
    if kind == "forecast":
        return dict(kind="forecast", height=_log_int(rng, 100, 720), width=_log_int(rng, 200, 1440),
                    channels=rng.choice([32, 64, 93, 138]), dim=192, depths=rng.choice(["2,2", "2,6,2", "1,3"]),
                    heads="6,12,6", wh=8, ww=rng.choice([8, 12]))
    return dict(kind="step", height=_log_int(rng, 100, 300), width=_log_int(rng, 200, 600), channels=rng.choice([32, 64, 96]),
                dim=rng.choice([96, 192]), depths="1,1", heads="3,6", wh=8, ww=rng.choice([8, 12]))


# ------------------------------------------------------------------------------------------------ shapes and weights
def _ints(text):
    return [int(v) for v in text.split(",")]


def _padded(case):
    """Grid padded to whole windows at half the patch resolution; (rows above, rows below, columns left, right)."""
    uh, uw = 4 * 2 * case["wh"], 4 * 2 * case["ww"]
    ph, pw = (-case["height"]) % uh, (-case["width"]) % uw
    return case["height"] + ph, case["width"] + pw, (ph // 2, ph - ph // 2, pw // 2, pw - pw // 2)


def _layer_heads(case):
    depths, heads = _ints(case["depths"]), _ints(case["heads"])
    return [h for d, h in zip(depths, heads) for _ in range(d)]


def _lin(name, fout, fin):
    return {name + ".weight": ((fout, fin), fin ** -0.5, 0.0), name + ".bias": ((fout,), 0.05, 0.0)}


def _norm(name, dim):
    return {name + ".weight": ((dim,), 0.1, 1.0), name + ".bias": ((dim,), 0.1, 0.0)}


def _conv(name, fout, fin, k, transposed=False):
    shape = (fin, fout, k, k) if transposed else (fout, fin, k, k)
    fan = fin if transposed else fin * k * k
    return {name + ".weight": (shape, fan ** -0.5, 0.0), name + ".bias": ((fout,), 0.05, 0.0)}


def _attn_shapes(prefix, dim, heads, wh, ww):
    out = _norm(prefix + "norm1", dim)
    out[prefix + "attn.relative_position_bias_table"] = (((2 * wh - 1) * (2 * ww - 1), heads), 0.3, 0.0)
    for part in ("q_linear", "k_linear", "v_linear", "proj"):
        out.update(_lin(prefix + "attn." + part, dim, dim))
    return out


def _mlp_shapes(prefix, dim):
    return {**_norm(prefix + "norm2", dim), **_lin(prefix + "fc1", 4 * dim, dim), **_lin(prefix + "fc2", dim, 4 * dim)}


def _shapes(case):
    """name -> (shape, spread, centre) of every parameter of the case."""
    kind, dim = case["kind"], case["dim"]
    if kind == "attn":
        return _attn_shapes("", dim, case["heads"], case["wh"], case["ww"])
    if kind == "mlp":
        return _mlp_shapes("", dim)
    if kind == "conv":
        return {**_conv("conv", dim, dim, 3), **_norm("gn", dim)}
    if kind == "stem":
        return {**_lin("embed", dim, case["patch"] ** 2 * case["channels"]), **_conv("conv", dim, dim, 3)}
    if kind == "up":
        return _conv("conv", dim, dim, 2, transposed=True)
    if kind == "head":
        return _lin("recovery", case["patch"] ** 2 * case["channels"], dim)
    feat = 16 * case["channels"]
    out = {**_lin("patch_embed.linear", dim, feat), **_lin("patch_recovery.linear", feat, dim)}
    for blk in ("down_blk", "up_blk"):
        out.update(_conv(blk + ".conv", dim, dim, 3) if blk == "down_blk" else _conv(blk + ".conv", dim, dim, 2, True))
        for i in (0, 3):
            out.update({**_conv(f"{blk}.b.{i}", dim, dim, 3), **_norm(f"{blk}.b.{i + 1}", dim)})
    for i, h in enumerate(_layer_heads(case)):
        out.update(_attn_shapes(f"layers.blocks.{i}.0.", dim, h, case["wh"], case["ww"]))
        out.update(_mlp_shapes(f"layers.blocks.{i}.1.", dim))
    return out


def _weights(case, seed):
    gen = torch.Generator(device=DEV).manual_seed(int(seed))
    return {name: (torch.randn(shape, generator=gen, device=DEV) * spread + centre).to(BF16).float()
            for name, (shape, spread, centre) in _shapes(case).items()}


def _inputs(case, seed):
    gen = torch.Generator(device=DEV).manual_seed(int(seed) + 7919)

    def field(*shape):
        return torch.randn(shape, generator=gen, device=DEV, dtype=BF16)

    kind, dim = case["kind"], case["dim"]
    if kind == "attn":
        rows = case["batch"] * case["nwh"] * case["nww"] * case["wh"] * case["ww"]
        return dict(x=field(rows, dim), dy=field(rows, dim))
    if kind == "mlp":
        return dict(x=field(case["rows"], dim), dy=field(case["rows"], dim))
    if kind == "conv":
        shape = (case["batch"], case["h"], case["w"], dim)
        return dict(x=field(*shape), dy=field(*shape))
    if kind == "stem":
        b, h, w = case["batch"], case["h"], case["w"]
        return dict(x=field(b * h * w, case["patch"] ** 2 * case["channels"]), dy=field(b, h // 2, w // 2, dim))
    if kind == "up":
        b, h, w = case["batch"], case["h"], case["w"]
        return dict(x=field(b, h, w, dim), dy=field(b, 2 * h, 2 * w, dim))

    def mask(*shape):
        return (torch.rand(shape, generator=gen, device=DEV, dtype=torch.float32) > 0.3).to(BF16)

    if kind == "head":
        feat = case["patch"] ** 2 * case["channels"]
        land = mask(case["rows"], 1).expand(case["rows"], feat).contiguous()
        shape = (case["rows"], feat)
        return dict(x=field(case["rows"], dim), patches=field(*shape), label=field(*shape) * land, mask=land)
    shape = (1, case["height"], case["width"], case["channels"])
    if kind == "forecast":
        return dict(x=field(*shape))
    land = mask(1, case["height"], case["width"], 1).expand(shape).contiguous()
    return dict(x=field(*shape), label=field(*shape) * land, mask=land)


# ------------------------------------------------------------------------------------------------ the framework's side
def _module(case):
    from terra_b200.models.hierarchical_swin import SequentialHierarchicalSwin
    from terra_b200.models.layers import MlpHalf, SwinAttentionHalf

    kind, dim = case["kind"], case["dim"]
    if kind == "attn":
        return SwinAttentionHalf(int(case["shifted"]), dim, (case["wh"], case["ww"]), case["heads"])
    if kind == "mlp":
        return MlpHalf(dim, 4 * dim)
    if kind == "conv":
        return torch.nn.ModuleDict(dict(conv=torch.nn.Conv2d(dim, dim, 3, padding=1), gn=torch.nn.GroupNorm(32, dim)))
    if kind == "stem":
        return torch.nn.ModuleDict(dict(embed=torch.nn.Linear(case["patch"] ** 2 * case["channels"], dim),
                                        conv=torch.nn.Conv2d(dim, dim, 3, stride=2, padding=1)))
    if kind == "up":
        return torch.nn.ModuleDict(dict(conv=torch.nn.ConvTranspose2d(dim, dim, 2, stride=2)))
    if kind == "head":
        return torch.nn.ModuleDict(dict(recovery=torch.nn.Linear(dim, case["patch"] ** 2 * case["channels"])))
    return SequentialHierarchicalSwin(2, num_channels=case["channels"], patch_size=4, window_size=(case["wh"], case["ww"]),
                                      height=case["height"], width=case["width"], embedding_dim=dim,
                                      depths=_ints(case["depths"]), num_heads=_ints(case["heads"]),
                                      padding_spec=dict(padded_shape=_padded(case)[:2]))


def prepare(case, seed):
    from terra_b200.ops.attention import WindowGeometry
    from terra_b200.optim.adamw import FusedAdamW
    from terra_b200.utils.flat_params import ParamArena

    mod = _module(case).to(DEV)
    weights = _weights(case, seed)
    with torch.no_grad():
        for name, p in mod.named_parameters():
            p.copy_(weights.pop(name))
    state = dict(case=case, mod=mod, arena=ParamArena(mod), **_inputs(case, seed))
    if case["kind"] == "attn":
        state["geo"] = WindowGeometry(case["batch"], case["nwh"], case["nww"], case["wh"], case["ww"])
    if case["kind"] == "step":
        state["opt"] = FusedAdamW(mod.parameters(), lr=1e-4, model=mod)
    if case["kind"] in ("attn", "mlp", "conv", "up", "head"):
        state["x"].requires_grad_(True)
    return state


def _grads(mod):
    """Parameter gradients by name; q, k and v as the one operand that the arena lays out (a key bias alone has the
    gradient zero, since it shifts all scores of a row)."""
    out = {n: p.grad for n, p in mod.named_parameters() if not any(f".{k}_linear." in "." + n for k in "qkv")}
    for name, m in mod.named_modules():
        for key, view in (getattr(m, "fused", None) or {}).items():
            out[f"{name}.{key}"] = view.grad
    return out


def run(state):
    from terra_b200.ops import blocks, conv
    from terra_b200.ops.loss import masked_loss

    case, mod = state["case"], state["mod"]
    kind, x = case["kind"], state["x"]
    if kind == "forecast":
        with torch.no_grad():
            return mod(x)
    if kind == "step":
        state["opt"].zero_grad()
        pred = mod(x)
        loss = masked_loss(pred, state["label"], state["mask"], "L1")
        loss.backward()
        state["opt"].step()
        return dict(pred=pred.detach(), loss=loss.detach(), grads=_grads(mod), weights=state["arena"].master)
    state["arena"].zero_grad()
    x.grad = None
    if kind == "head":
        pred = blocks.linear(x, mod["recovery"], residual=state["patches"])
        loss = masked_loss(pred, state["label"], state["mask"], "L1")
        loss.backward()
        return dict(pred=pred.detach(), loss=loss.detach(), dx=x.grad, grads=_grads(mod))
    if kind == "attn":
        y = blocks.attention_half(x, mod, state["geo"], case["shifted"])
    elif kind == "mlp":
        y = blocks.mlp_half(x, mod)
    elif kind == "conv":
        y = conv.groupnorm_silu(conv.conv3x3(x, mod["conv"]), mod["gn"], residual=x)
    elif kind == "stem":
        t = blocks.linear(x, mod["embed"], need_dx=False)
        y = conv.conv3x3(t.view(case["batch"], case["h"], case["w"], case["dim"]), mod["conv"], 2)
    else:
        y = conv.conv_transpose2x2(x, mod["conv"])
    y.backward(state["dy"])
    out = dict(y=y.detach(), grads=_grads(mod))
    if x.requires_grad:
        out["dx"] = x.grad
    return out


# ------------------------------------------------------------------------------------------------ what it cannot do without
def _params(case):
    return sum(math.prod(s[0]) for s in _shapes(case).values())


def _layer_flops(rows, dim, tokens):
    """Forward operations of one attention half and one MLP half."""
    return 8 * rows * dim * dim + 4 * rows * tokens * dim, 16 * rows * dim * dim


def _model_flops(case):
    ph, pw, _ = _padded(case)
    full, half, dim, feat = ph // 4 * (pw // 4), ph // 8 * (pw // 8), case["dim"], 16 * case["channels"]
    layers = sum(_layer_flops(half, dim, case["wh"] * case["ww"])) * len(_layer_heads(case))
    return layers + 4 * full * dim * feat + 18 * dim * dim * (3 * half + 2 * full) + 2 * full * dim * dim


def work(case):
    kind, dim, n = case["kind"], case["dim"], _params(case)
    state = 6 * n           # the bf16 weights read, the fp32 gradients written
    if kind in ("attn", "mlp"):
        rows = case["rows"] if kind == "mlp" else case["batch"] * case["nwh"] * case["nww"] * case["wh"] * case["ww"]
        tokens = 0 if kind == "mlp" else case["wh"] * case["ww"]
        return dict(bytes=8 * rows * dim + state, flops=3 * _layer_flops(rows, dim, tokens)[kind == "mlp"])
    if kind == "conv":
        pix = case["batch"] * case["h"] * case["w"]
        return dict(bytes=8 * pix * dim + state, flops=3 * 18 * pix * dim * dim)
    if kind == "stem":
        pix, feat = case["batch"] * case["h"] * case["w"], case["patch"] ** 2 * case["channels"]
        return dict(bytes=2 * pix * feat + pix * dim + state, flops=4 * pix * feat * dim + 3 * 18 * (pix // 4) * dim * dim)
    if kind == "up":
        pix = case["batch"] * case["h"] * case["w"]
        return dict(bytes=2 * pix * dim * 10 + state, flops=3 * 8 * pix * dim * dim)
    if kind == "head":
        rows, feat = case["rows"], case["patch"] ** 2 * case["channels"]
        return dict(bytes=2 * rows * (4 * feat + 2 * dim) + state, flops=6 * rows * feat * dim)
    field = 2 * case["height"] * case["width"] * case["channels"]
    if kind == "forecast":
        return dict(bytes=2 * field + 2 * n, flops=_model_flops(case))
    return dict(bytes=4 * field + state + 26 * n, flops=3 * _model_flops(case))


def tolerance(case):
    """bf16 activations between the kernels, fp32 sums. The layers are 0.2 to 0.5 % off a 64-bit evaluation. The head's
    gradient is that of an absolute value: where prediction and label all but meet its sign follows their rounding (1.8 % of
    the norm). The whole calls add up 10 layers (0.8 %) and a backward pass (2 %)."""
    return {"attn": {"rel": 1.5e-2}, "mlp": {"rel": 1.5e-2}, "conv": {"rel": 1e-2}, "stem": {"rel": 1e-2},
            "up": {"rel": 1e-2}, "head": {"rel": 6e-2}, "forecast": {"rel": 4e-2}, "step": {"rel": 8e-2}}[case["kind"]]


# ------------------------------------------------------------------------------------------------ the same in 64 bits
def _ln64(x, w, b):
    return TF.layer_norm(x, (x.shape[-1],), w, b, LN_EPS)


def _attn64(x, p, prefix, batch, nwh, nww, wh, ww, heads, shifted):
    """x + proj(attention(norm1(x))) on window-major rows; odd layers attend in the frame rolled by half a window."""
    dim, tokens = x.shape[1], wh * ww
    sh, sw = (wh // 2, ww // 2) if shifted else (0, 0)
    xn = _ln64(x, p[prefix + "norm1.weight"], p[prefix + "norm1.bias"])
    qkv = torch.cat([TF.linear(xn, p[f"{prefix}attn.{k}_linear.weight"], p[f"{prefix}attn.{k}_linear.bias"]) for k in "qkv"], 1)
    grid = qkv.view(batch, nwh, nww, wh, ww, 3 * dim).transpose(2, 3).reshape(batch, nwh * wh, nww * ww, 3 * dim)
    win = grid.roll((-sh, -sw), (1, 2)).view(batch, nwh, wh, nww, ww, 3 * dim).transpose(2, 3)
    q, k, v = win.reshape(batch * nwh * nww, tokens, 3, heads, dim // heads).permute(2, 0, 3, 1, 4)
    score = (q * (dim // heads) ** -0.5) @ k.transpose(-2, -1)
    at = torch.stack(torch.meshgrid(torch.arange(wh), torch.arange(ww), indexing="ij")).flatten(1).to(x.device)
    rel = at[:, :, None] - at[:, None, :]
    index = (rel[0] + wh - 1) * (2 * ww - 1) + rel[1] + ww - 1
    score = score + p[prefix + "attn.relative_position_bias_table"][index].permute(2, 0, 1)
    if shifted:
        rows, cols = torch.zeros(nwh * wh, device=x.device), torch.zeros(nww * ww, device=x.device)
        rows[-wh:-sh], rows[-sh:], cols[-ww:-sw], cols[-sw:] = 1, 2, 1, 2
        part = (rows[:, None] * 3 + cols).view(nwh, wh, nww, ww).transpose(1, 2).reshape(-1, tokens)
        apart = (part[:, :, None] != part[:, None, :]).double() * -100.0
        score = score + apart.repeat(batch, 1, 1)[:, None]
    o = torch.softmax(score, -1) @ v
    o = o.transpose(1, 2).reshape(batch, nwh, nww, wh, ww, dim).transpose(2, 3).reshape(batch, nwh * wh, nww * ww, dim)
    o = o.roll((sh, sw), (1, 2)).view(batch, nwh, wh, nww, ww, dim).transpose(2, 3).reshape(-1, dim)
    return x + TF.linear(o, p[prefix + "attn.proj.weight"], p[prefix + "attn.proj.bias"])


def _mlp64(x, p, prefix):
    xn = _ln64(x, p[prefix + "norm2.weight"], p[prefix + "norm2.bias"])
    hid = TF.gelu(TF.linear(xn, p[prefix + "fc1.weight"], p[prefix + "fc1.bias"]))
    return x + TF.linear(hid, p[prefix + "fc2.weight"], p[prefix + "fc2.bias"])


def _conv64(x, p, prefix, stride=1):
    """3 x 3 convolution with padding 1 on [B, H, W, C], tap by tap."""
    w, (_, height, width, _) = p[prefix + ".weight"], x.shape
    xp = TF.pad(x, (0, 0, 1, 1, 1, 1))
    y = p[prefix + ".bias"]
    for i in range(3):
        for j in range(3):
            y = y + xp[:, i:i + height:stride, j:j + width:stride] @ w[:, :, i, j].t()
    return y


def _up64(x, p, prefix):
    b, h, w, _ = x.shape
    weight = p[prefix + ".weight"]
    taps = torch.stack([torch.stack([x @ weight[:, :, i, j] for j in range(2)], 3) for i in range(2)], 2)
    return taps.reshape(b, 2 * h, 2 * w, weight.shape[1]) + p[prefix + ".bias"]


def _gn64(x, p, prefix, groups=32):
    b, h, w, c = x.shape
    t = x.reshape(b, h * w, groups, c // groups)
    mean = t.mean((1, 3), keepdim=True)
    var = ((t - mean) ** 2).mean((1, 3), keepdim=True)
    z = ((t - mean) * torch.rsqrt(var + GN_EPS)).reshape(b, h, w, c) * p[prefix + ".weight"] + p[prefix + ".bias"]
    return TF.silu(z)


def _model64(case, p, x):
    dim, wh, ww, feat = case["dim"], case["wh"], case["ww"], 16 * case["channels"]
    ph, pw, (top, bottom, left, right) = _padded(case)
    xp = TF.pad(x, (0, 0, left, right, top, bottom))
    patches = xp.view(1, ph // 4, 4, pw // 4, 4, -1).transpose(2, 3).reshape(1, ph // 4, pw // 4, feat)

    def residual(t, blk):
        h = _gn64(_conv64(t, p, blk + ".b.0"), p, blk + ".b.1")
        return _gn64(_conv64(h, p, blk + ".b.3"), p, blk + ".b.4") + t

    t = residual(_conv64(TF.linear(patches, p["patch_embed.linear.weight"], p["patch_embed.linear.bias"]), p, "down_blk.conv", 2),
                 "down_blk")
    nwh, nww = ph // 8 // wh, pw // 8 // ww
    rows = t.view(1, nwh, wh, nww, ww, dim).transpose(2, 3).reshape(-1, dim)
    for i, h in enumerate(_layer_heads(case)):
        rows = _attn64(rows, p, f"layers.blocks.{i}.0.", 1, nwh, nww, wh, ww, h, i % 2 == 1)
        rows = _mlp64(rows, p, f"layers.blocks.{i}.1.")
    t = rows.view(1, nwh, nww, wh, ww, dim).transpose(2, 3).reshape(1, ph // 8, pw // 8, dim)
    t = residual(_up64(t, p, "up_blk.conv"), "up_blk")
    y = TF.linear(t, p["patch_recovery.linear.weight"], p["patch_recovery.linear.bias"])
    y = y.view(1, ph // 4, pw // 4, 4, 4, -1).transpose(2, 3).reshape(1, ph, pw, -1)
    return y[:, top:top + case["height"], left:left + case["width"]] + x


def _grads64(p):
    """The gradients of ``p`` laid out as ``_grads`` gives them."""
    out = {}
    for name, t in p.items():
        head, _, tail = name.rpartition("_linear.")
        if head and head[-1] in "qkv":
            if head[-1] == "q":
                base = head[:-2]          # without ".q"
                out[f"{base}.qkv_{tail}"] = torch.cat([p[f"{base}.{k}_linear.{tail}"].grad for k in "qkv"])
        else:
            out[name] = t.grad
    return out


def _head64(p, t):
    """Recovery, masked L1 loss and their gradients, a block of rows at a time (the fields are large in 64 bits)."""
    w, b, n = p["recovery.weight"], p["recovery.bias"], t["label"].numel()
    pred = torch.empty(t["label"].shape, dtype=torch.float64, device=DEV)
    dx = torch.empty(t["x"].shape, dtype=torch.float64, device=DEV)
    gw, gb, total = torch.zeros_like(w), torch.zeros_like(b), torch.zeros((), dtype=torch.float64, device=DEV)
    for i in range(0, pred.shape[0], 65536):
        x, mask = t["x"][i:i + 65536].double(), t["mask"][i:i + 65536].double()
        y = torch.addmm(b, x, w.t()) + t["patches"][i:i + 65536].double()
        diff = y * mask - t["label"][i:i + 65536].double()
        total += diff.abs().sum()
        g = torch.sign(diff) * mask / n
        pred[i:i + 65536], dx[i:i + 65536] = y, g @ w
        gw += g.t() @ x
        gb += g.sum(0)
    return dict(pred=pred, loss=total / n, dx=dx, grads={"recovery.weight": gw, "recovery.bias": gb})


def exact(case, seed):
    kind = case["kind"]
    p = {k: v.double() for k, v in _weights(case, seed).items()}
    t = _inputs(case, seed)
    if kind == "head":
        return _head64(p, t)
    x = t["x"].double()
    if kind == "forecast":
        with torch.no_grad():
            return _model64(case, p, x)
    for v in p.values():
        v.requires_grad_(True)
    if kind == "step":
        pred = _model64(case, p, x)
        loss = (pred * t["mask"].double() - t["label"].double()).abs().mean()
        loss.backward()
        return dict(pred=pred.detach(), loss=loss.detach(), grads=_grads64(p), weights=None)
    if kind != "stem":
        x.requires_grad_(True)
    if kind == "attn":
        y = _attn64(x, p, "", case["batch"], case["nwh"], case["nww"], case["wh"], case["ww"], case["heads"], case["shifted"])
    elif kind == "mlp":
        y = _mlp64(x, p, "")
    elif kind == "conv":
        y = _gn64(_conv64(x, p, "conv"), p, "gn") + x
    elif kind == "stem":
        emb = TF.linear(x, p["embed.weight"], p["embed.bias"])
        y = _conv64(emb.view(case["batch"], case["h"], case["w"], case["dim"]), p, "conv", 2)
    else:
        y = _up64(x, p, "conv")
    y.backward(t["dy"].double())
    out = dict(y=y.detach(), grads=_grads64(p))
    if x.requires_grad:
        out["dx"] = x.grad
    return out
