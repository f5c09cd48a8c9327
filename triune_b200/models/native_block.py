"""Whole pre-norm blocks (``csrc/block/block_bind.cpp``): norm, recurrent mixer, norm with the residual, dense feed-forward, residual. One
native call without gradients; with them one in each direction, or two (the norm and the mixer; all that follows) for large blocks.

Issued op by op, the launches of a layer keep the host busy for 240 us (a prompt) to 950 us (forward and backward), which is what small
batches and chat turns cost; the native call issues the same launches. :func:`run` answers only for blocks of plain modules whose
parameters the kernels take as they are; everything else (hooks, adapters, quantised or replaced modules, other types and devices,
forward-mode and traced calls) gets None and runs module by module.
"""

from __future__ import annotations

from typing import Any, Optional

import torch
import torch.nn as nn
from torch.autograd import forward_ad

from .. import _ext, ops
from ..ops import gla_cuda
from .attention import HybridAttention, VectorisedGLA, format_cache, parse_cache
from .norms import RMSNorm
from .rotary import RotaryEmbedding

_TENSORS = (torch.Tensor, nn.Parameter)


def _plain(m: nn.Module, kind) -> bool:
    """Exactly this class, running nothing but the class's own forward pass."""
    return (type(m) is kind and "forward" not in m.__dict__
            and not (m._forward_hooks or m._forward_pre_hooks or m._backward_hooks or m._backward_pre_hooks))


def _rows(t, n, k, dev) -> bool:
    return (type(t) in _TENSORS and t.dtype == torch.bfloat16 and t.device == dev and t.shape == (n, k) and t.is_contiguous()
            and t.data_ptr() % 16 == 0)


def _vec(t, n, dev) -> bool:
    return t is None or (type(t) in _TENSORS and t.dtype == torch.bfloat16 and t.device == dev and t.shape == (n,) and t.is_contiguous()
                         and t.data_ptr() % 16 == 0)


# Elements of x up to which a block is one autograd function, not two. Such blocks wait for the host, to which the second function is 40 us (forward
# and backward over 2 x 300 x 384: 44 of 587 us; 7 x 256 x 768: 39 of 527). What the feed-forward saved stays until the mixer's gradients
# are there then, ten times x where it is four times as wide: 42 MB here. Above, that is memory the modules do not take.
ONE_FUNCTION = 1 << 21


def _buffers(params, want, returned=-1):
    """Where gradients of wanted parameters are added to, where they have such a buffer. The write strengths' weight (``returned``) has its
    gradient returned, wherever it is kept."""
    return [getattr(p, "main_grad", None) if p is not None and w and i != returned else None for i, (p, w) in enumerate(zip(params, want))]


def _forward_launches(T, delta):
    """Launches of the first half, forward."""
    return 6 if delta else 3 + 3 * (T >= 64) + (T % 64 != 0)


def _backward_launches(T, delta):
    return 17 if delta else 8 + 4 * (T >= 64) + 2 * (T % 64 != 0)


class _BlockFn(torch.autograd.Function):
    """x, the parameters up to the mixer and those after it -> the block's output; see ``block_forward`` and ``block_backward``."""

    @staticmethod
    def forward(ctx, x, norm1, qkvg, beta, out, norm2, up, up_bias, down, down_bias, cos, sin, H, D, eps1, eps2, scale, delta):
        mixer, after = (norm1, qkvg, beta), (out, norm2, up, up_bias, down, down_bias)
        y, *saved, status = _ext.ext().block_forward(x, mixer, after, cos, sin, H, D, eps1, eps2, scale, delta)
        ops._tick(_forward_launches(x.shape[1], delta) + 5)
        _note(status)
        ctx.save_for_backward(x, *mixer, *after, cos, sin, *saved)
        ctx.dims = (H, D, scale, delta)
        return y

    @staticmethod
    def backward(ctx, dy):
        x, *rest = ctx.saved_tensors
        params, cos, sin, saved = rest[:9], rest[9], rest[10], rest[11:]
        want_x, *want = ctx.needs_input_grad[:10]
        *grads, status = _ext.ext().block_backward(dy, x, params[:3], params[3:], _buffers(params, want, 2), want_x, want, cos, sin, saved, *ctx.dims)
        ops._tick(_backward_launches(x.shape[1], ctx.dims[3]) + 9)
        _note(status)
        return (*grads, None, None, None, None, None, None, None, None)


class _BlockMixerFn(torch.autograd.Function):
    """x and the parameters up to the mixer -> (output of the mixer, x); see ``mixer_forward`` and ``mixer_backward``. That x goes on from here
    lets its gradient from all that follows join in the norm's backward pass."""

    @staticmethod
    def forward(ctx, x, norm1, qkvg, beta, cos, sin, H, D, eps1, delta):
        params = (norm1, qkvg, beta)
        o, *saved, status = _ext.ext().mixer_forward(x, params, cos, sin, H, D, eps1, delta)
        ops._tick(_forward_launches(x.shape[1], delta))
        _note(status)
        ctx.save_for_backward(x, *params, cos, sin, *saved)
        ctx.dims = (H, D, delta)
        return o, x

    @staticmethod
    def backward(ctx, dout, ds):
        x, *rest = ctx.saved_tensors
        params, cos, sin, saved = rest[:3], rest[3], rest[4], rest[5:]
        want_x, *want = ctx.needs_input_grad[:4]
        *grads, status = _ext.ext().mixer_backward(dout, ds, x, params, _buffers(params, want, 2), want_x, want, cos, sin, saved, *ctx.dims)
        ops._tick(_backward_launches(x.shape[1], ctx.dims[2]))
        _note(status)
        return (*grads, None, None, None, None, None, None)


class _BlockRestFn(torch.autograd.Function):
    """The mixer's output, x and the parameters after the mixer -> the block's output; see ``rest_forward`` and ``rest_backward``."""

    @staticmethod
    def forward(ctx, o, x, out, norm2, up, up_bias, down, down_bias, eps2, scale):
        params = (out, norm2, up, up_bias, down, down_bias)
        y, *saved = _ext.ext().rest_forward(o, x, params, eps2, scale)
        ops._tick(5)
        ctx.save_for_backward(o, x, *params, *saved)
        ctx.scale = scale
        return y

    @staticmethod
    def backward(ctx, dy):
        o, x, *rest = ctx.saved_tensors
        params, saved = rest[:6], rest[6:]
        want = list(ctx.needs_input_grad[2:8])
        grads = _ext.ext().rest_backward(dy, o, x, params, _buffers(params, want), want, saved, ctx.scale)
        ops._tick(9)
        return (*grads, None, None)


def _note(status) -> None:
    if status is not None and status.numel():
        gla_cuda._note(status)


def _arena_ok(p) -> bool:
    g = getattr(p, "main_grad", None)
    return g is None or (g.is_cuda and g.dtype == torch.float32 and g.is_contiguous() and g.data_ptr() % 16 == 0 and g.shape == p.shape)


def run(norm1, attn, norm2, ffn, x, cache) -> Optional[Any]:
    """(output, new cache) of ``x + attn(norm1(x))`` followed by ``+ ffn(norm2(.))``, or None where the modules have to be called."""
    if not (type(x) in _TENSORS and x.is_cuda and x.dtype == torch.bfloat16 and x.dim() == 3 and x.shape[1] > 1 and x.shape[0] > 0
            and x.is_contiguous()):
        return None
    from .block import DenseFFN
    from .universal import SwiGLUFFN

    gated = type(ffn) is SwiGLUFFN
    if not (gated or type(ffn) is DenseFFN):
        return None
    if type(attn) is HybridAttention:
        if attn.use_sdpa or not _plain(attn, HybridAttention):
            return None
        attn = attn.gla
    grad = torch.is_grad_enabled()
    if (not _plain(attn, VectorisedGLA) or not _plain(norm1, RMSNorm) or not _plain(norm2, RMSNorm) or not _plain(ffn, type(ffn))
            or nn.modules.module._has_any_global_hook() or forward_ad._current_level >= 0 or torch.jit.is_tracing()
            or torch.compiler.is_compiling() or not _ext.use_kernels(x) or not _ext.ext_available() or (gated and grad)):
        return None
    out_proj, H, D, delta = attn.out_proj, attn.heads, attn.head_dim, attn.use_delta_rule
    if not _plain(out_proj, nn.Linear) or out_proj.bias is not None or D not in (64, 128) or getattr(attn, "qkvg_lora", None) is not None:
        return None
    plain_beta, beta = attn._plain_beta()
    if not plain_beta or (beta is not None and not delta):
        return None
    if gated:
        if not _plain(ffn.down, nn.Linear):
            return None
        up, up_bias, down, down_bias = ffn.gate_up, None, ffn.down.weight, None
    else:
        if len(ffn._modules) != 3:
            return None
        first, act, last = ffn._modules.values()
        if not (_plain(first, nn.Linear) and _plain(act, nn.GELU) and _plain(last, nn.Linear)):
            return None
        up, up_bias, down, down_bias = first.weight, first.bias, last.weight, last.bias
        if up_bias is None or down_bias is None:
            return None
    qkvg, out, w1, w2 = attn.qkvg_weight, out_proj.weight, norm1.weight, norm2.weight
    B, T, d = x.shape
    hd, dev, width = H * D, x.device, down.shape[1]
    if (d % 8 or d > 2048 or width % 32 or x.data_ptr() % 16 or not _rows(qkvg, 4 * hd, d, dev) or not _rows(out, d, hd, dev)
            or not _rows(up, (2 if gated else 1) * width, d, dev) or not _rows(down, d, width, dev) or not _vec(w1, d, dev) or not _vec(w2, d, dev)
            or not _vec(up_bias, width, dev) or not _vec(down_bias, d, dev) or (beta is not None and not (_rows(beta, H, d, dev) and H <= 16))):
        return None
    state, offset, fmt = parse_cache(cache)
    if torch.is_tensor(offset) or (grad and cache is not None) or offset < 0:
        return None
    if state is not None and not (type(state) is torch.Tensor and state.shape == (B, H, D, D) and state.device == dev):
        return None
    cos = sin = None
    if attn.use_rope:
        if not _plain(attn.rope, RotaryEmbedding):
            return None
        cos, sin = attn.rope.tables(T, dev, offset)
        if cos.dtype != torch.float32 or not cos.is_contiguous() or not sin.is_contiguous() or cos.shape[1] != D or cos.data_ptr() % 16 or sin.data_ptr() % 16:
            return None
    scale = 1.0 if delta else attn.out_scale
    mixer, after = (w1, qkvg, beta), (out, w2, up, up_bias, down, down_bias)
    if not grad:
        y, new_state, status = _ext.ext().block_infer(x, mixer, after, cos, sin, offset, state, H, D, norm1.eps, norm2.eps, scale, delta, gated)
        ops._tick(9 if delta else 7 + 3 * (T >= 64) + (T % 64 != 0))
        _note(status)
        return y, format_cache(new_state if cache is not None else None, cache, fmt, offset, T)
    # a mixer without gradients takes other kernels
    if not (x.requires_grad or w1.requires_grad or qkvg.requires_grad) or not all(p is None or _arena_ok(p) for p in (*mixer, *after)):
        return None
    if x.numel() <= ONE_FUNCTION:
        return _BlockFn.apply(x, *mixer, *after, cos, sin, H, D, norm1.eps, norm2.eps, scale, delta), None
    o, x = _BlockMixerFn.apply(x, *mixer, cos, sin, H, D, norm1.eps, delta)
    return _BlockRestFn.apply(o, x, *after, norm2.eps, scale), None
