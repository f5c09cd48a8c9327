"""One-launch decoding steps of dense recurrent models (``csrc/decode/dense_step.cu``).

:func:`plan` looks whether a model is one that the kernel states completely: a ``UniversalDenseTransformer`` of plain bf16 layers (gated
linear attention or Gated DeltaNet mixers, SwiGLU or GELU feed-forward) without hooks, adapters or replaced modules. Whatever else runs in
a model's forward pass keeps the captured step of its modules.
"""

from __future__ import annotations

from typing import List, Optional

import torch
import torch.nn as nn

from .. import _ext, ops
from ..models.attention import VectorisedGLA
from ..models.block import DenseFFN
from ..models.norms import RMSNorm
from ..models.rotary import RotaryEmbedding
from ..models.universal import SwiGLUFFN, UniversalBlock, UniversalDenseTransformer
from ..ops import gla_cuda

MAX_ROWS = 8  # sequences (csrc/decode/dense_step.cuh)
_PLAIN = (UniversalDenseTransformer, UniversalBlock, VectorisedGLA, SwiGLUFFN, DenseFFN, RMSNorm, RotaryEmbedding, nn.Linear, nn.Embedding,
          nn.ModuleList, nn.GELU)


def _plain(m: nn.Module) -> bool:
    """A module of exactly these classes that runs nothing but its class's forward pass."""
    return (type(m) in _PLAIN and "forward" not in vars(m) and getattr(m, "qkvg_lora", None) is None
            and not (m._forward_hooks or m._forward_pre_hooks))


def _weight(t: Optional[torch.Tensor], like: torch.Tensor) -> bool:
    return (t is None or (t.dtype == torch.bfloat16 and t.device == like.device and t.is_contiguous() and t.data_ptr() % 16 == 0
                          and type(t) in (torch.Tensor, nn.Parameter)))


class Step:
    def __init__(self, native):
        self.native, self.status = native, native.status

    def failed(self) -> bool:
        """Whether a step gave up on a wait. No step after it does anything, and what it left in the states and the output is not to be used."""
        return int(self.status) != 0

    def replay(self) -> None:
        """One token of every sequence, on the current stream."""
        self.native.replay()
        ops._tick(1)
        gla_cuda._note(self.status)


def plan(model, states: List[Optional[torch.Tensor]], token, out, pos, step) -> Optional[Step]:
    """The step of ``model`` from and into these buffers (states advanced in place, ``out[:, step] = token``, the next token, position and
    step count plus one), or None where the kernel does not cover it. The plan keeps the tensors that it reads."""
    if type(model) is not UniversalDenseTransformer or not _ext.use_kernels(token) or not _ext.ext_available():
        return None
    if nn.modules.module._has_any_global_hook() or not all(_plain(m) for m in model.modules()) or len(states) != len(model.layers):
        return None
    embed, head = model.embed_tokens.weight, model.lm_head.weight
    B, d = token.shape[0], embed.shape[1]
    if not model.layers or B > MAX_ROWS or d % 32 or model.lm_head.bias is not None or head.shape != embed.shape:
        return None
    first = model.layers[0]
    if type(first.attn) is not VectorisedGLA:
        return None
    H, D, delta, gated = first.attn.heads, first.attn.head_dim, first.attn.use_delta_rule, type(first.mlp) is SwiGLUFFN
    if D not in (64, 128):
        return None
    layers, scalars, weights = [], [], [embed, head, model.norm.weight]
    for layer, state in zip(model.layers, states):
        attn, mlp = layer.attn, layer.mlp
        if type(attn) is not VectorisedGLA or type(mlp) is not type(first.mlp) or type(mlp) not in (SwiGLUFFN, DenseFFN):
            return None
        if (attn.heads, attn.head_dim, attn.use_delta_rule) != (H, D, delta) or attn.out_proj.bias is not None:
            return None
        plain_beta, beta = attn._plain_beta()
        if not plain_beta or (beta is not None and not delta):
            return None
        if (not torch.is_tensor(state) or state.dtype != torch.float32 or state.shape != (B, H, D, D) or not state.is_contiguous()
                or state.device != token.device):
            return None
        cos, sin = attn.rope.tables(1, token.device, pos) if attn.use_rope else (None, None)
        up, up_bias, down = (mlp.gate_up, None, mlp.down) if gated else (mlp[0].weight, mlp[0].bias, mlp[2])
        width = down.weight.shape[1]
        if width % 32 or (gated and down.bias is not None) or (not gated and (up_bias is None or down.bias is None)):
            return None
        row = [layer.input_norm.weight, attn.qkvg_weight, beta, state, cos, sin, attn.out_proj.weight, layer.post_attn_norm.weight, up, up_bias,
               down.weight, down.bias]
        weights += [t for i, t in enumerate(row) if i not in (3, 4, 5)]
        layers.append([None if t is None else t.detach() for t in row])
        scalars.append([layer.input_norm.eps, 1.0 if delta else attn.out_scale, layer.post_attn_norm.eps])
    if not all(_weight(t, token) for t in weights):
        return None
    native = _ext.ext().DenseStepPlan(layers, scalars, embed.detach(), model.norm.weight.detach(), model.norm.eps, head.detach(), token, out, pos,
                                      step, delta, gated)
    return Step(native) if native.fits else None
