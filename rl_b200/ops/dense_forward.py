"""Inference pass of packed sequences through plain dense decoder layers in one native call (``rlb_dense_forward``): the kernels of the layer-by-layer
path without a trip through Python for each of them."""

from __future__ import annotations

import ctypes as C
import math
from typing import Optional, Sequence

import torch
from torch.nn.modules import module as _module

from . import attention as _attention
from . import functional as F
from . import lib as _L
from .lib import Counters, call, ptr, stream_ptr, use_native

_P, _I, _LL, _F = C.c_void_p, C.c_int, C.c_longlong, C.c_float
_WEIGHTS = ("norm1", "qkv", "o", "norm2", "gate_up", "down", "q_norm", "k_norm", "qkv_bias")


class _Layer(C.Structure):
    _fields_ = [(n, _P) for n in (*_WEIGHTS, "inv_freq", "k_cache", "v_cache")]


class _Forward(C.Structure):
    _fields_ = [(n, _P) for n in ("layers", "h", "out", "mid", "x", "qkv", "att", "gate_up", "act", "positions", "cu_seqlens", "slots", "status")]
    _fields_ += [(n, _I) for n in ("L", "T", "B", "d", "Hq", "Hkv", "D", "F", "block_size")]
    _fields_ += [("num_blocks", _LL), ("eps", _F), ("scale", _F)]


_L.register("rlb_dense_forward", [_P, _P])


def _weights(layer) -> Optional[tuple]:
    """The layer's tensors in the order of ``_WEIGHTS``, or None where it is anything but norm, attention, norm, gated unit on plain bf16 weights
    (adapters, quantised copies, hooks and replaced methods are the layer-by-layer path's)."""
    from rl_b200.models.transformer import Attention, DecoderLayer, DenseMLP

    if type(layer) is not DecoderLayer or layer.cfg.sandwich_norm:
        return None
    mods = layer._modules      # (attribute access of modules and parameters by name goes through a Python function each time)
    at, mlp = mods["self_attn"], mods["mlp"]
    if type(at) is not Attention or type(mlp) is not DenseMLP or not mlp.gated or mlp.act != "silu" or at.cp is not None or at.tp.world > 1 or mlp.tp.world > 1:
        return None
    if at.qkv_lora is not None or at.o_lora is not None or mlp.gate_up_lora is not None or mlp.down_lora is not None:
        return None
    for m in (layer, at, mlp):
        if m._forward_hooks or m._forward_pre_hooks or "forward" in m.__dict__:
            return None
    own, a, f = layer._parameters, at._parameters, mlp._parameters
    ws = (own["input_layernorm"], a["qkv_proj"], a["o_proj"], own["post_attention_layernorm"], f["gate_up_proj"], f["down_proj"], a.get("q_norm"), a.get("k_norm"),
          a.get("qkv_bias"))
    if any(w.dim() != 2 or not w.numel() for w in (ws[1], ws[2], ws[4], ws[5])):      # (sharded elsewhere)
        return None
    for w in ws:
        if w is not None and (w.dtype != torch.bfloat16 or not w.is_contiguous() or w.data_ptr() % 16 or "_rlb_qat" in w.__dict__ or "_rlb_q" in w.__dict__):
            return None
    return ws


def dense_forward(layers: Sequence, h: torch.Tensor, positions: torch.Tensor, inv_freqs: Sequence[torch.Tensor], cu_seqlens: torch.Tensor, max_seqlen: int, *,
                  slots: Optional[torch.Tensor] = None, k_caches: Sequence = (), v_caches: Sequence = ()) -> Optional[torch.Tensor]:
    """The residual stream after ``layers``, or None where this path does not cover them: then nothing has been done. ``inv_freqs``: one per layer.
    ``slots``: the rotated keys and the values also go to these places of the layers' caches."""
    c = layers[0].cfg if len(layers) else None
    if c is None or torch.is_grad_enabled() or not use_native(h) or h.dtype != torch.bfloat16 or not h.is_contiguous() or h.shape[0] == 0 or h.data_ptr() % 16:
        return None
    D = c.head_dim
    if D not in _attention.NATIVE_HEAD_DIMS or F._attn_impl is not _attention.attention_native or _module._has_any_global_hook() or type(h) is not torch.Tensor:
        return None
    if c.hidden_size % 8 or any(layer.window and max_seqlen > layer.window for layer in layers):
        return None
    if slots is not None and not all(k.dtype == torch.bfloat16 and k.is_contiguous() for k in (*k_caches, *v_caches)):
        return None
    weights = [_weights(layer) for layer in layers]
    if any(w is None for w in weights):
        return None
    at = layers[0].self_attn
    Hq, Hkv, (T, d), ff = at.hq, at.hkv, h.shape, layers[0].mlp.down_proj.shape[1]
    if ff % 8 or any(w[5].shape[1] != ff or w[1].shape != weights[0][1].shape for w in weights):
        return None
    keep = []      # what the call reads: on this stream until the kernels have run
    array = (_Layer * len(layers))()
    for i, (slot, w, freq) in enumerate(zip(array, weights, inv_freqs)):
        w = list(w)
        if w[8] is not None:
            w[8] = w[8].float()
            keep.append(w[8])
        for name, t in zip(_WEIGHTS, w):
            setattr(slot, name, ptr(t))
        slot.inv_freq = freq.data_ptr()
        if slots is not None:
            slot.k_cache, slot.v_cache = k_caches[i].data_ptr(), v_caches[i].data_ptr()
    positions, cu = positions.to(torch.int32), cu_seqlens.to(torch.int32)
    new = lambda *shape: torch.empty(shape, dtype=torch.bfloat16, device=h.device)      # noqa: E731
    out, mid, x, qkv, att, act = new(T, d), new(T, d), new(T, d), new(T, (Hq + 2 * Hkv) * D), new(T, Hq * D), new(T, ff)
    gu = new(T, 2 * ff)
    call("rlb_dense_forward", C.byref(_Forward(
        layers=C.cast(array, _P), h=ptr(h), out=ptr(out), mid=ptr(mid), x=ptr(x), qkv=ptr(qkv), att=ptr(att), gate_up=ptr(gu), act=ptr(act),
        positions=ptr(positions), cu_seqlens=ptr(cu), slots=ptr(slots),
        status=ptr(_L.status_word(h.device)), L=len(layers), T=T, B=cu.numel() - 1, d=d, Hq=Hq, Hkv=Hkv, D=D, F=ff,
        block_size=k_caches[0].shape[2] if slots is not None else 0,
        num_blocks=k_caches[0].shape[0] if slots is not None else 0, eps=c.rms_norm_eps,
        scale=c.attn_scale if c.attn_scale is not None else 1.0 / math.sqrt(D))), stream_ptr())
    Counters.launches += len(layers) * (9 + bool(c.qk_norm)) - 1
    return out
