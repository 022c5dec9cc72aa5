"""``forward_with_states`` of both model families as one native call (``csrc/stream.cu``): the kernels of the layer-by-layer route, issued without
a Python step, an autograd call and an allocation per kernel. A decoding step of 4 layers took 1.1 ms to issue that way for 0.3 ms of kernels.

Each function returns ``None`` for what it does not handle - a gradient wanted, another type, layout or device, tensor or context parallelism,
quantised layers, parameters that are fetched on use, hooks or replaced methods, transforms, forward mode and tracing, states that are not plain - and the
model takes the general route.

reference: ``src/model/model.zig:415-454`` (streaming with carried states), ``src/eval/evaluator.zig:419-470``.
"""
from __future__ import annotations

import ctypes
from typing import List, Optional

import torch
import torch.nn as nn
from torch.nn.modules import module as nn_module

from ..native import lib, plain_eager, stream_ptr
from ..ops import efla as eops
from ..ops.attention import DECODE_HEAD_DIMS, DECODE_ROWS
from ..ops.nn import _EW

_ACTS = {"swiglu": -1, "gelu": 0, **{k: v[0] for k, v in _EW.items() if k != "gelu"}}


def _plain_mode() -> bool:
    """Eager execution without a gradient (a state may be a dual tensor, whose tangent the layers refuse to drop), and no hooks on all modules."""
    return plain_eager() and not nn_module._has_any_global_hook()


def _eager(ids: torch.Tensor) -> bool:
    """CUDA token ids in plain eager execution."""
    return type(ids) is torch.Tensor and ids.is_cuda and ids.dtype == torch.int64 and ids.dim() == 2 and ids.numel() > 0 and _plain_mode()


_WRITTEN = []           # (attributes of a class, name, function), as the classes were written; live views of the attributes
_CALL = nn.Module.__call__


def stands_in_for(*names: str):
    """Marks a class whose methods of these names the native call does the work of: replaced on the class or on an instance, they are called again."""
    def mark(kind: type) -> type:
        _WRITTEN.extend((vars(kind), n, vars(kind)[n]) for n in names)
        return kind
    return mark


def _as_written() -> bool:
    """The marked classes still have the methods that they were written with, and modules are called as ever."""
    for attributes, name, f in _WRITTEN:
        if attributes.get(name) is not f or "__call__" in attributes:
            return False
    return nn.Module.__call__ is _CALL


def _plain(module: nn.Module, kind: type) -> bool:
    d = module.__dict__
    return type(module) is kind and "forward" not in d and not d["_forward_hooks"] and not d["_forward_pre_hooks"] and "_compiled_call_impl" not in d


def _same_norms(a, b, c) -> bool:
    return a.kind == b.kind == c.kind and a.eps == b.eps == c.eps


def _address(t: Optional[torch.Tensor], device, dtype=torch.bfloat16) -> int:
    """Where a contiguous, 16-byte aligned tensor lies; 0 for what the kernels cannot take as it is."""
    if type(t) not in (torch.Tensor, nn.Parameter) or t.dtype != dtype or t.device != device or not t.is_contiguous():
        return 0
    a = t.data_ptr()
    return a if a % 16 == 0 else 0


def _weights(device, out: List[int], *params) -> bool:
    """Appends the addresses of the parameters, given with their shapes (0 for an absent bias); False when one of them is not plain."""
    for w, shape in params:
        if w is None:
            out.append(0)
            continue
        if type(w) is not nn.Parameter or w.shape != shape or w.dtype != torch.bfloat16 or w.device != device or not w.is_contiguous() \
                or "_gemm_gather" in w.__dict__:
            return False
        a = w.data_ptr()
        if a % 16:
            return False
        out.append(a)
    return True


def _array(kind, values):
    return ctypes.addressof(arr := (kind * len(values))(*values)), arr


def _quantised(q) -> bool:
    return q is not None and q.enabled


def gpt_stream(model, ids: torch.Tensor, states: dict):
    """``(logits [B, T, V], states)`` of :meth:`GPTModel.forward_with_states`, or ``None``."""
    from .gpt import MLP, Attention, Block, GPTModel, Norm
    if not (_eager(ids) and _as_written() and type(model) is GPTModel and "hidden_states" not in model.__dict__ and model.dtype == torch.bfloat16):
        return None
    dev = ids.device
    B, S = ids.shape
    tok, pos, fin, blocks = model.embed_tokens, model.pos_embed, model.final_norm, model.blocks
    head = model.lm_head if model.lm_head is not None else tok
    pos0, D = states["pos"], tok.shape[1]
    if not _plain(fin, Norm) or not len(blocks) or not _plain(blocks[0], Block) or len(states["layers"]) != len(blocks) \
            or type(states["layers"][0]) is not dict or (pos is not None and pos0 + S > pos.shape[0]) or model.vocab_lo != 0:
        return None
    first, cache0 = blocks[0], states["layers"][0]
    if not (_plain(first.attn, Attention) and _plain(first.mlp, MLP)):
        return None
    at, act = first.attn, first.mlp.act
    H, Hkv, hd, F = at.n_heads, at.n_kv_heads, at.head_dim, first.mlp.down.shape[0]
    k0 = cache0.get("k")
    t = k0.shape[0] if k0 is not None else 0
    if (k0 is not None and not t) or act not in _ACTS or (act == "swiglu" and F % 8):
        return None
    if (hd not in DECODE_HEAD_DIMS or S * (H // Hkv) > DECODE_ROWS) if t else (hd % 8 or hd > 128):
        return None
    ptrs: List[int] = []
    V, N = head.shape[0], (H + 2 * Hkv) * hd
    vec = (D,)
    if V != model.cfg.model.vocab_size:
        return None
    if not _weights(dev, ptrs, (tok, (V, D)), (pos, pos.shape if pos is not None else ()), (fin.weight, vec), (fin.bias, vec), (head, (V, D))):
        return None
    if pos is not None and pos.shape[1] != D:
        return None
    outs = []
    per_layer: List[int] = []
    for blk, cache in zip(blocks, states["layers"]):
        if not _plain(blk, Block) or type(cache) is not dict:
            return None
        a, m, n1, n2 = blk.attn, blk.mlp, blk.ln1, blk.ln2
        if not (_plain(a, Attention) and _plain(m, MLP) and _plain(n1, Norm) and _plain(n2, Norm)) \
                or a.pc.tp_size != 1 or a.pc.cp_size != 1 or _quantised(a.quant) or _quantised(m.quant) or (blk.dropout > 0 and blk.training) \
                or (a.n_heads, a.n_kv_heads, a.head_dim, m.act, m.gated) != (H, Hkv, hd, act, act == "swiglu") or not _same_norms(fin, n1, n2):
            return None
        if not _weights(dev, per_layer, (n1.weight, vec), (n1.bias, vec), (a.w_qkv, (D, N)), (a.w_o, (H * hd, D)), (n2.weight, vec), (n2.bias, vec),
                        (m.up, (D, 2 * F if act == "swiglu" else F)), (m.down, (F, D))):
            return None
        k, v = cache.get("k"), cache.get("v")
        if t:
            if k is None or v is None or k.shape != (t, B, Hkv, hd) or v.shape != k.shape or k.requires_grad or v.requires_grad:
                return None
            ka, va = _address(k, dev), _address(v, dev)
            if not (ka and va):
                return None
        elif k is not None or v is not None:
            return None
        else:
            ka = va = 0
        ko, vo = (torch.empty((t + S, B, Hkv, hd), dtype=torch.bfloat16, device=dev) for _ in range(2))
        outs.append((ko, vo))
        per_layer += (ka, va, ko.data_ptr(), vo.data_ptr())
    ids_sb = ids.t().contiguous()
    logits = torch.empty((S, B, V), dtype=torch.bfloat16, device=dev)
    dims, keep_dims = _array(ctypes.c_longlong, (S, B, D, H, Hkv, hd, F, V, len(blocks), pos0, t, _ACTS[act], fin.kind, int(pos is not None)))
    work = torch.empty(lib.raw("elfa_gpt_stream_work")(dims) * 1024, dtype=torch.uint8, device=dev)
    p, keep = _array(ctypes.c_uint64, [ids_sb.data_ptr(), *ptrs, logits.data_ptr(), work.data_ptr(), *per_layer])
    lib.call("elfa_gpt_stream", p, dims, float(fin.eps), stream_ptr(logits))
    for cache, (ko, vo) in zip(states["layers"], outs):
        cache["k"], cache["v"] = ko, vo
    states["pos"] = pos0 + S
    return logits.transpose(0, 1), states


def efla_stream(model, ids: torch.Tensor, states: List[dict]):
    """``(logits [B, T, V], states)`` of :meth:`EflaModel.forward_with_states`, or ``None``."""
    from .efla_model import EflaBlock, EflaLayer, EflaModel, PrismLayer
    from .gpt import Norm
    if not (_eager(ids) and _as_written() and type(model) is EflaModel
            and model.__dict__.keys().isdisjoint(("hidden_states", "_embed", "_logits")) and model.dtype == torch.bfloat16 and model.pc.tp_size == 1):
        return None
    dev = ids.device
    B, T = ids.shape
    tok, fin, blocks = model.embed_tokens, model.final_norm, model.blocks
    head = model.lm_head if model.lm_head is not None else tok
    if not _plain(fin, Norm) or not len(blocks) or not _plain(blocks[0], EflaBlock) or len(states) != len(blocks) or type(states[0]) is not dict:
        return None
    D, first = tok.shape[1], blocks[0]
    if not _plain(first.efla, EflaLayer) or (first.prism is not None and not _plain(first.prism, PrismLayer)):
        return None
    H, d, act, F = first.efla.H, first.efla.d, first.act, first.mlp_up.shape[1]
    prism = first.prism is not None
    L, W = (first.prism.L, first.prism.conv_weight.shape[1]) if prism else (0, 1)
    if act not in _ACTS or act == "swiglu" or d not in (32, 64, 96, 128) or D % d or model.vocab_lo != 0:
        return None
    if prism and not (1 <= L <= 8 and W <= 128):
        return None
    tail0 = states[0].get("conv_tail") if prism else None
    tail = tail0.shape[1] if tail0 is not None else 0
    ptrs: List[int] = []
    V, vec = head.shape[0], (D,)
    if V != model.cfg.model.vocab_size or not _weights(dev, ptrs, (tok, (V, D)), (fin.weight, vec), (fin.bias, vec), (head, (V, D))):
        return None
    per_layer: List[int] = []
    forget: List[float] = []
    numbers, gate = tuple(str(i) for i in range(L)), (D, d)
    new_states = []
    for blk, st in zip(blocks, states):
        if not _plain(blk, EflaBlock) or type(st) is not dict:
            return None
        e, pr, n1, n2 = blk.efla, blk.prism, blk.ln1, blk.ln2
        if not (_plain(e, EflaLayer) and _plain(n1, Norm) and _plain(n2, Norm)) or blk.pc.tp_size != 1 or e.pc.tp_size != 1 \
                or (pr is not None) != prism or (prism and not (_plain(pr, PrismLayer) and pr.L == L and pr.d == d)) \
                or (e.H, e.d, blk.act) != (H, d, act) or not _same_norms(fin, n1, n2):
            return None
        s0, p0, ct = st.get("efla"), st.get("prism"), st.get("conv_tail")
        beta = e.beta_param
        sa = _address(s0, dev, torch.float32) if s0 is not None and s0.shape == (B, H, d, d) else 0
        if not sa or type(beta) is not nn.Parameter or beta.dtype != torch.float32 or beta.device != dev or beta.shape != (1,) or s0.requires_grad:
            return None
        conv = (pr.conv_weight, pr.conv_bias) if prism else (None, None)
        if not _weights(dev, per_layer, (n1.weight, vec), (n1.bias, vec), (e.w_k, (D, H * d)), (e.w_v, (D, H * d)), (e.w_o, (H * d, D))):
            return None
        per_layer.append(beta.data_ptr())
        if not _weights(dev, per_layer, (conv[0], (D, W)), (conv[1], vec), (n2.weight, vec), (n2.bias, vec), (blk.mlp_up, (D, F)), (blk.mlp_down, (F, D))):
            return None
        s1 = torch.empty_like(s0)
        per_layer += (sa, s1.data_ptr())
        p1 = new_tail = None
        if prism:
            pa = _address(p0, dev, torch.float32) if p0 is not None and p0.shape == (B, D // d, d, d) else 0
            if not pa or p0.requires_grad or (ct is not None) != bool(tail):
                return None
            if tail and (type(ct) is not torch.Tensor or ct.shape != (B, tail, D) or ct.dtype != torch.bfloat16 or ct.device != dev or ct.stride(2) != 1 or ct.stride(1) != D
                         or ct.requires_grad or ct.data_ptr() % 4 or ct.stride(0) % 2):       # read two channels, four bytes, at a time
                return None
            p1 = torch.empty_like(p0)
            xin = torch.empty((B, tail + T, D), dtype=torch.bfloat16, device=dev)
            new_tail = xin[:, -(W - 1):] if W > 1 else None
            per_layer += (pa, p1.data_ptr(), ct.data_ptr() if tail else 0, ct.stride(0) if tail else 0, xin.data_ptr())
            for ws in (pr.w_p, pr.w_beta, pr.w_k):
                own = ws._parameters               # by position; indexing the list looks each one up by name, a microsecond apiece
                if tuple(own) != numbers or len(ws) != L or not _weights(dev, per_layer, *[(w, gate) for w in own.values()]):
                    return None
            forget.append(float(pr.forget))
        else:
            if p0 is not None:
                return None
            per_layer += (0,) * 5
            forget.append(0.0)
        new_states.append({"efla": s1, "prism": p1, "conv_tail": new_tail})
    ids_c = ids.contiguous()
    logits = torch.empty((B, T, V), dtype=torch.bfloat16, device=dev)
    steps = eops._efla_step_tokens(B * H * d * d)
    dims, keep_dims = _array(ctypes.c_longlong, (B, T, D, H, d, F, V, len(blocks), L, W, _ACTS[act], fin.kind, int(prism), tail))
    work = torch.empty(lib.raw("elfa_efla_stream_work")(dims, steps) * 1024, dtype=torch.uint8, device=dev)
    p, keep = _array(ctypes.c_uint64, [ids_c.data_ptr(), *ptrs, logits.data_ptr(), work.data_ptr(), *per_layer])
    f, keep_f = _array(ctypes.c_float, forget)
    lib.call("elfa_efla_stream", p, dims, f, float(fin.eps), steps, stream_ptr(logits))
    return logits, new_states
