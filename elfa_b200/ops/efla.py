"""EFLA (error-free linear attention), PRISM refinement and ShortConv ops.

Math restated from the reference (all three are host loops there):

* EFLA recurrence per (batch, head) with state ``S [d, d]`` (row = key index, column = value index):
  ``lam = |k_t|^2``, ``c = (1 - exp(-beta*lam)) / lam`` (series ``beta - beta^2 lam/2 + beta^3 lam^2/6``
  for ``lam < 1e-6``), ``p = S^T k_t``, ``S += c * k_t (v_t - p)^T``, ``o_t = S^T k_t`` with the updated
  state (reference: ``src/model/efla.zig:27-49,275-329``; CUDA ``kernels/cuda/efla.cu:93-197``,
  ``kernels/cuda/efla_scan.cu:99-152``). Note ``o_t = p + c*lam*(v_t - p)``, which the kernels use.
* chunk / cross-device composition: the update is affine in ``S`` (``S' = (I - c k k^T) S + c k v^T``), so
  chunks compose as affine maps ``(A, B)``; the reference adds chunk states, which is only right for
  additive linear attention (``efla.zig:702-732``, ``efla.cu:534-552``).
* PRISM (``src/model/prism.zig:318-421``): ``u = ShortConv(x)``; residual ``r = v - u`` per group of ``d``
  channels; per iteration ``l``: ``p = sigmoid(u W_p^l)``, ``delta = gelu(p * r)``, ``r -= delta``,
  ``refined += delta``; output ``u + refined``. The fast-weight state it also maintains never feeds
  back into the output within a step; :func:`prism_state_update` computes it for state carry.
* ShortConv (``prism.zig:948-973``, ``kernels/cuda/convolution.cu:4-57``):
  ``y[b,t,c] = bias[c] + sum_w x[b,t-w,c] * weight[c,w]`` (zero for ``t-w < 0``).
"""
from __future__ import annotations

import ctypes
import functools
from typing import Optional, Tuple

import torch

from ..native import NativeError, lib, plain_eager, stream_ptr
from .gemm import gelu_tanh_ref, gemm, linear


def stable_coefficient(beta: torch.Tensor, lam: torch.Tensor) -> torch.Tensor:
    small = lam < 1e-6
    safe = torch.where(small, torch.ones_like(lam), lam)
    big = (1.0 - torch.exp(-beta * safe)) / safe
    ser = beta - 0.5 * beta * beta * lam + beta ** 3 * lam * lam / 6.0
    return torch.where(small, ser, big)


def efla_scan_ref(k: torch.Tensor, v: torch.Tensor, beta: torch.Tensor, state: Optional[torch.Tensor] = None
                  ) -> Tuple[torch.Tensor, torch.Tensor]:
    """k, v ``[B, T, H, d]`` → (o ``[B, T, H, d]``, final state ``[B, H, d, d]``), fp32, differentiable."""
    B, T, H, d = k.shape
    kf, vf = k.float(), v.float()
    S = torch.zeros(B, H, d, d, dtype=torch.float32, device=k.device) if state is None else state.float()
    outs = []
    b = beta.float().reshape(())
    for t in range(T):
        kt, vt = kf[:, t], vf[:, t]                       # [B, H, d]
        lam = (kt * kt).sum(-1)                           # [B, H]
        c = stable_coefficient(b, lam)
        p = torch.einsum("bhi,bhij->bhj", kt, S)
        S = S + c[..., None, None] * kt[..., :, None] * (vt - p)[..., None, :]
        outs.append(torch.einsum("bhij,bhi->bhj", S, kt))
    return torch.stack(outs, 1), S


def efla_scan_chunked_ref(k: torch.Tensor, v: torch.Tensor, beta: torch.Tensor, state: Optional[torch.Tensor] = None, chunk: int = 64
                          ) -> Tuple[torch.Tensor, torch.Tensor]:
    """The same recurrence in chunk-parallel (WY) form: everything inside a chunk of ``C`` tokens is matrix products,
    only ``T / C`` steps remain sequential. With ``K, V [C, d]`` the chunk's keys / values, ``c`` its coefficients and
    ``S0`` the state at its start, the pseudo-values ``u_t = c_t (v_t - S_{t-1}^T k_t)`` satisfy
    ``(I + diag(c) tril(K K^T, -1)) U = diag(c) (V - K S0)``, so with ``Tm = (I + diag(c) tril(K K^T, -1))^{-1} diag(c)``
    (a unit-lower-triangular solve, independent of the state and hence parallel over all chunks):
    ``U = Tm V - (Tm K) S0``, ``O = K S0 + tril(K K^T) U``, ``S_end = S0 + K^T U``.
    fp32, differentiable; equal to :func:`efla_scan_ref` up to rounding. The CUDA kernels take this form
    with 32 tokens per chunk; here it is their oracle and a faster CPU path for long sequences."""
    B, T, H, d = k.shape
    C = min(chunk, T)
    pad = (-T) % C
    kf, vf = k.float(), v.float()
    if pad:        # zero keys change nothing: their update and their output are zero
        kf = torch.nn.functional.pad(kf, (0, 0, 0, 0, 0, pad))
        vf = torch.nn.functional.pad(vf, (0, 0, 0, 0, 0, pad))
    nc = (T + pad) // C
    K = kf.view(B, nc, C, H, d).permute(0, 3, 1, 2, 4)                     # [B, H, nc, C, d]
    V = vf.view(B, nc, C, H, d).permute(0, 3, 1, 2, 4)
    c = stable_coefficient(beta.float().reshape(()), (K * K).sum(-1))      # [B, H, nc, C]
    G = K @ K.transpose(-1, -2)                                            # [B, H, nc, C, C]
    A = torch.eye(C, dtype=torch.float32, device=k.device) + c.unsqueeze(-1) * torch.tril(G, -1)
    W = torch.linalg.solve_triangular(A, c.unsqueeze(-1) * torch.cat((V, K), -1), upper=False, unitriangular=True)
    Wv, Wk = W[..., :d], W[..., d:]                                        # Tm V, Tm K
    Gi = torch.tril(G)
    S = torch.zeros(B, H, d, d, dtype=torch.float32, device=k.device) if state is None else state.float()
    outs = []
    for n in range(nc):                                                     # the only sequential part
        Kn = K[:, :, n]
        U = Wv[:, :, n] - Wk[:, :, n] @ S
        outs.append(Kn @ S + Gi[:, :, n] @ U)
        S = S + Kn.transpose(-1, -2) @ U
    o = torch.stack(outs, 2).permute(0, 2, 3, 1, 4).reshape(B, nc * C, H, d)
    return o[:, :T], S


_EFLA_CHUNK = 32           # tokens of a chunk of the tensor-core kernels


def _efla_step_tokens(states: int) -> int:
    """Up to this many tokens a call without a gradient goes token by token, in one launch; the chunked form takes two launches and two
    workspaces. ``states``: state elements of the call, ``B H d^2``. The line lies where whole calls cross, one after the other with the
    host's part included (microseconds, token form / chunked form):
    2^18 (1 x 16 heads of 64): T 64 21 / 31, T 112 27 / 31, T 128 31 / 31; 2^19 (8 x 16 of 64): T 112 30 / 31, T 128 33 / 31;
    2^20 (16 x 16 of 64): T 96 31 / 31, T 112 37 / 31; 2^21 (8 x 16 of 128): T 64 29 / 31, T 80 35 / 31;
    2^22 (8 x 32 of 128): T 32 29 / 31, T 48 42 / 31; 2^23 (16 x 32 of 128): T 17 31 / 33, T 24 39 / 35.
    Past 2^19 the device's time counts: the token form's grows with tokens times states."""
    return 112 if states <= 1 << 19 else max(16, min(96, (1 << 27) // states))


def _aligned(t: torch.Tensor) -> torch.Tensor:
    """``t``, contiguous and on a 16-byte boundary (the kernels copy 16 bytes at a time)."""
    if not t.is_contiguous():
        t = t.contiguous()
    return t if t.data_ptr() % 16 == 0 else t.clone()


@functools.lru_cache(maxsize=1024)
def _efla_segments(B: int, T: int, H: int, d: int, train: bool) -> int:
    """Into how many segments the kernels cut the walk over the chunks: a rule on the sizes alone, asked once for each."""
    return lib.raw("elfa_efla_segments_train" if train else "elfa_efla_segments")(B, T, H, d)


def _efla_scratch(n: int, k: torch.Tensor, B: int, H: int, d: int) -> torch.Tensor:
    """Start, map and offset of each segment."""
    return torch.empty(3 * n * B * H * d * d, dtype=torch.float32, device=k.device)


def _efla_forward(k, v, beta, state, want_grad):
    """``(o, final state)`` and, where a gradient is wanted, what backward needs; ``beta`` one fp32 number on the device."""
    B, T, H, d = k.shape
    kc, vc = _aligned(k), _aligned(v)
    o = torch.empty_like(kc)
    s_out = torch.empty((B, H, d, d), dtype=torch.float32, device=k.device)
    if state is not None and (state.dtype != torch.float32 or not state.is_contiguous()):
        state = state.float().contiguous()
    if not want_grad and (T <= 16 or T <= _efla_step_tokens(B * H * d * d)):
        lib.call("elfa_efla_scan_fwd", kc, vc, beta, state, o, s_out, B, T, H, d, stream_ptr(kc))
        return o, s_out
    nchunks = (T + _EFLA_CHUNK - 1) // _EFLA_CHUNK
    ckpt = torch.empty(B * H * nchunks * d * d, dtype=torch.float32, device=k.device) if want_grad else None
    nmat = torch.empty((B, H, nchunks, 3, _EFLA_CHUNK, _EFLA_CHUNK), dtype=torch.bfloat16, device=k.device)
    coef = torch.empty((B, H, nchunks, 4, _EFLA_CHUNK), dtype=torch.float32, device=k.device)
    cut = _efla_segments(B, T, H, d, want_grad)
    if cut > 1:
        lib.call("elfa_efla_chunk_fwd_cut", kc, vc, beta, state, o, s_out, ckpt, nmat, coef, _efla_scratch(cut, kc, B, H, d), cut, B, T, H, d, stream_ptr(kc))
    else:
        lib.call("elfa_efla_chunk_fwd", kc, vc, beta, state, o, s_out, ckpt, nmat, coef, B, T, H, d, stream_ptr(kc))
    return (o, s_out, kc, vc, ckpt, nmat, coef) if want_grad else (o, s_out)


_PLAIN = (torch.Tensor, torch.nn.Parameter)


def _without_autograd(k, v, beta, state) -> bool:
    """The call may go to the kernel directly (22.9 -> 15.7 us for one token, of which the kernel takes 3): plain eager execution, and tensors as the
    kernels take them on one device. Everything else goes through the autograd function, which converts, refuses or records as it always did."""
    return (type(k) in _PLAIN and type(v) in _PLAIN and type(beta) in _PLAIN and (state is None or type(state) in _PLAIN) and plain_eager()
            and v.dtype == torch.bfloat16 and v.shape == k.shape and beta.dtype == torch.float32 and beta.numel() == 1
            and v.device == k.device == beta.device and (state is None or state.device == k.device))


class _EflaScan(torch.autograd.Function):
    """CUDA path. Forward: chunks of 32 tokens on the tensor cores with the fp32 state in registers. Backward: the gradient of
    the state walks the chunks the same way, everything else is parallel over the chunks, from the chunk-boundary states that forward
    keeps when a gradient is wanted."""

    @staticmethod
    def forward(ctx, k, v, beta, state, want_grad):
        o, s_out, *keep = _efla_forward(k, v, beta.detach().float().reshape(1).contiguous(), state, want_grad)
        if want_grad:
            B, T, H, d = k.shape
            ctx.save_for_backward(*keep)
            ctx.cfg = (B, T, H, d, state is not None)
        return o, s_out

    @staticmethod
    def backward(ctx, do, ds_out):
        kc, vc, ckpt, nmat, coef = ctx.saved_tensors
        B, T, H, d, has_state = ctx.cfg
        dk = torch.empty_like(kc)
        dv = torch.empty_like(vc)
        dbeta = torch.empty(1, dtype=torch.float32, device=kc.device)
        terms = torch.empty(B * H * ((T + 31) // 32), dtype=torch.float32, device=kc.device)          # of dbeta, one per chunk
        ds0 = torch.empty((B, H, d, d), dtype=torch.float32, device=kc.device) if has_state else None
        dckpt = torch.empty_like(ckpt)
        dso = ds_out.float().contiguous() if ds_out is not None else None
        cut = _efla_segments(B, T, H, d, True)
        lib.call("elfa_efla_chunk_bwd_sum", kc, vc, nmat, coef, ckpt, _aligned(do), dso, dk, dv, terms, dbeta, ds0, dckpt,
                 _efla_scratch(cut, kc, B, H, d) if cut > 1 else None, cut, B, T, H, d, stream_ptr(kc))
        return dk, dv, dbeta, ds0, None


def efla_scan(k: torch.Tensor, v: torch.Tensor, beta: torch.Tensor, state: Optional[torch.Tensor] = None, chunk: int = 16
              ) -> Tuple[torch.Tensor, torch.Tensor]:
    """EFLA recurrence. CPU tensors use the differentiable reference loop; CUDA bf16 tensors use the
    native kernels when the head dimension is supported (multiple of 32, at most 128). ``chunk`` (a positive number) was the
    distance of the states kept for backward and has no effect any more: with a gradient wanted the kernels keep ``T / 32`` states (and about
    6.5 KB per 32 tokens and head), and backward as many again while it runs. A caller that passed more than 64 to save memory holds more."""
    d = k.shape[-1]
    if k.is_cuda and k.dtype == torch.bfloat16 and d % 32 == 0 and d <= 128:
        if chunk <= 0:
            raise NativeError("efla_scan: chunk must be positive")
        if _without_autograd(k, v, beta, state):
            return _efla_forward(k, v, beta, state, False)
        want = torch.is_grad_enabled() and any(t is not None and t.requires_grad for t in (k, v, beta, state))
        o, s = _EflaScan.apply(k, v, beta.reshape(1), state, want)
        return o, s
    # CPU / unsupported shapes: the chunk-parallel form for long sequences (same values up to fp32 rounding, a fraction of
    # the Python-loop time), the token-by-token oracle otherwise
    o, s = efla_scan_chunked_ref(k, v, beta, state, 64) if k.shape[1] > 64 else efla_scan_ref(k, v, beta, state)
    return o.to(k.dtype), s


def compose_affine(a1: torch.Tensor, b1: torch.Tensor, a2: torch.Tensor, b2: torch.Tensor) -> Tuple[torch.Tensor, torch.Tensor]:
    """Composition of two state maps ``S -> A S + B`` (1 applied first, then 2)."""
    return a2 @ a1, a2 @ b1 + b2


def chunk_affine_map(k: torch.Tensor, v: torch.Tensor, beta: torch.Tensor) -> Tuple[torch.Tensor, torch.Tensor]:
    """The affine map ``(A, B)`` of a block of tokens: ``S_end = A S_start + B`` with
    ``A = prod_t (I - c_t k_t k_t^T)`` and ``B`` the final state from a zero start. k, v ``[B, T, H, d]``.
    Used to stitch chunks or sequence-parallel ranks together exactly. Both come out of the scan itself:
    ``B`` is its final state from a zero start, ``A`` its final state for zero values started from the identity
    (then ``S_end = A I + 0``), so a block of any length costs two scans instead of a Python loop over its tokens."""
    B_, T, H, d = k.shape
    eye = torch.eye(d, dtype=torch.float32, device=k.device).expand(B_, H, d, d).contiguous()
    _, Bm = efla_scan(k, v, beta)
    _, A = efla_scan(k, torch.zeros_like(v), beta, eye)
    return A, Bm


# --------------------------------------------------------------------------------------- ShortConv
def shortconv_ref(x: torch.Tensor, weight: torch.Tensor, bias: Optional[torch.Tensor] = None) -> torch.Tensor:
    """x ``[B, T, C]``, weight ``[C, W]`` → causal depthwise convolution, fp32 math."""
    B, T, C = x.shape
    W = weight.shape[1]
    xf = torch.nn.functional.pad(x.float(), (0, 0, W - 1, 0))          # left pad time
    y = torch.zeros(B, T, C, dtype=torch.float32, device=x.device)
    for w in range(W):
        y = y + xf[:, W - 1 - w:W - 1 - w + T] * weight.float()[:, w]
    if bias is not None:
        y = y + bias.float()
    return y.to(x.dtype)


class _ShortConv(torch.autograd.Function):
    @staticmethod
    def forward(ctx, x, weight, bias):
        B, T, C = x.shape
        xc = x.contiguous()
        y = torch.empty_like(xc)
        lib.call("elfa_shortconv_fwd", xc, weight, bias, y, B, T, C, weight.shape[1], stream_ptr(xc))
        ctx.save_for_backward(xc, weight)
        ctx.has_bias = bias is not None
        return y

    @staticmethod
    def backward(ctx, dy):
        xc, weight = ctx.saved_tensors
        B, T, C = xc.shape
        W = weight.shape[1]
        dyc = dy.contiguous()
        dx = torch.empty_like(xc)
        slices = lib.raw("elfa_shortconv_bwd_slices")(B, T, C, W)
        kind = torch.bfloat16 if weight.dtype == torch.bfloat16 else torch.float32      # the last sum rounds
        dw = torch.empty((C, W), dtype=kind, device=xc.device)
        db = torch.empty(C, dtype=kind, device=xc.device) if ctx.has_bias else None
        part = torch.empty((slices, W + 1, C), dtype=torch.float32, device=xc.device)
        lib.call("elfa_shortconv_bwd_as", xc, weight, dyc, dx, dw, db, part, int(kind == torch.bfloat16), B, T, C, W, stream_ptr(xc))
        return dx, dw.to(weight.dtype), (db.to(weight.dtype) if db is not None else None)


def shortconv(x: torch.Tensor, weight: torch.Tensor, bias: Optional[torch.Tensor] = None) -> torch.Tensor:
    if x.is_cuda and x.dtype == torch.bfloat16:
        return _ShortConv.apply(x, weight, bias)
    return shortconv_ref(x, weight, bias)


# ------------------------------------------------------------------------------------------- PRISM
class _PrismRefine(torch.autograd.Function):
    """CUDA path: one kernel forward, one backward (recomputes the residuals; the gradient of the
    gates is summed over the groups inside the thread that owns the channel: no atomics)."""

    @staticmethod
    def forward(ctx, u, v, group_dim, *ps):
        B, T, D = u.shape
        uc, vc = u.contiguous(), v.contiguous()
        pcs = [p.contiguous() for p in ps]
        y = torch.empty_like(uc)
        arr = (ctypes.c_uint64 * len(pcs))(*[p.data_ptr() for p in pcs])
        lib.call("elfa_prism_fwd", uc, vc, ctypes.addressof(arr), y, B * T, D // group_dim, group_dim, len(pcs), stream_ptr(uc))
        ctx.save_for_backward(uc, vc, *pcs)
        ctx.group_dim = group_dim
        return y

    @staticmethod
    def backward(ctx, dy):
        uc, vc, *pcs = ctx.saved_tensors
        B, T, D = uc.shape
        d = ctx.group_dim
        dyc = dy.contiguous()
        du, dv = torch.empty_like(uc), torch.empty_like(vc)
        dps = [torch.empty((B, T, d), dtype=torch.float32, device=uc.device) for _ in pcs]
        parr = (ctypes.c_uint64 * len(pcs))(*[p.data_ptr() for p in pcs])
        darr = (ctypes.c_uint64 * len(pcs))(*[p.data_ptr() for p in dps])
        lib.call("elfa_prism_bwd", uc, vc, ctypes.addressof(parr), dyc, du, dv, ctypes.addressof(darr), B * T, D // d, d, len(pcs),
                 stream_ptr(uc))
        return (du, dv, None) + tuple(g.to(p.dtype) for g, p in zip(dps, pcs))


def _prism_weight_grads(ws, wanted, u: torch.Tensor, dz: torch.Tensor, d: int):
    """``u^T dz`` as the gradients of the gates' weights, one per column block of ``d``: returned, or added to a weight's ``main_grad``
    (overwritten when that is fresh). ``D x L d`` is a handful of tiles, so the product is cut along the tokens and the
    pieces are added up in order: the same bits on every call, in the deterministic mode and outside it (B 8, T 2048, D 1024, d 64, L 2:
    17 + 3 us; unsplit, one product per weight, 71 us each)."""
    L, (rows, D) = len(ws), u.shape
    outs, triples = [None] * L, []
    for l, w in enumerate(ws):
        if not wanted[l]:
            triples += [0, 0, 2 ** 64 - 1]
            continue
        to = getattr(w, "main_grad", None)
        if to is None:
            to = outs[l] = torch.empty((D, d), dtype=w.dtype, device=u.device)
            add = False
        else:
            add = not getattr(w, "_grad_fresh", False)
            w._grad_fresh = False
        f32 = to.dtype == torch.float32
        assert to.shape == (D, d) and to.stride(1) == 1 and (f32 or to.dtype == torch.bfloat16)
        triples += [to.data_ptr(), to.stride(0), (2 if add else 1) if f32 else (3 if add else 0)]
    if any(wanted):
        n = lib.raw("elfa_gemm_bf16_parts_count")(D, L * d, rows)
        parts = torch.empty((n, (D + 127) // 128 * 128, L * d), dtype=torch.float32, device=u.device)
        lib.call("elfa_gemm_bf16_parts", u, dz, parts, D, L * d, rows, u.stride(0), dz.stride(0), stream_ptr(u))
        shared = len({id(w) for w in ws}) < L       # one buffer for several iterations: one after the other
        for l in range(L if shared else 1):
            some = [x if not shared or i // 3 == l else (2 ** 64 - 1 if i % 3 == 2 else x) for i, x in enumerate(triples)]
            arr = (ctypes.c_uint64 * (3 * L))(*some)
            lib.call("elfa_prism_weight_sum", parts, n, parts.stride(0), D, d, L, ctypes.addressof(arr), stream_ptr(u))
    return outs


class _PrismGated(torch.autograd.Function):
    """The whole gate of the layer: the ``L`` logit products as one GEMM over the concatenated weights, gates and refinement in one
    kernel; backward is one kernel, one input-gradient GEMM with an addition into ``du``, and one split product for all weight gradients."""

    @staticmethod
    def forward(ctx, u, v, group_dim, *ws):
        B, T, D = u.shape
        uc, vc = _aligned(u).view(-1, D), _aligned(v).view(-1, D)
        wc = torch.cat(ws, 1) if len(ws) > 1 else _aligned(ws[0])
        z = gemm(uc, wc, b_mn=True)
        y = torch.empty_like(uc)
        lib.call("elfa_prism_gated_fwd", uc, vc, z, z.stride(0), y, B * T, D // group_dim, group_dim, len(ws), stream_ptr(uc))
        ctx.save_for_backward(uc, vc, wc, z)
        ctx.w_refs, ctx.group_dim, ctx.shape = ws, group_dim, u.shape
        return y.view(u.shape)

    @staticmethod
    def backward(ctx, dy):
        uc, vc, wc, z = ctx.saved_tensors
        rows, D = uc.shape
        d, L = ctx.group_dim, len(ctx.w_refs)
        dyc = _aligned(dy)
        du, dv, dz = torch.empty_like(uc), torch.empty_like(vc), torch.empty_like(z)
        lib.call("elfa_prism_gated_bwd", uc, vc, z, z.stride(0), dyc, du, dv, dz, rows, D // d, d, L, stream_ptr(uc))
        if ctx.needs_input_grad[0]:
            # two launches: the GEMM's own addition (add_aux) reads a lane's row at a time and takes longer than both for a contraction this
            # short (16384 x 1024 x 128: 76 us)
            g = gemm(dz, wc)
            lib.call("elfa_elementwise", 2, du, g, du, du.numel(), 1.0, stream_ptr(du))
        dws = _prism_weight_grads(ctx.w_refs, ctx.needs_input_grad[3:], uc, dz, d)
        return (du.view(ctx.shape), dv.view(ctx.shape), None, *dws)


def prism_gated_native(u: torch.Tensor, v: torch.Tensor, ws, group_dim: int) -> bool:
    """What the fused gate handles: CUDA bf16 on one device, at most eight iterations, groups and rows of whole 16-byte vectors."""
    D, dev = u.shape[-1], u.device
    return (u.is_cuda and v.shape == u.shape and all(t.dtype == torch.bfloat16 and t.device == dev for t in (u, v, *ws))
            and 1 <= len(ws) <= 8 and u.numel() > 0 and group_dim % 8 == 0 and D % group_dim == 0
            and all(w.shape == (D, group_dim) for w in ws))


def prism_gated_refine(u: torch.Tensor, v: torch.Tensor, ws, group_dim: int) -> torch.Tensor:
    """``prism_refine`` with the gates given by their weights: ``p_l = sigmoid(u @ ws[l])``, formed in fp32."""
    if prism_gated_native(u, v, ws, group_dim):
        return _PrismGated.apply(u, v, group_dim, *ws)
    return prism_refine(u, v, [torch.sigmoid(linear(u, w).float()) for w in ws], group_dim)


def prism_refine(u: torch.Tensor, v: torch.Tensor, p_list, group_dim: int) -> torch.Tensor:
    """``u``, ``v`` ``[B, T, D]``; ``p_list[l]`` ``[B, T, d]`` (already sigmoid-ed). Returns ``u + refined``."""
    if u.is_cuda and u.dtype == torch.bfloat16 and 1 <= len(p_list) <= 8 and all(p.dtype == torch.bfloat16 for p in p_list):
        return _PrismRefine.apply(u, v, group_dim, *p_list)
    return prism_refine_ref(u, v, p_list, group_dim)


def prism_refine_ref(u: torch.Tensor, v: torch.Tensor, p_list, group_dim: int) -> torch.Tensor:
    """Plain PyTorch form (CPU path and test oracle)."""
    B, T, D = u.shape
    G = D // group_dim
    r = (v.float() - u.float()).view(B, T, G, group_dim)
    refined = torch.zeros_like(r)
    for p in p_list:
        delta = gelu_tanh_ref(p.float().unsqueeze(2) * r)
        r = r - delta
        refined = refined + delta
    return (u.float() + refined.view(B, T, D)).to(u.dtype)


@torch.no_grad()
def prism_stream(u: torch.Tensor, v: torch.Tensor, w_p, w_beta, w_k, state: torch.Tensor, forget: float, group_dim: int
                 ) -> Tuple[torch.Tensor, torch.Tensor]:
    """Refinement and state carry of a block of tokens without a gradient: ``(u + refined, new state)``. All ``3 L`` projections are one
    GEMM over the concatenated weights, the refinement and the state carry one kernel each. For what
    :func:`prism_stream_native` accepts; :func:`prism_state_update` is the same update token by token."""
    B, T, D = u.shape
    L, d = len(w_p), group_dim
    uc, vc = _aligned(u), _aligned(v)
    z = gemm(uc.view(-1, D), torch.cat((*w_p, *w_beta, *w_k), 1), b_mn=True)
    y = torch.empty_like(uc)
    lib.call("elfa_prism_gated_fwd", uc, vc, z, z.stride(0), y, B * T, D // d, d, L, stream_ptr(uc))
    st = state.contiguous()
    out = torch.empty_like(st)               # of the contiguous state: a strided one would hand its strides on
    lib.call("elfa_prism_state", uc, vc, z, z.stride(0), L * d, 2 * L * d, st, out, B, T, D // d, d, L, float(forget), stream_ptr(uc))
    return y, out


def prism_stream_native(u: torch.Tensor, v: torch.Tensor, w_p, w_beta, w_k, state: torch.Tensor, group_dim: int) -> bool:
    d, dev = group_dim, u.device
    return (prism_gated_native(u, v, w_p, d) and len(w_beta) == len(w_k) == len(w_p) and d in (32, 64, 96, 128)
            and all(w.dtype == torch.bfloat16 and w.shape == w_p[0].shape and w.device == dev for w in (*w_beta, *w_k))
            and state.device == dev and state.dtype == torch.float32 and state.shape == (u.shape[0], u.shape[-1] // d, d, d))


@torch.no_grad()
def prism_state_update(state: torch.Tensor, deltas, betas, ks, forget: float) -> torch.Tensor:
    """Carries the PRISM fast-weight state ``[B, G, d, d]`` over a block of tokens.
    ``deltas[l]`` ``[B, T, G, d]``, ``betas[l]`` ``[B, T]``, ``ks[l]`` ``[B, T, d]`` (unit norm).
    Iteration 0: ``S <- a S - a b (S k) k^T + b delta k^T``; later iterations: ``S <- S + b delta k^T``."""
    S = state.float().clone()
    T = deltas[0].shape[1]
    for t in range(T):
        for l, (dl, bl, kl) in enumerate(zip(deltas, betas, ks)):
            k = kl[:, t].float()                              # [B, d]
            b = bl[:, t].float()[:, None, None, None]
            d_t = dl[:, t].float()                            # [B, G, d]
            outer = d_t[..., :, None] * k[:, None, None, :]   # [B, G, d, d]
            if l == 0:
                Sk = torch.einsum("bgij,bj->bgi", S, k)
                S = forget * S - forget * b * Sk[..., :, None] * k[:, None, None, :] + b * outer
            else:
                S = S + b * outer
    return S
