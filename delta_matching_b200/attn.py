"""The API route: `attention(q, k, v, ...)` -> O (B, N, H, D).  Forward: the CUDA quantizers (codes and scales; no transposed
twins exist in this build), then the fwd_fp8 op.  Backward: the dO quantizer (with the stale delta rowsum(dO * O) only in the
stale mode; the matched mode never reads O), the matched delta from pass 0, then pass 1 and pass 2, split per head group at
long context (split.py), then the GQA fold.  Saved for the backward: the fp8 codes, their scales, the LSE and, in the stale
mode, O.  Mirrors delta_matching/attn.py:37-127 of the reference.

In eager mode the whole route is one call into the native module (csrc/dm_torch.cpp): a forward + backward of a small shape is
bound by the host, and the same steps in Python took four to five times as long as the kernels.  Under torch.compile the
route is the autograd function below over two custom ops."""
from __future__ import annotations

import torch

from . import _lib, ops
from .core import _check_inputs


class _DMAttn(torch.autograd.Function):
    """The traceable route (torch.compile)."""

    @staticmethod
    def forward(ctx, q, k, v, causal, delta_mode):
        B, H, N, D = q.shape
        Hk = k.shape[1]
        O, Lse, Q8, Q8s, K8, K8s, V8, V8s = ops.attn_fwd(q.transpose(1, 2), k.transpose(1, 2), v.transpose(1, 2), causal)
        ctx.save_for_backward(Q8, Q8s, K8, K8s, V8, V8s, O, Lse)
        ctx.dims = (B, H, Hk, N, D)
        ctx.causal = causal
        ctx.delta_mode = delta_mode
        return O

    @staticmethod
    @torch.autograd.function.once_differentiable
    def backward(ctx, dO):
        B, H, Hk, N, D = ctx.dims
        Q8, Q8s, K8, K8s, V8, V8s, O, Lse = ctx.saved_tensors
        if dO.stride(-1) != 1:          # e.g. the expanded gradient of o.sum(): the quantizer reads rows with a unit lane stride
            dO = dO.contiguous()
        dq, dk, dv = ops.attn_bwd(dO, O, Lse, Q8, Q8s, K8, K8s, V8, V8s, B, H, Hk, ctx.causal, ctx.delta_mode == "matched")
        return dq.permute(0, 2, 1, 3), dk.permute(0, 2, 1, 3), dv.permute(0, 2, 1, 3), None, None


def _head_major(name, t):
    if not (isinstance(t, torch.Tensor) and t.dim() == 4):
        raise ValueError(f"delta_matching: {name} has to be a 4-D tensor laid out (batch, seqlen, nheads, headdim)")
    return t.transpose(1, 2)


def attention(q, k, v, causal, softmax_scale, mode, head_major):
    """q, k, v as (B, H, N, D) when head_major, else (B, N, H, D).  The native call answers None when an input breaks a rule of the
    contract; _check_inputs then raises that rule's exception."""
    if not torch.compiler.is_compiling() and (mode == "matched" or mode == "stale"):
        o = _lib.native().attn(q, k, v, causal, softmax_scale, mode == "matched", head_major)
        if o is not None:
            return o
    if not head_major:
        q, k, v = _head_major("q", q), _head_major("k", k), _head_major("v", v)
    _check_inputs(q, k, v, causal, softmax_scale, mode)
    return _DMAttn.apply(q, k, v, causal, mode)


def dm_attn_func_bhnd(q, k, v, causal=True, softmax_scale=None, delta_mode="stale"):
    """Attention on (B, H, N, D) inputs: q (B, H, N, D), k / v (B, Hk, N, D) bf16 on CUDA (any strides; H % Hk == 0) ->
    O (B, N, H, D) bf16 contiguous (the kernel's native output layout).  delta_mode: "stale" (delta = rowsum(dO * O)) or
    "matched" (the Delta-Matching backward; needs causal=True).  Input errors raise ValueError / TypeError /
    NotImplementedError (core._check_inputs)."""
    return attention(q, k, v, causal, softmax_scale, delta_mode, True)


class _DMAttnPlain(torch.autograd.Function):
    """The plain route: the same kernels driven op by op without the head-group split, always taking the stale delta in
    the dO quantizer pass and replacing it by the pass-0 delta in the matched mode (the shape of the reference's
    core._DMAttnPlain, delta_matching/core.py:178-261).  Bitwise the API route; kept as a cross-check of it."""

    @staticmethod
    def forward(ctx, q, k, v, causal, delta_mode):
        B, H, N, D = q.shape
        Hk = k.shape[1]
        qf, kf, vf = q.transpose(1, 2), k.transpose(1, 2), v.transpose(1, 2)
        Q8, Q8s = _lib.quant(0, qf)
        K8, K8s = _lib.quant(1, kf, _lib.kmean(kf))
        V8, V8s = _lib.quant(2, vf)
        O, Lse = _lib.fwd_fp8(Q8, K8, V8, Q8s, K8s, V8s, B, H, Hk, causal)
        ctx.save_for_backward(Q8, Q8s, K8, K8s, V8, V8s, O, Lse)
        ctx.dims = (B, H, Hk, N, D)
        ctx.causal = causal
        ctx.delta_mode = delta_mode
        return O

    @staticmethod
    @torch.autograd.function.once_differentiable
    def backward(ctx, dO):
        B, H, Hk, N, D = ctx.dims
        Q8, Q8s, K8, K8s, V8, V8s, O, Lse = ctx.saved_tensors
        dO8, dO8s, Dlt = _lib.quant_do(dO.contiguous(), O)
        if ctx.delta_mode == "matched":
            Dlt = _lib.delta_fp8(Q8, K8, V8, dO8, Q8s, K8s, V8s, dO8s, Lse, B, H, Hk, ctx.causal)
        dk, dv, ws = _lib.bwd_pass1(Q8, K8, V8, dO8, Q8s, K8s, V8s, dO8s, Lse, Dlt, B, H, Hk, ctx.causal)
        dq = _lib.bwd_pass2(ws, K8, B, H, Hk, N, D, ctx.causal)
        dk, dv = _lib.gqa_fold(dk, Hk), _lib.gqa_fold(dv, Hk)
        return dq.permute(0, 2, 1, 3), dk.permute(0, 2, 1, 3), dv.permute(0, 2, 1, 3), None, None


def dm_attn_func_plain(q, k, v, causal=True, softmax_scale=None, delta_mode="stale"):
    """The plain route on (B, H, N, D) inputs; returns O (B, N, H, D) bf16 contiguous.  Same contract as
    dm_attn_func_bhnd."""
    _check_inputs(q, k, v, causal, softmax_scale, delta_mode)
    return _DMAttnPlain.apply(q, k, v, causal, delta_mode)
