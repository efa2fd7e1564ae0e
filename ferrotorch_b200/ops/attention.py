"""Attention front-end: causal GQA FlashAttention forward/backward on packed QKV.

The packed layout is the QKV GEMM's own output: ``qkv[T, (Hq + 2*Hkv) * D]`` with
the query heads first, then the key heads, then the value heads, so no
transpose / repeat_kv copies are made (the reference's GPU path materialises
``[H,S,S]`` scores and repeats KV heads: ferrotorch-llama/src/gpu.rs:609-628,
ferrotorch-gpu/src/bf16.rs:1987).

``attention_heads`` is the same attention on three tensors of any strides, read in place.

``flash_fwd`` / ``flash_bwd`` dispatch to the tcgen05 kernels when the native
library exports them for the shape (D = 128, bf16); otherwise they evaluate the
same math with torch's scaled_dot_product_attention, which the GPU tests also
use as the oracle. ``backend()`` reports which one runs.
"""
from __future__ import annotations

import ctypes
import math
import os

import torch

from .. import _lib
from ..errors import InvalidArgument

_native_ok: bool | None = None
_Strides4, _Strides8 = ctypes.c_int64 * 12, ctypes.c_int64 * 24            # element strides (batch, head, position) of four and of eight operands


def _native_available() -> bool:
    global _native_ok
    if _native_ok is None:
        ok = False
        if os.environ.get("FT_ATTN_BACKEND", "") != "sdpa":
            try:
                ok = hasattr(_lib.kernels(), "ft_flash_fwd_strided")
            except Exception:
                ok = False
        _native_ok = ok
    return _native_ok


def _bwd_native() -> bool:
    return os.environ.get("FT_ATTN_BWD", "") != "sdpa" and hasattr(_lib.kernels(), "ft_flash_bwd_strided")


def backend(D: int = 128, dtype=torch.bfloat16, device_is_cuda: bool = True) -> str:
    return "tcgen05" if (device_is_cuda and _native_available() and D == 128 and dtype == torch.bfloat16) else "sdpa"


def _split(qkv2, B, S, Hq, Hkv, D):
    q = qkv2[:, : Hq * D].reshape(B, S, Hq, D).transpose(1, 2)
    k = qkv2[:, Hq * D: (Hq + Hkv) * D].reshape(B, S, Hkv, D).transpose(1, 2)
    v = qkv2[:, (Hq + Hkv) * D:].reshape(B, S, Hkv, D).transpose(1, 2)
    return q, k, v


def _sdpa(q, k, v, causal, scale):
    if q.is_cuda:
        return torch.nn.functional.scaled_dot_product_attention(q, k, v, is_causal=causal, scale=scale, enable_gqa=True)
    rep = q.shape[1] // k.shape[1]
    k, v = k.repeat_interleave(rep, 1), v.repeat_interleave(rep, 1)
    s = torch.matmul(q.float(), k.float().transpose(-1, -2)) * scale
    if causal:
        Sq, Sk = s.shape[-2:]
        s = s.masked_fill(torch.ones(Sq, Sk, dtype=torch.bool, device=s.device).triu(Sk - Sq + 1), float("-inf"))
    return torch.matmul(torch.softmax(s, -1), v.float()).to(q.dtype)


def _packed(qkv2: torch.Tensor, S: int, Hq: int, Hkv: int, D: int):
    """Addresses of q, k and v in packed rows, each with its element strides (batch, head, position)."""
    ld, at, size = qkv2.stride(0), qkv2.data_ptr(), qkv2.element_size()
    st = (S * ld, D, ld)
    return (at, st), (at + Hq * D * size, st), (at + (Hq + Hkv) * D * size, st)


def _launch_fwd(qkv, out: int, lse: torch.Tensor, B, S, Hq, Hkv, D, out_strides, causal, scale) -> None:
    (q, sq), (k, sk), (v, sv) = qkv
    _lib.call("ft_flash_fwd_strided", q, k, v, out, lse, B, S, Hq, Hkv, D, _Strides4(*sq, *sk, *sv, *out_strides), int(causal), float(scale), _lib.S())


def _launch_bwd(qkv, out, lse: torch.Tensor, dout, dqkv, B, S, Hq, Hkv, D, causal, scale) -> None:
    (q, sq), (k, sk), (v, sv) = qkv
    (dq, sdq), (dk, sdk), (dv, sdv) = dqkv
    stat = torch.empty(B * Hq * -(-S // 64) * 128, device=lse.device, dtype=torch.float32)
    _lib.call("ft_flash_bwd_strided", q, k, v, out[0], lse, dout[0], dq, dk, dv, stat, B, S, Hq, Hkv, D,
              _Strides8(*sq, *sk, *sv, *out[1], *dout[1], *sdq, *sdk, *sdv), int(causal), float(scale), _lib.S())


def flash_fwd(qkv2: torch.Tensor, B: int, S: int, Hq: int, Hkv: int, D: int, causal: bool = True, scale: float | None = None):
    """Returns (out ``[T, Hq*D]``, lse ``[B, Hq, S]`` f32 or None for the sdpa path)."""
    scale = scale if scale is not None else 1.0 / math.sqrt(D)
    if backend(D, qkv2.dtype, qkv2.is_cuda) == "tcgen05":
        out = torch.empty((B * S, Hq * D), device=qkv2.device, dtype=qkv2.dtype)
        lse = torch.empty((B, Hq, S), device=qkv2.device, dtype=torch.float32)
        _launch_fwd(_packed(qkv2, S, Hq, Hkv, D), out.data_ptr(), lse, B, S, Hq, Hkv, D, (S * Hq * D, D, Hq * D), causal, scale)
        return out, lse
    q, k, v = _split(qkv2, B, S, Hq, Hkv, D)
    o = _sdpa(q, k, v, causal, scale)
    return o.transpose(1, 2).reshape(B * S, Hq * D).contiguous(), None


def flash_bwd(qkv2, out2, lse, dout2, B, S, Hq, Hkv, D, causal: bool = True, scale: float | None = None) -> torch.Tensor:
    """Returns dqkv ``[T, (Hq+2Hkv)*D]`` in the packed layout."""
    scale = scale if scale is not None else 1.0 / math.sqrt(D)
    if lse is not None and backend(D, qkv2.dtype, qkv2.is_cuda) == "tcgen05" and _bwd_native():
        dqkv = torch.empty_like(qkv2)
        if not dout2.is_contiguous():
            dout2 = dout2.contiguous()
        rows = (S * Hq * D, D, Hq * D)
        _launch_bwd(_packed(qkv2, S, Hq, Hkv, D), (out2.data_ptr(), rows), lse, (dout2.data_ptr(), rows), _packed(dqkv, S, Hq, Hkv, D), B, S, Hq, Hkv, D, causal, scale)
        return dqkv
    with torch.enable_grad():
        leaf = qkv2.detach().requires_grad_(True)
        q, k, v = _split(leaf, B, S, Hq, Hkv, D)
        o = _sdpa(q, k, v, causal, scale).transpose(1, 2).reshape(B * S, Hq * D)
        (dqkv,) = torch.autograd.grad(o, leaf, dout2)
    return dqkv


class _AttnFn(torch.autograd.Function):
    @staticmethod
    def forward(ctx, qkv2, B, S, Hq, Hkv, D, causal, scale):
        out, lse = flash_fwd(qkv2, B, S, Hq, Hkv, D, causal, scale)
        ctx.save_for_backward(qkv2, out, lse if lse is not None else torch.empty(0))
        ctx.meta = (B, S, Hq, Hkv, D, causal, scale, lse is not None)
        return out

    @staticmethod
    def backward(ctx, dout):
        qkv2, out, lse = ctx.saved_tensors
        B, S, Hq, Hkv, D, causal, scale, has = ctx.meta
        return flash_bwd(qkv2, out, lse if has else None, dout.contiguous(), B, S, Hq, Hkv, D, causal, scale), *([None] * 7)


def attention_packed(qkv2, B, S, Hq, Hkv, D, causal=True, scale=None):
    """Differentiable attention on the packed QKV buffer."""
    return _AttnFn.apply(qkv2, B, S, Hq, Hkv, D, causal, scale)


def _readable(t: torch.Tensor):
    """``t`` ``[B, H, S, D]`` (a copy where its layout is not one that tile loads take) and its strides for the kernels: contiguous heads, everything else on 16-byte
    boundaries. The stride of a dimension of size one means nothing and is replaced."""
    B, H, S, D = t.shape
    if t.stride(3) == 1 and t.data_ptr() % 16 == 0:
        st = tuple(D if n == 1 else s for n, s in ((B, t.stride(0)), (H, t.stride(1)), (S, t.stride(2))))
        if all(s > 0 and s % 8 == 0 for s in st):
            return t, st
    t = t.contiguous()
    if t.data_ptr() % 16:                                   # contiguous already, from an odd place in its storage
        t = t.clone()
    return t, (H * S * D, S * D, D)


class _HeadsFn(torch.autograd.Function):
    """Attention on ``[B, H, S, D]`` operands read where they lie. The output is ``[B, S, H, D]``, the order that the projection behind it reads, and so are the
    buffers of the gradients."""

    @staticmethod
    def forward(ctx, q, k, v, causal, scale):
        B, Hq, S, D = q.shape
        Hkv = k.shape[1]
        (q_, sq), (k_, sk), (v_, sv) = _readable(q), _readable(k), _readable(v)
        out = torch.empty((B, S, Hq, D), device=q.device, dtype=q.dtype)
        lse = torch.empty((B, Hq, S), device=q.device, dtype=torch.float32)
        with _lib.on_device_of(q):
            _launch_fwd(((q_.data_ptr(), sq), (k_.data_ptr(), sk), (v_.data_ptr(), sv)), out.data_ptr(), lse, B, S, Hq, Hkv, D, (S * Hq * D, D, Hq * D), causal, scale)
        ctx.save_for_backward(q, k, v, out, lse)
        ctx.causal, ctx.scale = causal, scale
        return out

    @staticmethod
    def backward(ctx, dout):
        q, k, v, out, lse = ctx.saved_tensors
        B, Hq, S, D = q.shape
        Hkv = k.shape[1]
        out, dout = out.transpose(1, 2), dout.transpose(1, 2)
        if not _bwd_native():
            with torch.enable_grad():
                leaves = [t.detach().requires_grad_(True) for t in (q, k, v)]
                return (*torch.autograd.grad(_sdpa(*leaves, ctx.causal, ctx.scale), leaves, dout), None, None)
        (q_, sq), (k_, sk), (v_, sv), (o_, so), (do_, sdo) = (_readable(t) for t in (q, k, v, out, dout))
        grads = [torch.empty((B, S, h, D), device=q.device, dtype=q.dtype) for h in (Hq, Hkv, Hkv)]
        rows = [(t.data_ptr(), (S * h * D, D, h * D)) for t, h in zip(grads, (Hq, Hkv, Hkv))]
        with _lib.on_device_of(q):
            _launch_bwd(((q_.data_ptr(), sq), (k_.data_ptr(), sk), (v_.data_ptr(), sv)), (o_.data_ptr(), so), lse, (do_.data_ptr(), sdo), rows, B, S, Hq, Hkv, D,
                        ctx.causal, ctx.scale)
        return (*(t.transpose(1, 2) for t in grads), None, None)


def attention_heads(q, k, v, causal: bool = False, scale: float | None = None):
    """Differentiable attention on bf16 CUDA operands ``[B, H, S, D]`` of any strides (``k``, ``v`` ``[B, Hkv, S, D]``), ``D`` a multiple of 8 up to 128."""
    if k.shape != v.shape or k.shape[0] != q.shape[0] or k.shape[2:] != q.shape[2:] or k.device != q.device or v.device != q.device:
        raise InvalidArgument(f"attention operands do not fit: q {tuple(q.shape)} {q.device}, k {tuple(k.shape)} {k.device}, v {tuple(v.shape)} {v.device}")
    return _HeadsFn.apply(q, k, v, causal, scale if scale is not None else 1.0 / math.sqrt(q.shape[3])).transpose(1, 2)
