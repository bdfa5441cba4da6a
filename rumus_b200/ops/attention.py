"""FlashAttention autograd wrapper over the tcgen05 forward / backward kernels."""
from __future__ import annotations

import ctypes
import math
from ctypes import c_float, c_int, c_longlong, c_void_p
from typing import Optional

import torch

from . import native
from ._lib import check, count_launch, ptr, stream_ptr

P, LL, I, F = c_void_p, c_longlong, c_int, c_float
native.register_signature("rb_flash_attn_fwd", [I, I, P, P, P, P, P, P, P, P, I, I, I, I, I, I, F, P])
native.register_signature("rb_flash_attn_bwd", [I, I, P, P, P, P, P, P, P, P, P, P, P, P, P, P, P,
                                                I, I, I, I, I, I, F, P])
native.register_signature("rb_fa_dq_cast", [I, P, P, P, I, I, I, P])
native.register_signature("rb_attn_f32_fwd", [I] + [P] * 8 + [I] * 5 + [F, P])
native.register_signature("rb_attn_f32_bwd", [I] + [P] * 16 + [I] * 5 + [F, P])


def _strides3(t: torch.Tensor):
    """{batch, seq, head} strides (elements) of a [B, S, H, D] view whose last dim is dense."""
    assert t.dim() == 4 and t.stride(3) == 1
    arr = (c_longlong * 3)(t.stride(0), t.stride(1), t.stride(2))
    return arr


def _tma_ok(t: torch.Tensor) -> bool:
    return (t.stride(3) == 1 and t.data_ptr() % 16 == 0
            and all((t.stride(i) * t.element_size()) % 16 == 0 for i in range(3)))


def f32_max_rows(Sq: int, Sk: int, D: int, causal: bool) -> int:
    """Queries and keys up to which the 32-bit kernels are ahead of the batched products they replace.  A row's keys are a serial chain,
    which the products' tiles are not, and a key read from shared memory serves 128 / (D / 16) rows, so long rows, wide heads and rows
    without a mask are where the products catch up.  Forward and backward, of the products' time, 1 to 64 x 8 batches and heads:
    causal 0.16 to 0.83 up to 1024 keys; not causal, heads of 32 0.16 to 0.80 up to 1024, of 64 0.2 to 1.0 up to 768 and 1.05 at 1024, of
    128 0.3 to 1.0 up to 192 and 1.05 to 1.27 from 256; other numbers of keys than of queries 0.3 to 0.95 up to 384 (192 for
    heads of 128), 1.1 to 1.2 for 16 or 64 queries of 512 keys and more."""
    if Sq == Sk and (causal or D <= 32):
        return 1024
    if D <= 64:
        return 768 if Sq == Sk else 384
    return 192


def f32_covers(q, k, v, causal: bool) -> bool:
    """Whether heads of these shapes are what the 32-bit kernels (``csrc/kernels/attn_f32.cu``) read and write: the batch, the
    heads and their size of k and v are q's (the kernels step through all three by q's sizes), a key for every row, and no more
    batches and heads than a grid's third and second dimension hold."""
    if len(q) != 4 or len(k) != 4 or k != v:
        return False
    (B, Sq, H, D), Sk = q, k[1]
    return (k == (B, Sk, H, D) and D in (16, 32, 64, 128) and 0 < Sk and 0 < Sq and (Sk >= Sq or not causal)
            and B <= 65535 and H <= 65535)


def f32_covered(q, k, v, causal: bool) -> bool:
    """Whether the 32-bit kernels take these tensors; all others stay with the batched products."""
    return (q.is_cuda and q.dtype == k.dtype == v.dtype == torch.float32 and q.device == k.device == v.device
            and f32_covers(tuple(q.shape), tuple(k.shape), tuple(v.shape), causal)
            and max(q.shape[1], k.shape[1]) <= f32_max_rows(q.shape[1], k.shape[1], q.shape[3], causal))


def attn_f32_forward(q, k, v, causal: bool, scale: float):
    if not f32_covers(tuple(q.shape), tuple(k.shape), tuple(v.shape), causal):
        raise ValueError(f"32-bit attention kernels do not take heads {tuple(q.shape)}, {tuple(k.shape)}, {tuple(v.shape)}")
    B, Sq, H, D = q.shape
    q, k, v = (t if _tma_ok(t) else t.contiguous() for t in (q, k, v))
    o = torch.empty((B, Sq, H, D), dtype=torch.float32, device=q.device)
    lse = torch.empty((B, H, Sq), dtype=torch.float32, device=q.device)
    st = [_strides3(t) for t in (q, k, v)]
    check(native.lib().rb_attn_f32_fwd(D, ptr(q), ptr(k), ptr(v), *map(ctypes.addressof, st), ptr(o), ptr(lse), B, H, Sq, k.shape[1],
                                       int(causal), float(scale), stream_ptr()), "rb_attn_f32_fwd")
    count_launch()
    return o, lse, (q, k, v)


def attn_f32_backward(q, k, v, o, lse, dout, causal: bool, scale: float, out):
    """``out``: dq, dk, dv of the shapes of q, k, v, rows of numbers side by side."""
    B, Sq, H, D = q.shape
    if not _tma_ok(dout):
        dout = dout.contiguous()
    dq, dk, dv = out
    st, dst = [_strides3(t) for t in (q, k, v, dout)], [_strides3(t) for t in out]
    check(native.lib().rb_attn_f32_bwd(D, ptr(q), ptr(k), ptr(v), ptr(o), ptr(dout), ptr(lse), *map(ctypes.addressof, st), ptr(dq), ptr(dk),
                                       ptr(dv), *map(ctypes.addressof, dst), B, H, Sq, k.shape[1], int(causal), float(scale),
                                       stream_ptr()), "rb_attn_f32_bwd")
    count_launch()


def fa_forward(q, k, v, causal: bool, scale: float, out=None):
    """``out``: contiguous ``[B, Sq, H, D]`` tensor to write the heads into."""
    B, Sq, H, D = q.shape
    Bk, Sk, Hkv, Dk = k.shape
    # the kernels describe k and v by q's batch, head size and type
    if (Bk != B or Dk != D or v.shape != k.shape or Hkv == 0 or H % Hkv or not q.dtype == k.dtype == v.dtype
            or not q.device == k.device == v.device):
        raise ValueError(f"attention of heads {tuple(q.shape)}, {tuple(k.shape)}, {tuple(v.shape)} ({q.dtype}, {k.dtype}, {v.dtype}; "
                         f"{q.device}, {k.device}, {v.device})")
    L = native.lib()
    q, k, v = (t if _tma_ok(t) else t.contiguous() for t in (q, k, v))
    o = out if out is not None else torch.empty((B, Sq, H, D), dtype=q.dtype, device=q.device)
    assert o.is_contiguous() and o.shape == q.shape and o.dtype == q.dtype
    lse = torch.empty((B, H, Sq), dtype=torch.float32, device=q.device)
    qs, ks, vs = _strides3(q), _strides3(k), _strides3(v)
    rc = L.rb_flash_attn_fwd(native.dtype_code(q.dtype), D, ptr(q), ptr(k), ptr(v),
                             ctypes.addressof(qs), ctypes.addressof(ks), ctypes.addressof(vs),
                             ptr(o), ptr(lse), B, H, Hkv, Sq, Sk, 1 if causal else 0, float(scale),
                             stream_ptr())
    check(rc, "rb_flash_attn_fwd")
    count_launch()
    return o, lse, (q, k, v)


def fa_backward(q, k, v, o, lse, dout, causal: bool, scale: float, out=None):
    """dq, dk, dv.  ``out`` may give three preallocated [B,S,heads,128] views (e.g. slices of one
    packed d_qkv buffer): the kernels write straight into them."""
    L = native.lib()
    B, Sq, H, D = q.shape
    _, Sk, Hkv, _ = k.shape
    if not _tma_ok(dout):
        dout = dout.contiguous()
    dq32 = torch.empty((B, Sq, H, D), dtype=torch.float32, device=q.device)   # zeroed by the delta kernel
    if out is None:
        dq = torch.empty((B, Sq, H, D), dtype=q.dtype, device=q.device)
        dk = torch.empty((B, Sk, Hkv, D), dtype=q.dtype, device=q.device)
        dv = torch.empty((B, Sk, Hkv, D), dtype=q.dtype, device=q.device)
    else:
        dq, dk, dv = out
    assert dk.stride() == dv.stride() and dk.stride(3) == 1 and dq.stride(3) == 1
    sq_pad = (Sq + 63) // 64 * 64
    # delta | lse * log2 e; only rows of padding have to be cleared, the kernel writes all others
    stats = (torch.empty if sq_pad == Sq else torch.zeros)((2, B, H, sq_pad), dtype=torch.float32, device=q.device)
    qs, ks, vs, dos = _strides3(q), _strides3(k), _strides3(v), _strides3(dout)
    dkvs, dqs = _strides3(dk), _strides3(dq)
    rc = L.rb_flash_attn_bwd(native.dtype_code(q.dtype), D, ptr(q), ptr(k), ptr(v), ptr(o),
                             ptr(dout), ptr(lse), ctypes.addressof(qs), ctypes.addressof(ks),
                             ctypes.addressof(vs), ctypes.addressof(dos), ptr(stats), ptr(dq32),
                             ptr(dk), ptr(dv), ctypes.addressof(dkvs), B, H, Hkv, Sq, Sk,
                             1 if causal else 0, float(scale), stream_ptr())
    check(rc, "rb_flash_attn_bwd")
    rc = L.rb_fa_dq_cast(native.dtype_code(q.dtype), ptr(dq32), ptr(dq), ctypes.addressof(dqs),
                         B, Sq, H, stream_ptr())
    check(rc, "rb_fa_dq_cast")
    count_launch(3)
    return dq, dk, dv


class _FlashAttnFn(torch.autograd.Function):
    @staticmethod
    def forward(ctx, q, k, v, causal, scale):
        o, lse, (qc, kc, vc) = fa_forward(q, k, v, causal, scale)
        ctx.causal, ctx.scale = causal, scale
        ctx.save_for_backward(qc, kc, vc, o, lse)
        return o

    @staticmethod
    def backward(ctx, dout):
        q, k, v, o, lse = ctx.saved_tensors
        if q.shape[-1] == 128:
            dq, dk, dv = fa_backward(q, k, v, o, lse, dout, ctx.causal, ctx.scale)
        else:
            dq, dk, dv = _composed_backward(q, k, v, dout, ctx.causal, ctx.scale)
        return dq, dk, dv, None, None


class _AttnF32Fn(torch.autograd.Function):
    @staticmethod
    def forward(ctx, q, k, v, causal, scale):
        o, lse, (qc, kc, vc) = attn_f32_forward(q, k, v, causal, scale)
        ctx.causal, ctx.scale = causal, scale
        ctx.save_for_backward(qc, kc, vc, o, lse)
        return o

    @staticmethod
    def backward(ctx, dout):
        q, k, v, o, lse = ctx.saved_tensors
        out = [torch.empty(t.shape, dtype=t.dtype, device=t.device) for t in (q, k, v)]
        attn_f32_backward(q, k, v, o, lse, dout, ctx.causal, ctx.scale, out)
        return (*out, None, None)


def attention_f32(q, k, v, causal: bool = True, scale: Optional[float] = None):
    """32-bit attention by one kernel forward and one backward; for what ``f32_covered`` takes."""
    return _AttnF32Fn.apply(q, k, v, causal, scale if scale is not None else 1.0 / math.sqrt(q.shape[-1]))


class _FlashAttnPackedFn(torch.autograd.Function):
    """Attention on the packed projection output ``qkv [B, S, (H + 2*Hkv) * hd]``: the backward
    kernels write d_q, d_k, d_v into the three slices of one d_qkv buffer (no concatenation)."""

    @staticmethod
    def _heads(qkv, heads, kv_heads):
        B, S, n = qkv.shape
        hd = n // (heads + 2 * kv_heads)
        q, k, v = qkv.split([heads * hd, kv_heads * hd, kv_heads * hd], dim=-1)
        return q.view(B, S, heads, hd), k.view(B, S, kv_heads, hd), v.view(B, S, kv_heads, hd)

    @staticmethod
    def forward(ctx, qkv, heads, kv_heads, causal, scale):
        q, k, v = _FlashAttnPackedFn._heads(qkv, heads, kv_heads)
        o, lse, _ = (attn_f32_forward if qkv.dtype == torch.float32 else fa_forward)(q, k, v, causal, scale)
        ctx.causal, ctx.scale, ctx.heads, ctx.kv_heads = causal, scale, heads, kv_heads
        ctx.save_for_backward(qkv, o, lse)
        return o

    @staticmethod
    def backward(ctx, dout):
        qkv, o, lse = ctx.saved_tensors
        dqkv = torch.empty_like(qkv)
        q, k, v = _FlashAttnPackedFn._heads(qkv, ctx.heads, ctx.kv_heads)
        out = _FlashAttnPackedFn._heads(dqkv, ctx.heads, ctx.kv_heads)
        (attn_f32_backward if qkv.dtype == torch.float32 else fa_backward)(q, k, v, o, lse, dout, ctx.causal, ctx.scale, out=out)
        return dqkv, None, None, None, None


def flash_attention_packed(qkv, heads: int, kv_heads: int, causal: bool = True,
                           scale: Optional[float] = None):
    """``qkv`` is the fused projection output on a GPU, 16-byte aligned rows: 16-bit with head_dim 128, or 32-bit with heads that
    ``f32_covered`` takes."""
    hd = qkv.shape[-1] // (heads + 2 * kv_heads)
    if qkv.dtype != torch.float32 and hd != 128:      # the backward kernel's only head size
        raise ValueError(f"packed 16-bit attention has heads of 128, not {hd}")
    if qkv.dtype == torch.float32 and (qkv.data_ptr() % 16 or not qkv.is_contiguous()):
        qkv = qkv.clone(memory_format=torch.contiguous_format)      # the kernels move 16 bytes at a time, the gradient's rows too
    if scale is None:
        scale = 1.0 / math.sqrt(hd)
    return _FlashAttnPackedFn.apply(qkv, heads, kv_heads, causal, scale)


def _composed_backward(q, k, v, dout, causal, scale):
    """head_dim != 128: gradient through the batched-matmul + softmax kernels in fp32."""
    from . import functional as F
    with torch.enable_grad():
        qf, kf, vf = (t.detach().float().requires_grad_(True) for t in (q, k, v))
        if kf.shape[2] != qf.shape[2]:
            rep = qf.shape[2] // kf.shape[2]
            ke, ve = kf.repeat_interleave(rep, dim=2), vf.repeat_interleave(rep, dim=2)
        else:
            ke, ve = kf, vf
        o = F._sdpa_composed(qf, ke, ve, causal, scale)
        gq, gk, gv = torch.autograd.grad(o, (qf, kf, vf), dout.float())
    return gq.to(q.dtype), gk.to(k.dtype), gv.to(v.dtype)


def flash_attention_cuda(q, k, v, causal: bool = True, scale: Optional[float] = None):
    """q: [B, Sq, H, D], k/v: [B, Sk, Hkv, D] (bf16/fp16, D in {64, 128}); returns [B, Sq, H, D]."""
    D = q.shape[-1]
    if D not in (64, 128):
        from . import functional as F
        return F._sdpa_composed(q.float(), k.float(), v.float(), causal, scale).to(q.dtype)
    scale = scale if scale is not None else 1.0 / math.sqrt(D)
    return _FlashAttnFn.apply(q, k, v, causal, scale)
