"""Autograd binding of the tcgen05 flash-attention kernels (``csrc/flash_attn.cu``)."""
from __future__ import annotations

import contextlib
import ctypes
import math
from typing import Optional

import torch

from . import lib

_f = {}
_FORCE_ONE_TILE = False  # tests flip this to exercise the one-tile forward kernel on every shape


def _fwd():
    if "f" not in _f:
        c = lib
        _f["f"] = lib.fn("lvb_flash_attn_fwd", [c.c_void_p] * 7 + [c.c_int] * 4 + [c.c_float, c.c_float, c.c_int, c.c_void_p, c.c_void_p])
    return _f["f"]


def _fwd_hd():
    """Head size 64 or 128, causal or not (one query tile per CTA)."""
    if "fh" not in _f:
        c = lib
        _f["fh"] = lib.fn("lvb_flash_attn_fwd_hd", [c.c_void_p] * 8 + [c.c_int] * 7 + [c.c_float, c.c_float, c.c_int, c.c_void_p, c.c_void_p])
    return _f["fh"]


def _fwd2_hd():
    """Head size 64 or 128, causal or not, sequences of any length: two query tiles per CTA."""
    if "f2h" not in _f:
        c = lib
        _f["f2h"] = lib.fn("lvb_flash_attn_fwd2_hd", [c.c_void_p] * 10 + [c.c_int] * 7 + [c.c_float, c.c_float, c.c_int, c.c_void_p, c.c_void_p])
    return _f["f2h"]


def _bwd_hd():
    if "bh" not in _f:
        c = lib
        _f["bh"] = lib.fn("lvb_flash_attn_bwd_hd", [c.c_void_p] * 14 + [c.c_int] * 7 + [c.c_float, c.c_float, c.c_int, c.c_void_p, c.c_void_p],
                          launches=2)
    return _f["bh"]


def _bwd2():
    """Causal, head size 128."""
    if "b2" not in _f:
        c = lib
        _f["b2"] = lib.fn("lvb_flash_attn_bwd2", [c.c_void_p] * 14 + [c.c_int] * 4 + [c.c_float, c.c_float, c.c_int, c.c_void_p, c.c_void_p],
                          launches=2)
    return _f["b2"]


def _segment_ranges(q_seg, k_seg):
    """(lowest, highest) segment id per 128 rows of each sequence of ``q_seg [B, S]`` and then of ``k_seg [B, Sk]``, by which the kernels leave blocks out."""
    if q_seg is None:
        return None
    if "r" not in _f:
        c = lib
        _f["r"] = lib.fn("lvb_segment_ranges", [c.c_void_p] * 2 + [c.c_int] * 3 + [c.c_void_p] * 2)
    (B, S), Sk = q_seg.shape, k_seg.shape[1]
    out = torch.empty(B * (-(-S // 128) - (-Sk // 128)), 2, dtype=torch.int32, device=q_seg.device)
    lib.check_rc(_f["r"](q_seg.data_ptr(), k_seg.data_ptr(), B, S, Sk, out.data_ptr(), lib.stream_ptr()), "lvb_segment_ranges")
    return out


# The backward pass runs on the software-pipelined kernel (``csrc/flash_attn_bwd2.cu``); ``LEVANTER_B200_FLASH_BWD=serial`` selects
# the one-buffer kernel (``csrc/flash_attn_bwd.cu``).
import os as _os

BWD_PIPELINED = _os.environ.get("LEVANTER_B200_FLASH_BWD", "pipelined") != "serial"


# Activation checkpointing that keeps attention outputs (utils/remat.py:checkpoint_layer): during the first pass of a
# checkpointed layer the forward below appends (o, lse) to ``_keep``; during the recomputation it takes them back from
# ``_replay`` in the same order and launches nothing.
_keep: Optional[list] = None
_replay: Optional[list] = None


@contextlib.contextmanager
def keeping_outputs(store: list):
    global _keep
    prev, _keep = _keep, store
    try:
        yield store
    finally:
        _keep = prev


@contextlib.contextmanager
def replaying_outputs(store: list):
    global _replay
    prev, _replay = _replay, list(store)
    try:
        yield
    finally:
        _replay = prev


def _rows(t: torch.Tensor) -> torch.Tensor:
    """``t [B, S, H, D]`` as the kernels' tensor maps can describe it: rows that hold their heads side by side, at 16-byte aligned strides."""
    B, S, H, D = t.shape
    ok = (t.stride(3) == 1 and (H == 1 or t.stride(2) == D) and (S == 1 or (t.stride(1) >= H * D and t.stride(1) % 8 == 0))
          and (B == 1 or (t.stride(0) >= H * D and t.stride(0) % 8 == 0)) and t.data_ptr() % 16 == 0)
    return t if ok else t.clone(memory_format=torch.contiguous_format)


def _strides(*ts):
    """(sequence, row) strides in elements; those of a size of one are not meant to be read, but have to be valid."""
    out = []
    for t in ts:
        B, S, H, D = t.shape
        row = t.stride(1) if S > 1 else H * D
        out += [t.stride(0) if B > 1 else S * row, row]
    return (ctypes.c_longlong * len(out))(*out)


def _attend(q, k, v, q_seg, k_seg, scale, soft_cap, window, causal, sink):
    """``(o, lse, ranges)`` of rows as :func:`_rows` has them."""
    B, S, Hq, D = q.shape
    Sk, Hkv = k.shape[1], k.shape[2]  # Sk differs from S only for cross attention (no causal part)
    ranges = _segment_ranges(q_seg, k_seg)
    if _replay:
        o, lse2 = _replay.pop(0)
        if o.shape != q.shape:
            raise RuntimeError("the recomputation of a checkpointed layer called attention in a different order than its first pass")
        return o, lse2, ranges
    o = torch.empty(B, S, Hq, D, dtype=q.dtype, device=q.device)
    lse2 = torch.empty(B, Hq, S, dtype=torch.float32, device=q.device)
    tail = (float(scale), float(soft_cap or 0.0), int(window or 0), lib.status_buffer().data_ptr(), lib.stream_ptr())
    if not _FORCE_ONE_TILE:
        rc = _fwd2_hd()(q.data_ptr(), k.data_ptr(), v.data_ptr(), _strides(q, k, v), o.data_ptr(), lse2.data_ptr(), lib.ptr(q_seg), lib.ptr(k_seg),
                        lib.ptr(ranges), lib.ptr(sink), B, S, Sk, Hq, Hkv, D, int(bool(causal)), *tail)
    else:
        q, k, v = q.contiguous(), k.contiguous(), v.contiguous()
        if D != 128 or not causal or sink is not None:
            rc = _fwd_hd()(q.data_ptr(), k.data_ptr(), v.data_ptr(), o.data_ptr(), lse2.data_ptr(), lib.ptr(q_seg), lib.ptr(k_seg), lib.ptr(sink), B, S, Sk,
                           Hq, Hkv, D, int(bool(causal)), *tail)
        else:
            rc = _fwd()(q.data_ptr(), k.data_ptr(), v.data_ptr(), o.data_ptr(), lse2.data_ptr(), lib.ptr(q_seg), lib.ptr(k_seg), B, S, Hq, Hkv, *tail)
    lib.check_rc(rc, "lvb_flash_attn_fwd")
    if _keep is not None:
        _keep.append((o, lse2))
    return o, lse2, ranges


def _attend_backward(do, q, k, v, o, lse2, q_seg, k_seg, ranges, dk, dv, scale, soft_cap, window, causal):
    """Writes ``dk`` and ``dv`` (rows with the same strides) and returns ``(dq in fp32, delta)``."""
    B, S, Hq, D = q.shape
    Sk, Hkv = k.shape[1], k.shape[2]
    do = do.contiguous()
    if do.dtype != torch.bfloat16:
        do = do.to(torch.bfloat16)
    dq32 = torch.zeros(B, S, Hq, D, dtype=torch.float32, device=q.device)
    delta = torch.empty(B, Hq, S, dtype=torch.float32, device=q.device)
    args = (q.data_ptr(), k.data_ptr(), v.data_ptr(), _strides(q, k, v, dk), o.data_ptr(), do.data_ptr(), lse2.data_ptr(), delta.data_ptr(), dq32.data_ptr(),
            dk.data_ptr(), dv.data_ptr(), lib.ptr(q_seg), lib.ptr(k_seg), lib.ptr(ranges))
    tail = (float(scale), float(soft_cap or 0.0), int(window or 0), lib.status_buffer().data_ptr(), lib.stream_ptr())
    if D == 128 and causal and BWD_PIPELINED:
        rc = _bwd2()(*args, B, S, Hq, Hkv, *tail)
    else:  # the kernels templated on the head size; the pipelined one is causal, 128 only
        rc = _bwd_hd()(*args, B, S, Sk, Hq, Hkv, D, int(bool(causal)), *tail)
    lib.check_rc(rc, "lvb_flash_attn_bwd")
    return dq32, delta


class _FlashFn(torch.autograd.Function):
    @staticmethod
    def forward(ctx, q, k, v, q_seg, k_seg, scale, soft_cap, window, causal=True, sink=None):
        if sink is not None:
            sink = sink.detach().float().contiguous()
        q, k, v = _rows(q), _rows(k), _rows(v)
        o, lse2, ranges = _attend(q, k, v, q_seg, k_seg, scale, soft_cap, window, causal, sink)
        ctx.save_for_backward(q, k, v, o, lse2, q_seg, k_seg, sink, ranges)
        ctx.args = (scale, soft_cap, window, causal)
        return o

    @staticmethod
    def backward(ctx, do):
        q, k, v, o, lse2, q_seg, k_seg, sink, ranges = ctx.saved_tensors
        dk, dv = (torch.empty(t.shape, dtype=t.dtype, device=t.device) for t in (k, v))
        dq32, delta = _attend_backward(do, q, k, v, o, lse2, q_seg, k_seg, ranges, dk, dv, *ctx.args)
        dsink = None
        if sink is not None and ctx.needs_input_grad[9]:
            # the sink column's probability is 2^(sink log2 e - lse2); its value row is zero, so its logit's gradient is
            # -p_sink * delta summed over batch and queries (delta = rowsum(dO * O), left in the scratch by the kernel)
            dsink = -(torch.exp2(sink.view(1, -1, 1) * 1.4426950408889634 - lse2) * delta).sum(dim=(0, 2))
        return dq32.to(torch.bfloat16), dk, dv, None, None, None, None, None, None, dsink


class _FlashJoint(torch.autograd.Function):
    """Attention of ``qkv [B, S, 3, H, D]``, the rows of a joint projection: nothing is copied apart, and the gradient is written as those rows."""

    @staticmethod
    def forward(ctx, qkv, q_seg, k_seg, scale, soft_cap, window, causal):
        if not (qkv.stride(4) == 1 and qkv.stride(3) == qkv.shape[4] and qkv.stride(2) == qkv.shape[3] * qkv.shape[4]):
            qkv = qkv.contiguous()
        q, k, v = (_rows(t) for t in qkv.unbind(2))
        o, lse2, ranges = _attend(q, k, v, q_seg, k_seg, scale, soft_cap, window, causal, None)
        ctx.save_for_backward(q, k, v, o, lse2, q_seg, k_seg, ranges)
        ctx.args = (scale, soft_cap, window, causal)
        return o

    @staticmethod
    def backward(ctx, do):
        q, k, v, o, lse2, q_seg, k_seg, ranges = ctx.saved_tensors
        B, S, H, D = q.shape
        d = torch.empty(B, S, 3, H, D, dtype=q.dtype, device=q.device)
        dq32, _ = _attend_backward(do, q, k, v, o, lse2, q_seg, k_seg, ranges, d[:, :, 1], d[:, :, 2], *ctx.args)
        d[:, :, 0].copy_(dq32)
        return d, None, None, None, None, None, None


def _mask_parts(mask, B: int, S: int, Sk: int, device):
    """``(q_seg, k_seg, window, causal)`` of a structured mask."""
    if mask is None:
        return None, None, 0, False
    if mask.chunk_size is not None:
        if mask.segment_ids is None:
            mask = mask.with_segment_ids(torch.zeros(B, S, dtype=torch.int32, device=device))
        mask = mask.chunks_as_segments()  # a chunk is a segment of its own
    q_seg = k_seg = None
    if mask.segment_ids is not None:
        q_seg, k_seg = mask.segment_ids
        q_seg = q_seg.to(torch.int32).expand(B, S).contiguous()
        k_seg = k_seg.to(torch.int32).expand(B, Sk).contiguous()
    causal = bool(mask.is_causal)
    if causal and Sk != S:
        raise ValueError("a causal mask needs as many keys as queries")
    return q_seg, k_seg, mask.sliding_window or 0, causal


PAD_SEGMENT = -2  # segment id of the rows that the one-tile kernel's sequences are padded with: they see only one another


def flash_attention_cuda(q, k, v, mask, *, logits_soft_cap: Optional[float] = None, scaling_factor: Optional[float] = None,
                         sink: Optional[torch.Tensor] = None):
    """``q[B,S,Hq,D]``, ``k/v[B,S,Hkv,D]`` bf16, D = 64 or 128; ``mask`` is ``None`` (every key visible) or an ``AttentionMask``
    made of causal / sliding-window / segment-id parts.  Any sequence length, and rows with strides of their own (slices of a wider
    projection).  ``sink [Hq]``: a learned logit per head that joins the softmax denominator (a key column whose value row is zero)."""
    scale = scaling_factor if scaling_factor is not None else 1.0 / math.sqrt(q.shape[-1])
    B, S, Sk = q.shape[0], q.shape[1], k.shape[1]
    q_seg, k_seg, window, causal = _mask_parts(mask, B, S, Sk, q.device)
    pad = pad_k = 0
    if _FORCE_ONE_TILE:  # whole tiles only
        pad = (-S) % 128
        pad_k = pad if Sk == S else (-Sk) % 128
        if pad or pad_k:
            if q_seg is None:
                q_seg = torch.zeros(B, S, dtype=torch.int32, device=q.device)
                k_seg = torch.zeros(B, Sk, dtype=torch.int32, device=q.device)
            q_seg = torch.nn.functional.pad(q_seg, (0, pad), value=PAD_SEGMENT)
            k_seg = torch.nn.functional.pad(k_seg, (0, pad_k), value=PAD_SEGMENT)
            q = torch.nn.functional.pad(q, (0, 0, 0, 0, 0, pad))
            k, v = (torch.nn.functional.pad(t, (0, 0, 0, 0, 0, pad_k)) for t in (k, v))
    o = _FlashFn.apply(q, k, v, q_seg, k_seg, scale, logits_soft_cap, window, causal, sink)
    return o[:, :S] if pad else o


def flash_attention_joint_cuda(qkv, mask, *, scaling_factor: float):
    """:func:`flash_attention_cuda` of the rows ``qkv [B, S, 3, H, D]`` of a joint projection."""
    B, S = qkv.shape[:2]
    q_seg, k_seg, window, causal = _mask_parts(mask, B, S, S, qkv.device)
    return _FlashJoint.apply(qkv, q_seg, k_seg, scaling_factor, None, window, causal)
