"""The carried-state loop of the chunked gated delta rule (``csrc/delta_rule.cu``).

Given, for every chunk ``n`` of 64 tokens, the tiles that can be computed for all chunks at once

* ``w [.., N, C, dk]`` and ``u [.., N, C, dv]`` (the WY factors of the chunk),
* ``qg [.., N, C, dk]`` (queries times their decay from the chunk start), ``kd [.., N, C, dk]`` (keys times their decay to
  the chunk end), ``P [.., N, C, C]`` (decayed, causally masked query-key scores) and ``a [.., N]`` (decay over the chunk),

:func:`chunk_state_scan` runs ::

    v_new = u_n - w_n S;   o_n = qg_n S + P_n v_new;   S = a_n S + kd_n^T v_new

over the chunks and returns ``(o [.., N, C, dv], final S [.., dk, dv])``.  :func:`gated_delta_rule` makes those tiles too
(``csrc/delta_chunks.cu``): the whole rule from rows of q, k, v and the gates, and its gradients.  On a B200 both directions are one kernel launch
(the state never leaves shared memory); elsewhere the same loop runs on PyTorch ops, which is also the test oracle.  The
reference framework has no counterpart (the model family is an addition)."""
from __future__ import annotations

import ctypes
from typing import Optional, Tuple

import torch

from . import lib

CHUNK = 64


def _supported(w: torch.Tensor, u: torch.Tensor) -> bool:
    return (w.is_cuda and lib.available() and w.shape[-2] == CHUNK and w.shape[-1] in (64, 128)
            and u.shape[-1] % 64 == 0 and w.dtype == torch.float32)


def chunk_state_scan_reference(w, qg, kd, P, u, a, S0: Optional[torch.Tensor] = None) -> Tuple[torch.Tensor, torch.Tensor]:
    """The loop on PyTorch ops (differentiable by autograd)."""
    N = w.shape[-3]
    dk, dv = w.shape[-1], u.shape[-1]
    S = w.new_zeros(*w.shape[:-3], dk, dv) if S0 is None else S0.to(w.dtype)
    outs = []
    for n in range(N):
        v_new = u[..., n, :, :] - w[..., n, :, :] @ S
        outs.append(qg[..., n, :, :] @ S + P[..., n, :, :] @ v_new)
        S = S * a[..., n, None, None] + kd[..., n, :, :].transpose(-1, -2) @ v_new
    return torch.stack(outs, dim=-3), S


_fwd = _bwd = _slices = None


def _bind():
    global _fwd, _bwd, _slices
    if _fwd is None:
        P = lib.c_void_p
        _fwd = lib.fn("lvb_delta_rule_fwd", [P] * 10 + [lib.c_int] * 5 + [P])
        _bwd = lib.fn("lvb_delta_rule_bwd", [P] * 16 + [lib.c_int] * 5 + [P])
        _slices = lib.fn("lvb_delta_rule_bwd_slices", [lib.c_int], launches=0)


class _ChunkStateScan(torch.autograd.Function):
    @staticmethod
    def forward(ctx, w, qg, kd, P, u, a, S0, exact):
        _bind()
        lead = w.shape[:-3]
        N, C, dk = w.shape[-3:]
        dv = u.shape[-1]
        BH = 1
        for s in lead:
            BH *= s
        w, qg, kd, P, u, a = (t.contiguous() for t in (w, qg, kd, P, u, a))
        S0c = None if S0 is None else S0.float().contiguous()
        need_grad = any(ctx.needs_input_grad)
        out = torch.empty(*lead, N, C, dv, dtype=torch.float32, device=w.device)
        S_final = torch.empty(*lead, dk, dv, dtype=torch.float32, device=w.device)
        S_hist = torch.empty(*lead, N, dk, dv, dtype=torch.float32, device=w.device) if need_grad else None
        rc = _fwd(lib.ptr(w), lib.ptr(qg), lib.ptr(kd), lib.ptr(P), lib.ptr(u), lib.ptr(a), lib.ptr(S0c), lib.ptr(out),
                  lib.ptr(S_hist), lib.ptr(S_final), BH, N, dk, dv, int(exact), lib.stream_ptr())
        lib.check_rc(rc, "delta_rule_fwd")
        if need_grad:
            ctx.save_for_backward(w, qg, kd, P, u, a, S_hist)
        ctx.dims = (lead, BH, N, C, dk, dv, bool(exact), S0 is not None)
        return out, S_final

    @staticmethod
    def backward(ctx, dout, dS_final):
        w, qg, kd, P, u, a, S_hist = ctx.saved_tensors
        lead, BH, N, C, dk, dv, exact, has_s0 = ctx.dims
        dev = w.device
        ns = _slices(dv)
        dout = torch.zeros_like(u) if dout is None else dout.float().contiguous()
        dSf = None if dS_final is None else dS_final.float().contiguous()
        dw, dqg, dkd = (torch.empty(ns, *lead, N, C, dk, dtype=torch.float32, device=dev) for _ in range(3))
        dP = torch.empty(ns, *lead, N, C, C, dtype=torch.float32, device=dev)
        da = torch.empty(ns, *lead, N, dtype=torch.float32, device=dev)
        du = torch.empty_like(u)
        dS0 = torch.empty(*lead, dk, dv, dtype=torch.float32, device=dev) if has_s0 else None
        rc = _bwd(lib.ptr(w), lib.ptr(qg), lib.ptr(kd), lib.ptr(P), lib.ptr(u), lib.ptr(a), lib.ptr(S_hist), lib.ptr(dout),
                  lib.ptr(dSf), lib.ptr(dw), lib.ptr(dqg), lib.ptr(dkd), lib.ptr(dP), lib.ptr(da), lib.ptr(du), lib.ptr(dS0),
                  BH, N, dk, dv, int(exact), lib.stream_ptr())
        lib.check_rc(rc, "delta_rule_bwd")
        # the per-slice partial sums are added in slice order, so the gradients do not depend on scheduling
        return dw.sum(0), dqg.sum(0), dkd.sum(0), dP.sum(0), du, da.sum(0), dS0, None


def chunk_state_scan(w, qg, kd, P, u, a, S0: Optional[torch.Tensor] = None, *, exact: bool = False):
    """See the module docstring.  ``exact`` makes the kernel use fp32 FMAs instead of TF32 tensor-core products."""
    if not _supported(w, u):  # CPU, or a shape the kernel does not cover (chunk != 64, d_k not 64/128, d_v % 64 != 0)
        return chunk_state_scan_reference(w, qg, kd, P, u, a, S0)
    return _ChunkStateScan.apply(w, qg, kd, P, u, a, S0, exact)


def _view4(t: torch.Tensor) -> torch.Tensor:
    """``t [B, L, H, d]`` as the kernels can read it: rows of unit stride, read four numbers at a time."""
    ok = t.stride(3) == 1 and all(s % 4 == 0 for s in t.stride()[:3]) and t.data_ptr() % (4 * t.element_size()) == 0
    return t if ok else t.clone(memory_format=torch.contiguous_format)


def gated_delta_rule_supported(q, k, v, chunk_size: int = CHUNK) -> bool:
    """Whether :func:`gated_delta_rule` takes ``q, k [.., dk]`` and ``v [.., dv]``."""
    return (q.is_cuda and lib.available() and chunk_size == CHUNK and q.numel() > 0 and q.shape[-1] in (64, 128) and v.shape[-1] % 64 == 0
            and v.shape[-1] > 0 and q.dtype == k.dtype == v.dtype and q.dtype in (torch.float32, torch.bfloat16) and q.shape[:-1] == v.shape[:-1]
            and q.shape == k.shape and q.device == k.device == v.device)


_chunks = {}


def _chunk_kernels():
    if not _chunks:
        P, i, f = lib.c_void_p, lib.c_int, lib.c_float
        _chunks["fwd"] = lib.fn("lvb_delta_chunks_fwd", [P] * 13 + [i] * 7 + [f, P])
        _chunks["bwd"] = lib.fn("lvb_delta_chunks_bwd", [P] * 17 + [i] + [P] * 5 + [i] * 7 + [f, P])
        _chunks["norm"] = lib.fn("lvb_delta_out_norm_fwd", [P] * 4 + [i] * 4 + [f, i, P])
        _chunks["norm_bwd"] = lib.fn("lvb_delta_out_norm_bwd", [P] * 7 + [i] * 5 + [f, i, P])
    return _chunks


def _strides(q, k, v, g, beta):
    return (ctypes.c_longlong * 15)(*(s for t in (q, k, v, g, beta) for s in t.stride()[:3]))


class _GatedDeltaRule(torch.autograd.Function):
    """The tiles of all chunks (``csrc/delta_chunks.cu``), then the loop over them; backward the loop, then the tiles."""

    @staticmethod
    def forward(ctx, q, k, v, g, beta, S0, scale, normalize, exact):
        _bind()
        B, L, H, dk = q.shape
        dv, N = v.shape[3], -(-L // CHUNK)
        q, k, v = _view4(q), _view4(k), _view4(v)
        need_grad = any(ctx.needs_input_grad)
        new = lambda *shape: torch.empty(*shape, dtype=torch.float32, device=q.device)  # noqa: E731
        w, qg, kd = (new(B, H, N, CHUNK, dk) for _ in range(3))
        P, u, a = new(B, H, N, CHUNK, CHUNK), new(B, H, N, CHUNK, dv), new(B, H, N)
        T = new(B, H, N, CHUNK, CHUNK) if need_grad else None
        bf16 = int(q.dtype == torch.bfloat16)
        rc = _chunk_kernels()["fwd"](q.data_ptr(), k.data_ptr(), v.data_ptr(), g.data_ptr(), beta.data_ptr(), _strides(q, k, v, g, beta), w.data_ptr(),
                                     qg.data_ptr(), kd.data_ptr(), P.data_ptr(), u.data_ptr(), a.data_ptr(), lib.ptr(T), B, L, H, dk, dv, bf16,
                                     int(normalize), float(scale), lib.stream_ptr())
        lib.check_rc(rc, "delta_chunks_fwd")
        S0c = None if S0 is None else S0.float().contiguous()
        out, S_final = new(B, H, N, CHUNK, dv), new(B, H, dk, dv)
        S_hist = new(B, H, N, dk, dv) if need_grad else None
        rc = _fwd(w.data_ptr(), qg.data_ptr(), kd.data_ptr(), P.data_ptr(), u.data_ptr(), a.data_ptr(), lib.ptr(S0c), out.data_ptr(), lib.ptr(S_hist),
                  S_final.data_ptr(), B * H, N, dk, dv, int(exact), lib.stream_ptr())
        lib.check_rc(rc, "delta_rule_fwd")
        if need_grad:
            ctx.save_for_backward(q, k, v, g, beta, w, qg, kd, P, u, a, T, S_hist)
        ctx.args = (bf16, int(normalize), float(scale), S0 is not None, int(exact))
        return out, S_final

    @staticmethod
    def backward(ctx, dout, dS_final):
        q, k, v, g, beta, w, qg, kd, P, u, a, T, S_hist = ctx.saved_tensors
        bf16, normalize, scale, has_s0, exact = ctx.args
        (B, L, H, dk), (N, dv) = q.shape, (w.shape[2], v.shape[3])
        ns = _slices(dv)
        new = lambda *shape: torch.empty(*shape, dtype=torch.float32, device=q.device)  # noqa: E731
        dout = torch.zeros_like(u) if dout is None else dout.float().contiguous()
        dSf = None if dS_final is None else dS_final.float().contiguous()
        dw, dqg, dkd = (new(ns, B, H, N, CHUNK, dk) for _ in range(3))
        dP, da, du = new(ns, B, H, N, CHUNK, CHUNK), new(ns, B, H, N), torch.empty_like(u)
        dS0 = new(B, H, dk, dv) if has_s0 else None
        rc = _bwd(w.data_ptr(), qg.data_ptr(), kd.data_ptr(), P.data_ptr(), u.data_ptr(), a.data_ptr(), S_hist.data_ptr(), dout.data_ptr(), lib.ptr(dSf),
                  dw.data_ptr(), dqg.data_ptr(), dkd.data_ptr(), dP.data_ptr(), da.data_ptr(), du.data_ptr(), lib.ptr(dS0), B * H, N, dk, dv, exact,
                  lib.stream_ptr())
        lib.check_rc(rc, "delta_rule_bwd")
        dq, dk_, dv_ = (torch.empty(B, L, H, d, dtype=q.dtype, device=q.device) for d in (dk, dk, dv))
        dg, dbeta = new(B, L, H), new(B, L, H)
        rc = _chunk_kernels()["bwd"](q.data_ptr(), k.data_ptr(), v.data_ptr(), g.data_ptr(), beta.data_ptr(), _strides(q, k, v, g, beta), w.data_ptr(),
                                     P.data_ptr(), u.data_ptr(), a.data_ptr(), T.data_ptr(), dw.data_ptr(), dqg.data_ptr(), dkd.data_ptr(), dP.data_ptr(),
                                     da.data_ptr(), du.data_ptr(), ns, dq.data_ptr(), dk_.data_ptr(), dv_.data_ptr(), dg.data_ptr(), dbeta.data_ptr(),
                                     B, L, H, dk, dv, bf16, normalize, scale, lib.stream_ptr())
        lib.check_rc(rc, "delta_chunks_bwd")
        return dq, dk_, dv_, dg, dbeta, dS0, None, None, None


def gated_delta_rule(q, k, v, g, beta, S0: Optional[torch.Tensor] = None, *, scale: float, normalize: bool = False,
                     exact: bool = False) -> Tuple[torch.Tensor, torch.Tensor]:
    """The gated delta rule over ``q, k [B, L, H, dk]``, ``v [B, L, H, dv]`` (bf16 or fp32), ``g`` (log decay) and ``beta [B, L, H]`` fp32 ->
    ``(out [B, H, ceil(L / 64), 64, dv], final state [B, H, dk, dv])`` in fp32; rows past ``L`` of the last chunk are no results.  Queries are
    multiplied by ``scale``; with ``normalize`` queries and keys are divided by their 2-norms first.  ``exact`` as in :func:`chunk_state_scan`.  For what
    :func:`gated_delta_rule_supported` takes.  Gates or a state of another size, or on another device, raise."""
    B, L, H, dk = q.shape
    for t in (g, beta, S0):
        if t is not None and t.device != q.device:
            raise RuntimeError(f"the gates and the state have to be where the queries are ({q.device}), not on {t.device}")
    for t in (g, beta):  # the kernels read what the queries' shape says
        if t.shape != (B, L, H):
            raise RuntimeError(f"gates of shape {tuple(t.shape)} for {B} sequences of {L} positions and {H} heads")
    S0 = None if S0 is None else S0.reshape(B, H, dk, v.shape[3])
    return _GatedDeltaRule.apply(q, k, v, g.float(), beta.float(), S0, scale, normalize, exact)


class _OutNorm(torch.autograd.Function):
    @staticmethod
    def forward(ctx, o, gate, weight, eps):
        B, L, H, dv = gate.shape
        o, gate, w = o.contiguous(), gate.contiguous(), weight.float().contiguous()
        y = torch.empty_like(gate)
        bf16 = int(gate.dtype == torch.bfloat16)
        rc = _chunk_kernels()["norm"](o.data_ptr(), gate.data_ptr(), w.data_ptr(), y.data_ptr(), B, L, H, dv, float(eps), bf16, lib.stream_ptr())
        lib.check_rc(rc, "delta_out_norm_fwd")
        ctx.save_for_backward(o, gate, weight)
        ctx.args = (float(eps), bf16)
        return y

    @staticmethod
    def backward(ctx, dy):
        o, gate, weight = ctx.saved_tensors
        eps, bf16 = ctx.args
        B, L, H, dv = gate.shape
        dy, w = dy.to(gate.dtype).contiguous(), weight.float().contiguous()
        d_o, dgate = torch.empty_like(o), torch.empty_like(gate)
        blocks = min(592, -(-B * L * H // 8))  # four per SM
        part = torch.empty(blocks, dv, dtype=torch.float32, device=o.device)
        rc = _chunk_kernels()["norm_bwd"](o.data_ptr(), gate.data_ptr(), w.data_ptr(), dy.data_ptr(), d_o.data_ptr(), dgate.data_ptr(), part.data_ptr(),
                                          blocks, B, L, H, dv, eps, bf16, lib.stream_ptr())
        lib.check_rc(rc, "delta_out_norm_bwd")
        return d_o, dgate, part.sum(0).to(weight.dtype) if ctx.needs_input_grad[2] else None, None


def gated_out_norm(o, gate, weight, eps: float) -> torch.Tensor:
    """``o * rsqrt(mean(o^2) + eps) * weight * silu(gate)`` of the ``out`` of :func:`gated_delta_rule`, as ``gate [B, L, H, dv]`` is laid out."""
    return _OutNorm.apply(o, gate, weight, eps)
