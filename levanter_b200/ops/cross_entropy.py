"""LM-head GEMM + cross-entropy without ever holding ``[tokens, vocab]``.

Forward: the CTA-pair GEMM (``csrc/gemm_pair.cu``) consumes its accumulators in the epilogue: every lane owns a row and keeps the
running maximum and sum of exponentials of its column tile, so that a logit is never stored; ``lvb_ce_combine`` joins the column tiles
to the log-sum-exp and the loss.  Backward: the same product again, whose epilogue writes the logits' gradient in bf16 for a chunk of
tokens, and two more products with it, dX (K = vocabulary, split over CTA pairs) and dW.

A vocabulary that is no multiple of 8 (GPT-2's 50257) used to take library products in fp32.  There the gradient is held as two bf16 parts side by
side in the row, the rounded number and what the rounding lost: 16 bits of mantissa; up to ``THREE_PARTS`` tokens as three, 24 bits.  Both products run
over all parts in one accumulation, the lowest first.  What is left is the tensor cores' accumulator, which cuts off what it cannot hold: against 64
bits dW in an fp32 buffer is off by 4e-7 for 300 tokens, 1.3e-6 for 999 and 4.9e-6 for 8192 (two parts with the rounded numbers first: 1.4e-6,
3.1e-6, 1.2e-5; fp32 library products 3e-7 to 6e-7), where a bf16 gradient is off by 1.65e-3 either way.  The loss is off by 0.7 to 1.1e-7, an fp32
unit in the last place, for the library's 4 to 5e-8.  A training step of four GPT-2 layers over 8192 tokens (768 wide) went from 43.1 to
9.9 ms with it; the products of the head took 30.7 ms of that in fp32, the passes over logits 8 more.

While a copy-job provider is set (fully sharded training: plain GEMMs carry the next layer's weight gather) and for vocabularies up to 128 the
logits pass through memory in fp32 chunks instead (``lvb_ce_stats``, ``lvb_ce_grad``).

Same mathematics as the reference's vocab-blockwise loss (src/levanter/models/loss.py:251-507: online logsumexp forward, recompute in
backward, ``dlogits = (g_loss + g_logz) * p - g_loss * onehot``), tiled over tokens instead of vocab because the
GEMM wants long K-major rows of the head matrix.
"""
from __future__ import annotations

from typing import Optional

import torch

from . import gemm as _gemm
from . import lib
from .gemm import gemm

_f = {}
_buffers: dict = {}


def _stats():
    if "s" not in _f:
        c = lib
        _f["s"] = lib.fn("lvb_ce_stats", [c.c_void_p, c.c_longlong, c.c_void_p, c.c_void_p, c.c_void_p, c.c_int, c.c_int, c.c_float, c.c_void_p, c.c_void_p])
    return _f["s"]


def _grad():
    if "g" not in _f:
        c = lib
        _f["g"] = lib.fn("lvb_ce_grad", [c.c_void_p, c.c_longlong] + [c.c_void_p] * 5 + [c.c_longlong, c.c_int, c.c_int, c.c_float, c.c_void_p])
    return _f["g"]


def _buffer(key, shape, dtype, device):
    k = (key, torch.cuda.current_device())
    b = _buffers.get(k)
    n = 1
    for s in shape:
        n *= s
    if b is None or b.numel() < n or b.dtype != dtype:
        b = torch.empty(n, dtype=dtype, device=device)
        _buffers[k] = b
    return b[:n].view(*shape)


def chunk_rows_for(vocab: int, budget_bytes: int = 1 << 30) -> int:
    rows = budget_bytes // (vocab * 4)
    rows = max(256, (rows // 256) * 256)
    return min(rows, 16384)


def _head(name):
    if name not in _f:
        c = lib
        P, i, f, ll = c.c_void_p, c.c_int, c.c_float, c.c_longlong
        _f[name] = lib.fn(name, {
            "lvb_head_ce_stats": [P] * 5 + [i] * 5 + [f, P, P],
            "lvb_ce_combine": [P, i] + [P] * 4 + [i, i, f, P, P],
            "lvb_head_ce_grad": [P] * 7 + [ll] + [i] * 7 + [f, P, P],
            "lvb_head_ce_product": [P] * 3 + [i] * 3 + [ll] + [i] * 7 + [P] * 3}[name])
    return _f[name]


GRAD_BYTES = 3 << 29  # of the logits' gradient at once
# Tokens up to which a gradient in parts has a third one.  dW sums over the tokens, and from about a thousand on the accumulator hides what the third part
# adds (300 tokens: 1.02e-6 without it, 4.2e-7 with it; 999: 1.254e-6, 1.253e-6), while it makes both products half as long again (8192 tokens: 1 ms).
THREE_PARTS = 1024


def _grad_chunk(T: int, row_bytes: int) -> int:
    """Tokens per chunk of the backward pass: equal chunks of whole 256-row tiles, none above ``GRAD_BYTES``."""
    most = max(256, GRAD_BYTES // row_bytes // 256 * 256)
    n = -(-T // most)
    return -(-(-(-T // n)) // 256) * 256


def _dx_splits(tiles: int, k_blocks: int, pairs: int, out_bytes: int) -> int:
    """CTA pairs per 256 x 256 tile of dX.  K is the whole vocabulary there and a narrow model has few tiles (4096 x 768: 48 on 74 pairs), so a
    product takes its waves times K per split, 0.44 us for a block of 64 (of K) and a tile at the tensor cores' rate; every split also writes its sums in
    fp32 (``out_bytes`` each) and they are read again, at 5 TB/s and 3 us more.  At least 16 K blocks each, and sums of at most ``GRAD_BYTES`` in all."""
    def cost(s):
        return -(-tiles * s // pairs) * -(-k_blocks // s) * 0.44 + (3.0 + 2 * s * out_bytes / 5e6 if s > 1 else 0.0)

    most = max(1, min(8, k_blocks // 16, GRAD_BYTES // max(1, out_bytes)))
    return min(range(1, most + 1), key=lambda s: (cost(s), s))


def _plain_gradients(x, weight, targets, cap, z, dloss, wanted):
    """Differentiable ``(dx, dw)`` on framework ops."""
    logits = x.float() @ weight.float().t()
    if cap > 0.0:
        logits = torch.tanh(logits / cap) * cap
    lse = torch.logsumexp(logits, dim=-1)
    V = weight.shape[0]
    at = logits.gather(1, targets.long().clamp(0, V - 1)[:, None])[:, 0]
    loss = lse - torch.where((targets >= 0) & (targets < V), at, torch.zeros_like(at)) + z * lse * lse
    asked = [t for t, w in zip((x, weight), wanted) if w]
    got = iter(torch.autograd.grad(loss, asked, dloss.float(), create_graph=True))
    return tuple(next(got) if w else None for w in wanted[:2])


def _tma_rows(t: torch.Tensor) -> torch.Tensor:
    """``t [rows, cols]`` as the tensor maps can describe it: rows of unit stride that do not overlap, at 16-byte aligned strides."""
    ok = t.stride(1) == 1 and t.stride(0) >= t.shape[1] and t.stride(0) % 8 == 0 and t.data_ptr() % 16 == 0
    return t if ok else t.clone(memory_format=torch.contiguous_format)


class _HeadCE(torch.autograd.Function):
    """See the module docstring.  ``parts``: of the gradient, 1 to 3."""

    @staticmethod
    def forward(ctx, x, weight, targets, soft_cap, z_weight, chunk_rows, parts):
        T, E = x.shape
        V = weight.shape[0]
        given = (x, weight)
        ctx.weight_ref = weight
        x, weight = _tma_rows(x), _tma_rows(weight)
        tg = targets.to(torch.int32).contiguous()
        tiles = -(-V // 256)
        part = torch.empty(tiles, T, 2, dtype=torch.float32, device=x.device)
        tl, lse, loss = (torch.empty(T, dtype=torch.float32, device=x.device) for _ in range(3))
        cap, z = float(soft_cap or 0.0), float(z_weight or 0.0)
        st, stream = lib.status_buffer().data_ptr(), lib.stream_ptr()
        lib.check_rc(_head("lvb_head_ce_stats")(x.data_ptr(), weight.data_ptr(), tg.data_ptr(), part.data_ptr(), tl.data_ptr(), T, V, E, x.stride(0),
                                                weight.stride(0), cap, st, stream), "lvb_head_ce_stats")
        lib.check_rc(_head("lvb_ce_combine")(part.data_ptr(), tiles, tg.data_ptr(), tl.data_ptr(), lse.data_ptr(), loss.data_ptr(), T, V, z, st, stream),
                     "lvb_ce_combine")
        ctx.save_for_backward(*given, tg, lse)
        ctx.args = (cap, z, chunk_rows, parts)
        ctx.mark_non_differentiable(lse)
        return loss, lse

    @staticmethod
    def backward(ctx, dloss, _dlse):
        x, weight, tg, lse = ctx.saved_tensors
        cap, z, chunk_rows, parts = ctx.args
        if parts > 1 and torch.is_grad_enabled():  # create_graph: these vocabularies have had second derivatives, from library products
            return _plain_gradients(x, weight, tg, cap, z, dloss, ctx.needs_input_grad) + (None,) * 5
        T, E = x.shape
        V = weight.shape[0]
        x, weight = _tma_rows(x), _tma_rows(weight)
        g_loss = dloss.float().contiguous()
        g_logz = (g_loss * (2.0 * z) * lse).contiguous() if z != 0.0 else None
        cols = -(-V // 64) * 64
        ldd = parts * cols
        chunk = chunk_rows or _grad_chunk(T, 2 * ldd)
        d = torch.empty(min(chunk, T), ldd, dtype=torch.bfloat16, device=x.device)
        dx = torch.empty(T, E, dtype=x.dtype, device=x.device) if ctx.needs_input_grad[0] else None
        dw = acc = None
        flags = 0
        if ctx.needs_input_grad[1]:
            main_grad = getattr(ctx.weight_ref, "main_grad", None)
            if main_grad is not None:
                if main_grad.shape != (V, E) or main_grad.stride(1) != 1 or main_grad.dtype not in (torch.float32, torch.bfloat16):
                    raise ValueError("main_grad has to be a row-major fp32 or bf16 buffer of the weight's shape")
                acc, flags = main_grad, _gemm.F_ACCUMULATE | (_gemm.F_OUT_F32 if main_grad.dtype == torch.float32 else 0)
            else:  # fp32 sums over several chunks, rounded once; the products of a single chunk are rounded as they are made
                dw = acc = torch.empty(V, E, dtype=weight.dtype if chunk >= T else torch.float32, device=x.device)
                flags = 0 if chunk >= T else _gemm.F_OUT_F32
        st, stream = lib.status_buffer().data_ptr(), lib.stream_ptr()
        pairs = torch.cuda.get_device_properties(x.device).multi_processor_count // 2
        for r0 in range(0, T, chunk):
            n = min(chunk, T - r0)
            xs, out = x[r0:r0 + n], None if dx is None else dx[r0:r0 + n]
            lib.check_rc(_head("lvb_head_ce_grad")(xs.data_ptr(), weight.data_ptr(), tg[r0:].data_ptr(), lse[r0:].data_ptr(), g_loss[r0:].data_ptr(),
                                                   0 if g_logz is None else g_logz[r0:].data_ptr(), d.data_ptr(), ldd, cols, parts, n, V, E, x.stride(0),
                                                   weight.stride(0), cap, st, stream), "lvb_head_ce_grad")
            if out is not None:
                splits = _dx_splits(-(-n // 256) * -(-E // 256), parts * cols // 64, pairs, 4 * n * E)
                ws = torch.empty(splits * n * E, dtype=torch.float32, device=x.device) if splits > 1 else None
                lib.check_rc(_head("lvb_head_ce_product")(d.data_ptr(), weight.data_ptr(), out.data_ptr(), n, V, E, ldd, cols, parts, weight.stride(0), E, 0, 0,
                                                          splits, lib.ptr(ws), st, stream), "lvb_head_ce_product")
            if acc is not None:
                lib.check_rc(_head("lvb_head_ce_product")(d.data_ptr(), xs.data_ptr(), acc.data_ptr(), n, V, E, ldd, cols, parts, x.stride(0), acc.stride(0), 1,
                                                          flags, 1, 0, st, stream), "lvb_head_ce_product")
                flags |= _gemm.F_ACCUMULATE
        if dw is not None:
            dw = dw.to(weight.dtype)
        return dx, dw, None, None, None, None, None


class _FusedLinearCE(torch.autograd.Function):
    @staticmethod
    def forward(ctx, x, weight, targets, soft_cap, z_weight, chunk_rows):
        T, E = x.shape
        V = weight.shape[0]
        x = x.contiguous()
        tg = targets.to(torch.int32).contiguous()
        lse = torch.empty(T, dtype=torch.float32, device=x.device)
        tl = torch.empty(T, dtype=torch.float32, device=x.device)
        chunk = chunk_rows or chunk_rows_for(V)
        Vp = (V + 3) // 4 * 4
        logits = _buffer("logits", (min(chunk, T), Vp), torch.float32, x.device)
        cap = float(soft_cap) if soft_cap is not None else 0.0
        st = lib.status_buffer().data_ptr()
        for r0 in range(0, T, chunk):
            n = min(chunk, T - r0)
            lg = logits[:n, :V] if Vp != V else logits[:n]
            gemm(x[r0:r0 + n], weight, out=lg)
            rc = _stats()(lg.data_ptr(), lg.stride(0), tg[r0:].data_ptr(), lse[r0:].data_ptr(), tl[r0:].data_ptr(), n, V, cap,
                          st, lib.stream_ptr())
            lib.check_rc(rc, "lvb_ce_stats")
        ctx.save_for_backward(x, weight, tg, lse)
        ctx.cap, ctx.z, ctx.chunk = cap, float(z_weight or 0.0), chunk
        ctx.weight_ref = weight
        loss = lse - tl
        if ctx.z != 0.0:
            loss = loss + ctx.z * lse * lse
        ctx.mark_non_differentiable(lse)
        return loss, lse

    @staticmethod
    def backward(ctx, dloss, _dlse):
        x, weight, tg, lse = ctx.saved_tensors
        T, E = x.shape
        V = weight.shape[0]
        chunk = ctx.chunk
        Vp = (V + 3) // 4 * 4
        Vd = (V + 7) // 8 * 8
        logits = _buffer("logits", (min(chunk, T), Vp), torch.float32, x.device)
        dlog = _buffer("dlogits", (min(chunk, T), Vd), torch.bfloat16, x.device)
        g_loss = dloss.float().contiguous()
        g_logz = (g_loss * (2.0 * ctx.z) * lse).contiguous() if ctx.z != 0.0 else None
        dx = torch.empty_like(x) if ctx.needs_input_grad[0] else None
        need_dw = ctx.needs_input_grad[1]
        main_grad = getattr(ctx.weight_ref, "main_grad", None) if need_dw else None
        dw = None
        if need_dw and main_grad is None:
            dw = torch.zeros(V, E, dtype=torch.float32, device=x.device)
        acc = main_grad if main_grad is not None else dw
        for r0 in range(0, T, chunk):
            n = min(chunk, T - r0)
            lg = logits[:n, :V] if Vp != V else logits[:n]
            gemm(x[r0:r0 + n], weight, out=lg)
            dl = dlog[:n, :V] if Vd != V else dlog[:n]
            rc = _grad()(lg.data_ptr(), lg.stride(0), tg[r0:].data_ptr(), lse[r0:].data_ptr(), g_loss[r0:].data_ptr(),
                         g_logz[r0:].data_ptr() if g_logz is not None else 0, dl.data_ptr(), dl.stride(0), n, V, ctx.cap,
                         lib.stream_ptr())
            lib.check_rc(rc, "lvb_ce_grad")
            if dx is not None:
                gemm(dl, weight, b_mn=True, out=dx[r0:r0 + n])
            if need_dw:
                gemm(dl, x[r0:r0 + n], a_mn=True, b_mn=True, out=acc, accumulate=True)
        if dw is not None:
            dw = dw.to(weight.dtype)
        return dx, dw, None, None, None, None


def fused_linear_cross_entropy(x: torch.Tensor, weight: torch.Tensor, targets: torch.Tensor, *, soft_cap: Optional[float] = None,
                               z_weight: Optional[float] = None, chunk_rows: Optional[int] = None):
    """Per-token ``(loss, logsumexp)`` of ``softmax(x @ weight.T)`` against ``targets``; ``x[T,E]`` bf16, ``weight[V,E]`` bf16."""
    V = weight.shape[0]
    if V > 128 and x.shape[0] > 0 and _gemm._copy_job_provider is None:
        return _HeadCE.apply(x, weight, targets, soft_cap, z_weight, chunk_rows, 1 if V % 8 == 0 else 3 if x.shape[0] <= THREE_PARTS else 2)
    return _FusedLinearCE.apply(x, weight, targets, soft_cap, z_weight, chunk_rows)


def _only_first_derivatives() -> bool:
    """No function transform (vmap, jvp, ...) and no forward-mode level is active: the kernels define first derivatives only."""
    return not torch._C._are_functorch_transforms_active() and torch.autograd.forward_ad._current_level < 0


def kernel_ok(x: torch.Tensor, weight: torch.Tensor) -> bool:
    if not (x.is_cuda and lib.available() and x.dtype == torch.bfloat16 and weight.dtype == torch.bfloat16 and x.shape[-1] % 8 == 0):
        return False
    if weight.shape[0] % 8 == 0:
        return True
    return weight.shape[0] > 128 and _gemm._copy_job_provider is None and _only_first_derivatives()
