"""bf16 GEMM on tcgen05 tensor cores (see ``csrc/gemm_bf16.cu``) and the ``linear`` autograd op on top of it.

Replaces the dense projections that the reference lowers through ``hnn.Linear`` /
``hax.dot`` (src/levanter/layers/attention.py:1606-1635, src/levanter/models/llama.py:273-280).
"""
from __future__ import annotations

from typing import Optional

import torch

from . import lib

F_OUT_F32 = 1
F_ACCUMULATE = 2
F_BIAS = 4
F_RESIDUAL = 8
F_BIAS_F32 = 16
F_SQUARED_RELU = 32

_gemm_fn = None


def _fn():
    global _gemm_fn
    if _gemm_fn is None:
        c = lib
        _gemm_fn = lib.fn(
            "lvb_gemm_bf16",
            [c.c_void_p, c.c_void_p, c.c_void_p, c.c_int, c.c_int, c.c_int, c.c_int, c.c_int, c.c_int, c.c_int,
             c.c_int, c.c_int, c.c_float, c.c_void_p, c.c_void_p, c.c_int, c.c_int, c.c_void_p, c.c_void_p],
        )
    return _gemm_fn


def _rowmajor_2d(t: torch.Tensor) -> torch.Tensor:
    if t.dim() != 2:
        raise ValueError(f"expected a 2-D tensor, got {tuple(t.shape)}")
    if t.stride(1) != 1 or t.stride(0) % 8 != 0 or t.data_ptr() % 16 != 0:
        t = t.contiguous()
    return t


def gemm_reference(a, b, *, a_mn=False, b_mn=False, out=None, out_dtype=torch.bfloat16, accumulate=False,
                   bias=None, residual=None, alpha=1.0, squared_relu=False):
    """PyTorch fp32 statement of :func:`gemm` (used on CPU and as the test oracle)."""
    af = (a.t() if a_mn else a).float()
    bf = (b if b_mn else b.t()).float()
    c = alpha * (af @ bf)
    if bias is not None:
        c = c + bias.float()
    if squared_relu:
        c = torch.relu(c).square()
    if residual is not None:
        c = c + residual.float()
    if out is not None:
        if accumulate:
            c = c + out.float()
        out.copy_(c.to(out.dtype))
        return out
    return c.to(out_dtype)


def gemm(
    a: torch.Tensor,
    b: torch.Tensor,
    *,
    a_mn: bool = False,
    b_mn: bool = False,
    out: Optional[torch.Tensor] = None,
    out_dtype: torch.dtype = torch.bfloat16,
    accumulate: bool = False,
    bias: Optional[torch.Tensor] = None,
    residual: Optional[torch.Tensor] = None,
    alpha: float = 1.0,
    max_ctas: int = 0,
    squared_relu: bool = False,
) -> torch.Tensor:
    """``C[M,N] = alpha * op(A) @ op(B)^T (+bias) (+residual) (+C)``; ``squared_relu`` applies ``max(., 0)^2`` to the product
    and bias before the residual and the old ``C`` are added.

    ``a`` is ``[M,K]`` (``a_mn=False``) or ``[K,M]`` (``a_mn=True``); ``b`` is ``[N,K]`` or ``[K,N]``.
    Inputs are bf16; the accumulator is fp32; ``out`` may be bf16 or fp32.
    """
    if not (a.is_cuda and lib.available()):
        return gemm_reference(a, b, a_mn=a_mn, b_mn=b_mn, out=out, out_dtype=out_dtype, accumulate=accumulate,
                              bias=bias, residual=residual, alpha=alpha, squared_relu=squared_relu)
    if a.dtype != torch.bfloat16 or b.dtype != torch.bfloat16:
        raise TypeError("gemm expects bf16 operands")
    a = _rowmajor_2d(a)
    b = _rowmajor_2d(b)
    if a_mn:
        K, M = a.shape
    else:
        M, K = a.shape
    if b_mn:
        Kb, N = b.shape
    else:
        N, Kb = b.shape
    if K != Kb:
        raise ValueError(f"reduction dims differ: {K} vs {Kb}")
    if out is None:
        out = torch.empty((M, N), dtype=out_dtype, device=a.device)
        if accumulate:
            raise ValueError("accumulate=True needs out=")
    else:
        if out.shape != (M, N) or out.stride(1) != 1:
            raise ValueError("out has the wrong shape or is not row-major")
    flags = 0
    if out.dtype == torch.float32:
        flags |= F_OUT_F32
    elif out.dtype != torch.bfloat16:
        raise TypeError("out must be bf16 or fp32")
    if accumulate:
        flags |= F_ACCUMULATE
    if squared_relu:
        flags |= F_SQUARED_RELU
    if bias is not None:
        flags |= F_BIAS
        if bias.dtype == torch.float32:
            flags |= F_BIAS_F32
        bias = bias.contiguous()
    ldr = 0
    if residual is not None:
        flags |= F_RESIDUAL
        if residual.dtype != torch.bfloat16 or residual.stride(-1) != 1:
            residual = residual.to(torch.bfloat16).contiguous()
        residual = residual.view(M, N) if residual.dim() != 2 else residual
        ldr = residual.stride(0)
    if _use_skinny(M, N) and not a_mn and not b_mn and max_ctas == 0:
        # a few row blocks (decode steps, small batches): the weight-streaming kernel
        rc = _skinny_fn()(
            a.data_ptr(), b.data_ptr(), out.data_ptr(), M, N, K, a.stride(0), b.stride(0), out.stride(0), flags, float(alpha),
            lib.ptr(bias), lib.ptr(residual), ldr, 0, 0, _skinny_workspace(a.device, M, N),
            lib.status_buffer().data_ptr(), lib.stream_ptr(),
        )
        lib.check_rc(rc, "lvb_gemm_skinny")
        return out
    if _copy_job_provider is not None and N > 128 and max_ctas == 0:
        job = _copy_job_provider(2.0 * M * N * K)
        if job is not None:
            table, u0, u1, srcs, n_srcs, dst = job
            rc = (_cj_pair_fn() if (PAIR_ENABLED and M > 128) else _cj_fn())(
                a.data_ptr(), b.data_ptr(), out.data_ptr(), M, N, K, a.stride(0), b.stride(0), out.stride(0),
                int(a_mn), int(b_mn), flags, float(alpha), lib.ptr(bias), lib.ptr(residual), ldr,
                table, u0, u1, srcs, n_srcs, dst, lib.status_buffer().data_ptr(), lib.stream_ptr(),
            )
            lib.check_rc(rc, "lvb_gemm_bf16_copy_job")
            return out
    pair = PAIR_ENABLED and N > 128 and M > 128
    if pair and not a_mn and not b_mn and max_ctas == 0 and _use_pair_splitk(M, N, K):
        rc = _pair_splitk_fn()(
            a.data_ptr(), b.data_ptr(), out.data_ptr(), M, N, K, a.stride(0), b.stride(0), out.stride(0), flags, float(alpha),
            lib.ptr(bias), lib.ptr(residual), ldr, 0, _splitk_workspace(a.device), lib.status_buffer().data_ptr(), lib.stream_ptr(),
        )
        lib.check_rc(rc, "lvb_gemm_bf16_pair_splitk")
        return out
    rc = (_pair_fn() if pair else _fn())(
        a.data_ptr(), b.data_ptr(), out.data_ptr(), M, N, K, a.stride(0), b.stride(0), out.stride(0),
        int(a_mn), int(b_mn), flags, float(alpha), lib.ptr(bias), lib.ptr(residual), ldr, int(max_ctas),
        lib.status_buffer().data_ptr(), lib.stream_ptr(),
    )
    lib.check_rc(rc, "lvb_gemm_bf16_pair" if pair else "lvb_gemm_bf16")
    return out


# Large products run on CTA pairs (``csrc/gemm_pair.cu``: 256 x 256 tiles, tcgen05 cta_group::2); ``LEVANTER_B200_GEMM_PAIR=0``
# keeps everything on the one-CTA kernel.
import os as _os

PAIR_ENABLED = _os.environ.get("LEVANTER_B200_GEMM_PAIR", "1") != "0"
_pair = None


def _pair_fn():
    global _pair
    if _pair is None:
        c = lib
        _pair = lib.fn(
            "lvb_gemm_bf16_pair",
            [c.c_void_p, c.c_void_p, c.c_void_p, c.c_int, c.c_int, c.c_int, c.c_int, c.c_int, c.c_int, c.c_int,
             c.c_int, c.c_int, c.c_float, c.c_void_p, c.c_void_p, c.c_int, c.c_int, c.c_void_p, c.c_void_p],
        )
    return _pair


_pair_splitk = None
SPLITK_MODE = _os.environ.get("LEVANTER_B200_SMALL_M", "splitk")  # what 128 < M products with few tiles run on: splitk | stream | general


def _pair_splitk_fn():
    global _pair_splitk
    if _pair_splitk is None:
        c = lib
        _pair_splitk = lib.fn("lvb_gemm_bf16_pair_splitk",
                              [c.c_void_p, c.c_void_p, c.c_void_p] + [c.c_int] * 7 + [c.c_float, c.c_void_p, c.c_void_p, c.c_int, c.c_int,
                                                                                       c.c_void_p, c.c_void_p, c.c_void_p], launches=2)
    return _pair_splitk


def _use_pair_splitk(M: int, N: int, K: int) -> bool:
    """Few 256 x 256 tiles (at most half the 74 SM pairs) and a K long enough to split, N % 4 == 0: the decode-size
    projections, where whole-K tiles would leave most SMs idle."""
    tiles = ((M + 255) // 256) * ((N + 255) // 256)
    return SPLITK_MODE == "splitk" and tiles <= 37 and K >= 1024 and N % 4 == 0


def _splitk_workspace(device) -> int:
    """The split-K scratch shared with the streaming kernel (tiles x splits <= 74 pieces of 256 x 256 fp32 fit in it)."""
    ws = _skinny_ws.get(device)
    if ws is None:
        ws = _skinny_ws[device] = torch.empty(8 * _SKINNY_SPLIT_MAX_TILES * 128 * 128 * 4, dtype=torch.uint8, device=device)
    return ws.data_ptr()


# A provider of copy jobs (``flops -> (table_ptr, u0, u1, src_ptr_array, n_srcs, dst_ptr) | None``): when one is set, dense
# GEMMs ask it before every launch and, given a job, run the kernel variant whose extra warp carries out the copies beside
# the tensor cores (the next layer's weight gather of fully sharded training, ``parallel/zero3.py``).
_copy_job_provider = None
_cj = None


def set_copy_job_provider(fn) -> None:
    global _copy_job_provider
    _copy_job_provider = fn


_cj_pair = None


def _cj_pair_fn():
    global _cj_pair
    if _cj_pair is None:
        c = lib
        _cj_pair = lib.fn("lvb_gemm_bf16_pair_copy_job",
                          [c.c_void_p, c.c_void_p, c.c_void_p] + [c.c_int] * 9 + [c.c_float, c.c_void_p, c.c_void_p, c.c_int,
                                                                                   c.c_void_p, c.c_int, c.c_int, c.c_void_p, c.c_int, c.c_void_p,
                                                                                   c.c_void_p, c.c_void_p])
    return _cj_pair


def _cj_fn():
    global _cj
    if _cj is None:
        c = lib
        _cj = lib.fn("lvb_gemm_bf16_copy_job",
                     [c.c_void_p, c.c_void_p, c.c_void_p] + [c.c_int] * 9 + [c.c_float, c.c_void_p, c.c_void_p, c.c_int,
                                                                              c.c_void_p, c.c_int, c.c_int, c.c_void_p, c.c_int, c.c_void_p,
                                                                              c.c_void_p, c.c_void_p])
    return _cj


SKINNY_MAX_ROWS = 128          # up to here the weight-streaming kernel always runs
SKINNY_MAX_ROWS_NARROW = 512   # up to here it runs when the general kernel's 256 x 256 tiles would leave most SMs idle
_SKINNY_NARROW_TILES = int(_os.environ.get("LEVANTER_B200_SKINNY_NARROW_TILES", "48"))
_skinny = None


def _use_skinny(M: int, N: int) -> bool:
    if M <= SKINNY_MAX_ROWS:
        return True
    if M > SKINNY_MAX_ROWS_NARROW or SPLITK_MODE != "stream":
        return False
    return ((M + 255) // 256) * ((N + 255) // 256) <= _SKINNY_NARROW_TILES


def _skinny_fn():
    global _skinny
    if _skinny is None:
        c = lib
        _skinny = lib.fn("lvb_gemm_skinny", [c.c_void_p, c.c_void_p, c.c_void_p] + [c.c_int] * 7 + [c.c_float, c.c_void_p, c.c_void_p,
                                                                                                  c.c_int, c.c_int, c.c_int, c.c_void_p, c.c_void_p,
                                                                                                  c.c_void_p], launches=2)
    return _skinny


_skinny_ws = {}


def _skinny_workspace(device, M: int, N: int) -> int:
    """Address of the per-device scratch for the split-K partials of the streaming kernel, or 0 when the launcher will not
    split (wide outputs already give every SM a tile).  Successive GEMMs on a stream reuse the scratch safely: each one's
    second kernel has consumed it before the next one's first kernel writes it."""
    if ((M + 127) // 128) * ((N + 127) // 128) > _SKINNY_SPLIT_MAX_TILES:
        return 0
    ws = _skinny_ws.get(device)
    if ws is None:
        ws = _skinny_ws[device] = torch.empty(8 * _SKINNY_SPLIT_MAX_TILES * 128 * 128 * 4, dtype=torch.uint8, device=device)
    return ws.data_ptr()


_SKINNY_SPLIT_MAX_TILES = 74  # more 128 x 128 tiles than half the SMs: the launcher does not split K


_col_sum = None


def col_sum(x: torch.Tensor, dtype: torch.dtype) -> torch.Tensor:
    """Sums of the columns of bf16 ``x [rows, cols]`` in fp32, as ``dtype`` where that is bf16 and as fp32 otherwise."""
    global _col_sum
    rows, cols = x.shape
    if not (x.is_cuda and lib.available() and rows > 0 and cols % 8 == 0 and x.stride(1) == 1 and x.stride(0) % 8 == 0 and x.data_ptr() % 16 == 0):
        return x.float().sum(0)
    if _col_sum is None:
        c = lib
        _col_sum = (lib.fn("lvb_col_sum", [c.c_void_p, c.c_longlong, c.c_void_p, c.c_int, c.c_void_p, c.c_int, c.c_int, c.c_void_p], launches=2),
                    lib.fn("lvb_col_sum_shares", [c.c_int] * 2, launches=0))
    out = torch.empty(cols, dtype=dtype if dtype == torch.bfloat16 else torch.float32, device=x.device)
    scratch = torch.empty(_col_sum[1](rows, cols) * cols, dtype=torch.float32, device=x.device)
    rc = _col_sum[0](x.data_ptr(), x.stride(0), out.data_ptr(), int(out.dtype == torch.bfloat16), scratch.data_ptr(), rows, cols, lib.stream_ptr())
    lib.check_rc(rc, "lvb_col_sum")
    return out


_few_dw = None


def few_outputs_dw(dy: torch.Tensor, x: torch.Tensor, out_dtype: torch.dtype) -> Optional[torch.Tensor]:
    """``dy^T x`` of rows ``dy [rows, outputs]`` and ``x [rows, cols]`` with few outputs and many rows, or None where the GEMM is the better form.  Its
    few tiles walk all rows, 5 us and 5.1 more per 1024 rows whatever the columns (16384 rows: 88); the lanes' time goes with rows x outputs x columns.
    us, lanes / GEMM: 8 x 1024 over 1024 rows 7.1 / 9.9, over 16384 15 / 88; 16 x 1024 8.4 / 9.9, 26 / 88; 32 x 1024 11.7 / 9.8, over 2048 13.9 / 15.1, over
    16384 46 / 88; 8 x 4096 11.7 / 10.0, 13.9 / 15.2, 72 / 100; 16 x 4096 over 2048 21.9 / 15.2, over 16384 134 / 97."""
    global _few_dw
    (rows, outputs), cols = dy.shape, x.shape[1]
    if not (0 < outputs <= 32 and rows >= 1024 and outputs * cols <= min(16 * rows, 32768) and x.is_cuda and lib.available() and outputs % 8 == 0 and cols % 8 == 0 and out_dtype in (torch.bfloat16, torch.float32)
            and dy.dtype == x.dtype == torch.bfloat16 and all(t.stride(1) == 1 and t.stride(0) % 8 == 0 and t.data_ptr() % 16 == 0 for t in (dy, x))):
        return None
    if _few_dw is None:
        c = lib
        _few_dw = (lib.fn("lvb_few_outputs_dw", [c.c_void_p, c.c_longlong] * 2 + [c.c_void_p, c.c_int, c.c_void_p] + [c.c_int] * 3 + [c.c_void_p], launches=2),
                   lib.fn("lvb_few_outputs_dw_shares", [c.c_int] * 3, launches=0))
    out = torch.empty(outputs, cols, dtype=out_dtype, device=x.device)
    scratch = torch.empty(_few_dw[1](rows, outputs, cols) * outputs * cols, dtype=torch.float32, device=x.device)
    rc = _few_dw[0](dy.data_ptr(), dy.stride(0), x.data_ptr(), x.stride(0), out.data_ptr(), int(out_dtype == torch.bfloat16), scratch.data_ptr(), rows, outputs,
                    cols, lib.stream_ptr())
    lib.check_rc(rc, "lvb_few_outputs_dw")
    return out


def _linear_rows(x, weight, bias, residual):
    shp = x.shape
    y = gemm(x.reshape(-1, shp[-1]), weight, bias=bias, residual=None if residual is None else residual.reshape(-1, weight.shape[0]))
    return y.view(*shp[:-1], weight.shape[0])


def _weight_grad(weight, dy2, x2) -> Optional[torch.Tensor]:
    """``dy^T x`` for a parameter, or None when it goes into the parameter's own buffer (see :class:`_LinearFn`)."""
    main_grad = getattr(weight, "main_grad", None)
    sink = getattr(weight, "grad_sink", None)
    if sink is not None:
        sink(dy2, x2)  # fully sharded weights: the product is reduce-scattered to the rows' owners as it is computed
        return None
    if main_grad is not None:
        gemm(dy2, x2, a_mn=True, b_mn=True, out=main_grad, accumulate=True)
        return None
    dtype = weight.dtype if weight.dtype in (torch.bfloat16, torch.float32) else torch.float32
    dw = few_outputs_dw(dy2, x2, dtype)
    return dw if dw is not None else gemm(dy2, x2, a_mn=True, b_mn=True, out_dtype=dtype)


class _LinearFn(torch.autograd.Function):
    """y = x W^T (+ b).  ``weight`` is ``[out, in]``.

    If ``weight`` carries a ``main_grad`` attribute (an fp32 buffer of the same shape, owned by the
    sharded-gradient engine) the weight gradient is accumulated straight into it by the GEMM
    epilogue and autograd sees no dense weight gradient.  If it carries a ``grad_sink`` (weights that exist only as
    row slices per rank, ``parallel/zero3.py``) the two operands of the weight-gradient product are handed to it.
    """

    @staticmethod
    def forward(ctx, x, weight, bias, residual=None):
        ctx.save_for_backward(x.reshape(-1, x.shape[-1]), weight)
        ctx.has_bias = bias is not None
        ctx.bias_dtype = None if bias is None else bias.dtype
        ctx.has_res = residual is not None
        ctx.x_shape = x.shape
        ctx.weight_ref = weight
        return _linear_rows(x, weight, bias, residual)

    @staticmethod
    def backward(ctx, dy):
        x2, weight = ctx.saved_tensors
        dy2 = dy.reshape(-1, dy.shape[-1])
        if dy2.dtype != torch.bfloat16:
            dy2 = dy2.to(torch.bfloat16)
        dx = dw = db = None
        if ctx.needs_input_grad[0]:
            dx = gemm(dy2, weight, b_mn=True).view(ctx.x_shape)
        if ctx.needs_input_grad[1]:
            dw = _weight_grad(ctx.weight_ref, dy2, x2)
        if ctx.has_bias and ctx.needs_input_grad[2]:
            db = col_sum(dy2, ctx.bias_dtype)
        dres = dy if ctx.has_res else None
        return dx, dw, db, dres


def _tma_shapes_ok(weight: torch.Tensor) -> bool:
    """Forward, input-gradient and weight-gradient GEMMs each read ``weight`` or the activations with one of the two feature
    sizes as the row stride, and a TMA row stride must be a multiple of 16 bytes: both sizes must be multiples of 8 (a
    router with 4 experts, for one, goes to the library GEMM)."""
    return weight.dim() == 2 and weight.shape[0] % 8 == 0 and weight.shape[1] % 8 == 0


def linear(x: torch.Tensor, weight: torch.Tensor, bias: Optional[torch.Tensor] = None) -> torch.Tensor:
    """Linear layer on the tcgen05 GEMM when running bf16 on a B200; ``F.linear`` otherwise."""
    if x.is_cuda and lib.available() and x.dtype == torch.bfloat16 and weight.dtype == torch.bfloat16 and _tma_shapes_ok(weight):
        return _linear_rows(x, weight, bias, None) if lib.plain_call() else _LinearFn.apply(x, weight, bias, None)
    return torch.nn.functional.linear(x, weight, bias)


def linear_residual(x: torch.Tensor, weight: torch.Tensor, bias: Optional[torch.Tensor], residual: Optional[torch.Tensor]) -> torch.Tensor:
    """``x W^T + b + residual`` with the residual added in the GEMM epilogue (one pass over the output)."""
    if residual is None:
        return linear(x, weight, bias)
    if weight.dtype != x.dtype:
        weight = weight.to(x.dtype)
        bias = bias.to(x.dtype) if bias is not None else None
    if x.is_cuda and lib.available() and x.dtype == torch.bfloat16 and residual.dtype == torch.bfloat16 and _tma_shapes_ok(weight):
        return _linear_rows(x, weight, bias, residual) if lib.plain_call() else _LinearFn.apply(x, weight, bias, residual)
    return torch.nn.functional.linear(x, weight, bias) + residual


class _LinearManyFn(torch.autograd.Function):
    """Several projections of the same rows: every product of the backward pass adds its input gradient to that of the ones before it in its
    epilogue, and one function stands where there were several."""

    @staticmethod
    def forward(ctx, x, *weights):
        ctx.save_for_backward(x.reshape(-1, x.shape[-1]), *weights)
        ctx.x_shape = x.shape
        ctx.refs = weights
        ctx.set_materialize_grads(False)  # a product that nothing uses has no gradient, and its weight none
        return tuple(_linear_rows(x, w, None, None) for w in weights)

    @staticmethod
    def backward(ctx, *dys):
        x2, *weights = ctx.saved_tensors
        dx, dws = None, []
        for i, (dy, w, ref) in enumerate(zip(dys, weights, ctx.refs)):
            if dy is None:
                dws.append(None)
                continue
            dy2 = dy.reshape(-1, dy.shape[-1])
            if dy2.dtype != torch.bfloat16:
                dy2 = dy2.to(torch.bfloat16)
            if ctx.needs_input_grad[0]:
                dx = gemm(dy2, w, b_mn=True, out=dx, accumulate=dx is not None)
            dws.append(_weight_grad(ref, dy2, x2) if ctx.needs_input_grad[1 + i] else None)
        return (None if dx is None else dx.view(ctx.x_shape), *dws)


MANY_ROWS = 2048


def linear_many(x: torch.Tensor, weights):
    """``[x W^T for W in weights]`` on the tcgen05 GEMM, or None where :func:`linear` would not take it for all of them, and for more rows than the
    host's part bounds.  What one function saves is autograd's work per projection; on the device an epilogue that reads back what it adds to costs as much
    as a pass of its own or more (input gradients of six projections 1024 wide: 1500 rows 88 us, 70 with added passes; 16384 rows 284, 236; of two
    2048 wide 81, 76 and 555, 555).  Gated DeltaNet, two layers: 1500 rows 5.40 -> 4.95 ms, 16384 rows 22.96 -> 23.71."""
    if not (x.numel() <= MANY_ROWS * x.shape[-1] and x.is_cuda and lib.available() and x.dtype == torch.bfloat16 and all(w.dtype == torch.bfloat16 and _tma_shapes_ok(w) for w in weights)):
        return None
    return _LinearManyFn.apply(x, *weights)
