"""Basic modules: Linear, Embedding, RmsNorm, LayerNorm, Dropout.

These replace the Haliax ``hnn`` modules the reference is built from.  Weights are kept as plain 2-D
``[out, in]`` matrices (what the tcgen05 GEMM consumes).  Each parameter carries the metadata needed to write
it in the reference's checkpoint layout:

``lev_shape``        the articulated shape, e.g. ``(kv_head, q_per_group, head_size, embed)``
``lev_transposed``   True when the reference stores ``[in..., out...]`` (``out_first=False``, GPT-2 style)
``tp_dim``           which local dim is tensor-parallel sharded (None when replicated)

Class names matter: the default weight-decay mask excludes parameters whose class-qualified path contains
``LayerNorm``, ``RmsNorm`` or ``Embedding`` (src/levanter/optim/config.py:149-161).
"""
from __future__ import annotations

import math
import threading
from typing import Optional, Sequence, Tuple

import torch
import torch.nn as nn
import torch.nn.functional as F


def _prod(xs: Sequence[int]) -> int:
    out = 1
    for x in xs:
        out *= int(x)
    return out


def trunc_normal_(t: torch.Tensor, std: float) -> torch.Tensor:
    with torch.no_grad():
        return nn.init.trunc_normal_(t, mean=0.0, std=std, a=-3 * std, b=3 * std)


class Linear(nn.Module):
    """``y = x W^T + b`` with ``W`` stored ``[out, in]``; bf16 CUDA inputs run on the tcgen05 GEMM."""

    def __init__(self, in_features: int, out_features: int, *, bias: bool = False, init_std: Optional[float] = None,
                 lev_out: Optional[Tuple[int, ...]] = None, lev_in: Optional[Tuple[int, ...]] = None,
                 out_first: bool = True, parallel=None, device=None, dtype=None):
        super().__init__()
        self.in_features = in_features
        self.out_features = out_features
        self.weight = nn.Parameter(torch.empty(out_features, in_features, device=device, dtype=dtype))
        std = init_std if init_std is not None else 1.0 / math.sqrt(in_features)
        if self.weight.device.type != "meta":
            trunc_normal_(self.weight, std)
        lev_out = tuple(lev_out) if lev_out is not None else (out_features,)
        lev_in = tuple(lev_in) if lev_in is not None else (in_features,)
        assert _prod(lev_out) == out_features and _prod(lev_in) == in_features
        self.weight.lev_shape = (lev_out + lev_in) if out_first else (lev_in + lev_out)
        self.weight.lev_transposed = not out_first
        kind = parallel[0] if parallel is not None and parallel[1] is not None and parallel[1].size > 1 else None
        self.weight.tp_dim = {None: None, "column": 0, "row": 1}[kind]
        if bias:
            self.bias = nn.Parameter(torch.zeros(out_features, device=device, dtype=dtype))
            self.bias.lev_shape = lev_out
            self.bias.lev_transposed = False
            self.bias.tp_dim = 0 if kind == "column" else None
        else:
            self.register_parameter("bias", None)

    def forward(self, x: torch.Tensor, *, skip_bias: bool = False) -> torch.Tensor:
        from .ops.gemm import linear

        b = None if skip_bias else self.bias
        w = self.weight
        if w.dtype != x.dtype:
            w = w.to(x.dtype)
            b = b.to(x.dtype) if b is not None else None
        return linear(x, w, b)

    def extra_repr(self):
        return f"in={self.in_features}, out={self.out_features}, bias={self.bias is not None}"


class FusedRows:
    """One matrix (or vector) whose row slices are the given parameters: projections that read the same rows become one product when
    a model serves, and nothing is stored twice.  :meth:`get` returns it; None for parameters in training, which belong to the gradient engine's own
    flat buffers.  Parameters that are not (or, after a move or a conversion, no longer) its slices are copied there and re-pointed first, unless
    ``build`` is off or a CUDA graph has recorded where they lie (:meth:`hold`): its replays would go on reading the storage that was left.
    ``pad``: zero rows at the end."""

    def __init__(self, pad: int = 0):
        self.pad = pad
        self._held: set = set()  # addresses of parameters that a graph reads one by one

    def _whole(self, params: Sequence[torch.Tensor]) -> Optional[torch.Tensor]:
        """The matrix when its storage consists of the parameters in their order and the padding, and of nothing else."""
        first = params[0]
        storage = first.untyped_storage()
        base = at = storage.data_ptr()
        for p in params:  # a tensor inside the live storage is a slice of it
            if p.data_ptr() != at or p.dtype != first.dtype or not p.is_contiguous():
                return None
            at += p.nbytes
        width = first.stride(0)
        if storage.nbytes() != at - base + self.pad * width * first.itemsize:
            return None
        return first.detach().as_strided((storage.nbytes() // (width * first.itemsize), *first.shape[1:]), first.stride(), 0)

    def hold(self, params: Sequence[torch.Tensor]) -> None:
        """Called where the parameters are read one by one; while a graph is captured they stay where they are from then on."""
        if params and params[0].is_cuda and torch.cuda.is_current_stream_capturing():
            self._held.update(p.data_ptr() for p in params)

    def get(self, params: Sequence[torch.Tensor], build: bool = True) -> Optional[torch.Tensor]:
        if any(getattr(p, "main_grad", None) is not None or getattr(p, "grad_sink", None) is not None for p in params):
            return None
        whole = self._whole(params)
        if whole is not None:
            return whole
        self.hold(params)  # (under capture the copy would be recorded and not made)
        if not build or any(p.is_inference() or p.data_ptr() in self._held for p in params):
            return None
        with _LAYING_OUT:
            whole = self._whole(params)  # another thread may have come first
            if whole is not None:
                return whole
            with torch.inference_mode(False), torch.no_grad():
                rows = list(params)
                if self.pad:
                    rows.append(rows[0].new_zeros(self.pad, *rows[0].shape[1:]))
                whole = torch.cat(rows)
            at = 0
            for p in params:
                if p.is_cuda:  # the copy reads it on this stream, whatever stream it was made on
                    p.data.record_stream(torch.cuda.current_stream(p.device))
                p.data = whole[at:at + p.shape[0]]
                at += p.shape[0]
        return whole


_LAYING_OUT = threading.Lock()


class Embedding(nn.Module):
    """Token embedding ``weight[vocab, embed]`` with ``unembed`` for tied LM heads."""

    def __init__(self, num_embeddings: int, embedding_dim: int, *, init_std: float = 0.02, device=None, dtype=None):
        super().__init__()
        self.num_embeddings = num_embeddings
        self.embedding_dim = embedding_dim
        self.weight = nn.Parameter(torch.empty(num_embeddings, embedding_dim, device=device, dtype=dtype))
        if self.weight.device.type != "meta":
            trunc_normal_(self.weight, init_std)
        self.weight.lev_shape = (num_embeddings, embedding_dim)
        self.weight.lev_transposed = False
        self.weight.tp_dim = None

    def forward(self, ids: torch.Tensor) -> torch.Tensor:
        from .ops.embedding import embedding

        return embedding(ids, self.weight)

    embed = forward

    def unembed(self, x: torch.Tensor) -> torch.Tensor:
        from .ops.gemm import linear

        w = self.weight if self.weight.dtype == x.dtype else self.weight.to(x.dtype)
        return linear(x, w, None)

    def resize_embeddings(self, new_size: int, init_std: float = 0.02) -> "Embedding":
        """Return a copy with ``new_size`` rows; new rows are freshly initialised."""
        new = Embedding(new_size, self.embedding_dim, init_std=init_std, device=self.weight.device, dtype=self.weight.dtype)
        n = min(new_size, self.num_embeddings)
        with torch.no_grad():
            new.weight[:n].copy_(self.weight[:n])
        return new


class RmsNorm(nn.Module):
    """``x * rsqrt(mean(x^2) + eps) * weight (+ bias)`` computed in fp32."""

    def __init__(self, dim: int, eps: float = 1e-6, use_weight: bool = True, use_bias: bool = False, device=None, dtype=None):
        super().__init__()
        self.dim = dim
        self.eps = eps
        if use_weight:
            self.weight = nn.Parameter(torch.ones(dim, device=device, dtype=dtype))
            self.weight.lev_shape = (dim,)
        else:
            self.register_parameter("weight", None)
        if use_bias:
            self.bias = nn.Parameter(torch.zeros(dim, device=device, dtype=dtype))
            self.bias.lev_shape = (dim,)
        else:
            self.register_parameter("bias", None)

    def forward(self, x: torch.Tensor, fork: bool = False):
        """``fork``: ``(norm(x), x)``, see ``ops.norm.norm_and_input``."""
        from .ops.norm import norm_and_input, rms_norm

        return norm_and_input(x, self.weight, self.bias, self.eps, layer_norm=False) if fork else rms_norm(x, self.weight, self.bias, self.eps)

    def from_stream(self, x: torch.Tensor, rows: Optional[torch.Tensor] = None) -> torch.Tensor:
        """The norm of an fp32 residual stream, in the weight's dtype (``rows``: of these rows only)."""
        from .ops.residual_stream import rms_norm_stream

        assert self.weight is not None and self.bias is None
        return rms_norm_stream(x, self.weight, self.eps, rows=rows)


class GroupedRmsNorm(RmsNorm):
    """:class:`RmsNorm` whose rows are split into ``groups`` equal consecutive parts with a root mean square each."""

    def __init__(self, dim: int, groups: int, eps: float = 1e-6, device=None, dtype=None):
        super().__init__(dim, eps=eps, device=device, dtype=dtype)
        if groups <= 0 or dim % groups != 0:
            raise ValueError(f"a row of {dim} elements has no {groups} equal groups")
        self.groups = groups

    def in_fp32(self, x: torch.Tensor) -> torch.Tensor:
        from .ops.depth_stream import grouped_rms_norm

        return grouped_rms_norm(x, self.weight, self.eps, self.groups)

    def forward(self, x: torch.Tensor) -> torch.Tensor:
        return self.in_fp32(x).to(x.dtype)

    def from_stream(self, x: torch.Tensor, rows: Optional[torch.Tensor] = None) -> torch.Tensor:
        from .ops.depth_stream import norm_of_depths

        if torch.is_grad_enabled():
            x = x if rows is None else x.index_select(0, rows.long())
            return self.in_fp32(x).to(self.weight.dtype)
        y = norm_of_depths(x.reshape(1, -1, self.dim), self.weight, self.eps, groups=self.groups, rows=rows)
        return y.view_as(x) if rows is None else y


class LayerNorm(nn.Module):
    def __init__(self, dim: int, eps: float = 1e-5, use_weight: bool = True, use_bias: bool = True, device=None, dtype=None):
        super().__init__()
        self.dim = dim
        self.eps = eps
        if use_weight:
            self.weight = nn.Parameter(torch.ones(dim, device=device, dtype=dtype))
            self.weight.lev_shape = (dim,)
        else:
            self.register_parameter("weight", None)
        if use_bias:
            self.bias = nn.Parameter(torch.zeros(dim, device=device, dtype=dtype))
            self.bias.lev_shape = (dim,)
        else:
            self.register_parameter("bias", None)

    def forward(self, x: torch.Tensor, fork: bool = False):
        """``fork``: ``(norm(x), x)``, see ``ops.norm.norm_and_input``."""
        from .ops.norm import layer_norm, norm_and_input

        return norm_and_input(x, self.weight, self.bias, self.eps, layer_norm=True) if fork else layer_norm(x, self.weight, self.bias, self.eps)


def plain(m: nn.Module, *kinds: type) -> bool:
    """Whether ``m`` is one of these classes itself and a call of it is its ``forward`` and nothing else: no hook of any kind that would have to see the
    call, its gradients or its result, and no ``forward`` of the instance.  Only then may a layer do the module's work in another way."""
    return (type(m) in kinds and not m._forward_hooks and not m._forward_pre_hooks and not m._backward_hooks and not m._backward_pre_hooks
            and "forward" not in m.__dict__ and not torch.nn.modules.module._has_any_global_hook())


def fork_norm(norm: nn.Module, x: torch.Tensor) -> Tuple[torch.Tensor, torch.Tensor]:
    """``(norm(x), x)`` of any norm module; this module's own add the two gradients of ``x`` in the norm's backward pass."""
    return norm(x, fork=True) if plain(norm, RmsNorm, LayerNorm) else (norm(x), x)


def linear_many(x: torch.Tensor, *projections: nn.Module):
    """The projections of the same rows, one by one; in training their input gradients are summed in the epilogues of their products."""
    from .ops.gemm import linear_many as many

    if x.requires_grad and torch.is_grad_enabled() and all(plain(m, Linear) and m.bias is None and getattr(m.weight, "grad_sink", None) is None
                                                          for m in projections):
        got = many(x, [m.weight for m in projections])
        if got is not None:
            return got
    return tuple(m(x) for m in projections)


class Dropout(nn.Module):
    """Dropout that is inert at ``p == 0`` or in eval mode (all shipped configs use ``p = 0``)."""

    def __init__(self, p: float = 0.0):
        super().__init__()
        self.p = p

    def forward(self, x: torch.Tensor) -> torch.Tensor:
        if self.p == 0.0 or not self.training:
            return x
        from .ops.dropout import dropout

        return dropout(x, self.p, training=True)
