"""``torch.library`` custom ops of the CUDA path, with autograd.

Namespace ``natten_b200``.  The rank-specific ops keep the schemas of the
reference's ``natten_mps::*`` ops (``src/natten_mps/_torch_ops.py:39-42, 82-85,
286-289, 583-586``) so code written against them only changes the namespace:

    na{1,2,3}d_qk(query, key, kernel_size, dilation, stride, is_causal, scale?) -> Tensor
    na{1,2,3}d_av(attn, value, kernel_size, dilation, stride, is_causal) -> Tensor
    na{1,2,3}d_fwd(query, key, value, kernel_size, stride, dilation, is_causal, scale?) -> Tensor
    na{1,2,3}d_varlen_fwd(query, key, value, sizes, kernel_size, dilation, scale?) -> Tensor

They are thin compositions of four rank-generic ops that own the kernels:

    na_fused      -> (out, lse)   fused forward; GQA, additional tokens, extents
    na_fused_bwd  -> (dq, dk, dv, d_extra_k, d_extra_v)
    na_qk / na_qk_bwd,  na_qk_rpb / na_qk_rpb_bwd,  na_av / na_av_bwd

Schemas and ``Meta`` shape functions are here; the ``CUDA`` and autograd kernels are
native (``csrc/torch_ops.cpp``).  Nothing is registered for other devices: calling an op
with CPU tensors fails in the dispatcher instead of silently running something else.
"""
from __future__ import annotations

import os
from typing import List, Sequence

import torch

LIB = torch.library.Library("natten_b200", "DEF")


def _strided(spatial: Sequence[int], stride: Sequence[int]) -> List[int]:
    return [(n - 1) // s + 1 for n, s in zip(spatial, stride)]


# ---------------------------------------------------------------------------
# rank-generic fused op
# ---------------------------------------------------------------------------
LIB.define(
    "na_fused(Tensor query, Tensor key, Tensor value, Tensor? extra_k, Tensor? extra_v, "
    "Tensor? extents, int[] kernel_size, int[] stride, int[] dilation, bool[] is_causal, "
    "float scale) -> (Tensor, Tensor)")
LIB.define(
    "na_fused_bwd(Tensor query, Tensor key, Tensor value, Tensor? extra_k, Tensor? extra_v, "
    "Tensor? extents, Tensor out, Tensor lse, Tensor dout, Tensor? dlse, int[] kernel_size, "
    "int[] stride, int[] dilation, bool[] is_causal, float scale) "
    "-> (Tensor, Tensor, Tensor, Tensor, Tensor)")


@torch.library.impl(LIB, "na_fused", "Meta")
def _na_fused_meta(query, key, value, extra_k, extra_v, extents, kernel_size, stride, dilation,
                   is_causal, scale):
    rank = query.ndim - 3
    osp = _strided(query.shape[1:1 + rank], stride)
    out = query.new_empty((query.shape[0], *osp, query.shape[-2], value.shape[-1]))
    acc = torch.float64 if query.dtype == torch.float64 else torch.float32
    lse = query.new_empty((query.shape[0], *osp, query.shape[-2]), dtype=acc)
    return out, lse


@torch.library.impl(LIB, "na_fused_bwd", "Meta")
def _na_fused_bwd_meta(query, key, value, extra_k, extra_v, extents, out, lse, dout, dlse,
                       kernel_size, stride, dilation, is_causal, scale):
    dek = torch.empty_like(extra_k) if extra_k is not None else query.new_empty(0)
    dev = torch.empty_like(extra_v) if extra_v is not None else query.new_empty(0)
    return (query.new_empty(query.shape), key.new_empty(key.shape), value.new_empty(value.shape),
            dek, dev)


# ---------------------------------------------------------------------------
# rank-generic split ops
# ---------------------------------------------------------------------------
LIB.define("na_qk(Tensor query, Tensor key, int[] kernel_size, int[] dilation, int[] stride, "
           "bool[] is_causal, float? scale) -> Tensor")
LIB.define("na_qk_bwd(Tensor dlogits, Tensor query, Tensor key, int[] kernel_size, int[] dilation, "
           "int[] stride, bool[] is_causal, float? scale) -> (Tensor, Tensor)")
LIB.define("na_av(Tensor attn, Tensor value, int[] kernel_size, int[] dilation, int[] stride, "
           "bool[] is_causal) -> Tensor")
LIB.define("na_av_bwd(Tensor dout, Tensor attn, Tensor value, int[] kernel_size, int[] dilation, "
           "int[] stride, bool[] is_causal) -> (Tensor, Tensor)")
LIB.define("na_qk_rpb(Tensor query, Tensor key, Tensor rpb, int[] kernel_size, int[] dilation, float? scale) -> Tensor")
LIB.define("na_qk_rpb_bwd(Tensor dlogits, Tensor query, Tensor key, int[] rpb_shape, int[] kernel_size, "
           "int[] dilation, float? scale) -> (Tensor, Tensor, Tensor)")


@torch.library.impl(LIB, "na_qk", "Meta")
def _na_qk_meta(query, key, kernel_size, dilation, stride, is_causal, scale):
    rank = query.ndim - 3
    ktot = 1
    for x in kernel_size:
        ktot *= x
    return query.new_empty((query.shape[0], *_strided(query.shape[1:1 + rank], stride),
                            query.shape[-2], ktot))


@torch.library.impl(LIB, "na_qk_bwd", "Meta")
def _na_qk_bwd_meta(dlogits, query, key, kernel_size, dilation, stride, is_causal, scale):
    return query.new_empty(query.shape), key.new_empty(key.shape)


@torch.library.impl(LIB, "na_av", "Meta")
def _na_av_meta(attn, value, kernel_size, dilation, stride, is_causal):
    return value.new_empty((*attn.shape[:-1], value.shape[-1]))


@torch.library.impl(LIB, "na_av_bwd", "Meta")
def _na_av_bwd_meta(dout, attn, value, kernel_size, dilation, stride, is_causal):
    return attn.new_empty(attn.shape, dtype=value.dtype), value.new_empty(value.shape)


@torch.library.impl(LIB, "na_qk_rpb", "Meta")
def _na_qk_rpb_meta(query, key, rpb, kernel_size, dilation, scale):
    ktot = 1
    for x in kernel_size:
        ktot *= x
    return query.new_empty((*query.shape[:-1], ktot))


@torch.library.impl(LIB, "na_qk_rpb_bwd", "Meta")
def _na_qk_rpb_bwd_meta(dlogits, query, key, rpb_shape, kernel_size, dilation, scale):
    return query.new_empty(query.shape), key.new_empty(key.shape), query.new_empty(rpb_shape)


# ---------------------------------------------------------------------------
# rank-specific names with the reference's schemas
# ---------------------------------------------------------------------------
def _define_rank_ops(rank: int) -> None:
    LIB.define(f"na{rank}d_qk(Tensor query, Tensor key, int[] kernel_size, int[] dilation, "
               "int[] stride, bool[] is_causal, float? scale) -> Tensor")
    LIB.define(f"na{rank}d_av(Tensor attn, Tensor value, int[] kernel_size, int[] dilation, "
               "int[] stride, bool[] is_causal) -> Tensor")
    LIB.define(f"na{rank}d_fwd(Tensor query, Tensor key, Tensor value, int[] kernel_size, "
               "int[] stride, int[] dilation, bool[] is_causal, float? scale) -> Tensor")
    LIB.define(f"na{rank}d_varlen_fwd(Tensor query, Tensor key, Tensor value, Tensor sizes, "
               "int[] kernel_size, int[] dilation, float? scale) -> Tensor")

    def _check(t, what):
        if t.ndim != rank + 3:
            raise ValueError(f"na{rank}d {what} must have {rank + 3} dimensions, got {t.ndim}.")

    def qk(query, key, kernel_size, dilation, stride, is_causal, scale):
        _check(query, "query")
        return torch.ops.natten_b200.na_qk(query, key, kernel_size, dilation, stride, is_causal, scale)

    def av(attn, value, kernel_size, dilation, stride, is_causal):
        _check(value, "value")
        return torch.ops.natten_b200.na_av(attn, value, kernel_size, dilation, stride, is_causal)

    def fwd(query, key, value, kernel_size, stride, dilation, is_causal, scale):
        _check(query, "query")
        sc = float(query.shape[-1] ** -0.5 if scale is None else scale)
        return torch.ops.natten_b200.na_fused(query, key, value, None, None, None, kernel_size,
                                              stride, dilation, is_causal, sc)[0]

    def varlen_fwd(query, key, value, sizes, kernel_size, dilation, scale):
        _check(query, "query")
        sc = float(query.shape[-1] ** -0.5 if scale is None else scale)
        ones, no = [1] * rank, [False] * rank
        return torch.ops.natten_b200.na_fused(query, key, value, None, None, sizes, kernel_size,
                                              ones, dilation, no, sc)[0]

    for name, fn in ((f"na{rank}d_qk", qk), (f"na{rank}d_av", av), (f"na{rank}d_fwd", fwd),
                     (f"na{rank}d_varlen_fwd", varlen_fwd)):
        LIB.impl(name, fn, "CompositeImplicitAutograd")


for _rank in (1, 2, 3):
    _define_rank_ops(_rank)

OP_NAMES = ("na_fused", "na_fused_bwd", "na_qk", "na_qk_bwd", "na_qk_rpb", "na_qk_rpb_bwd", "na_av", "na_av_bwd") + tuple(
    f"na{r}d_{s}" for r in (1, 2, 3) for s in ("qk", "av", "fwd", "varlen_fwd"))


# ---------------------------------------------------------------------------
# native kernels of the ops, and the functional API's native entry points
# ---------------------------------------------------------------------------
class _NotBuilt:
    """Stands in for the native module in a tree that has not been built: shapes (Meta) still work, calls with
    CUDA tensors fail."""

    def __getattr__(self, name):
        def call(*args):
            if any(isinstance(a, torch.Tensor) and a.is_cuda for a in args):
                raise RuntimeError(f"{_NATIVE_PATH} is missing: build it with `python -m natten_mps_b200._build` "
                                   "(there is no fallback implementation)")
            return NotImplemented
        return call


_NATIVE_PATH = os.path.join(os.path.dirname(os.path.abspath(__file__)), "_native.so")
if os.path.exists(_NATIVE_PATH):
    from . import _native as native      # registers the CUDA and autograd kernels
else:
    native = _NotBuilt()
