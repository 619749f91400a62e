"""Tensor-level front end without autograd: allocates outputs and launches on the current CUDA stream.

The functions here take already-validated, already-normalised arguments (tuples
per axis).  They accept GQA shapes, additional key/value tokens and per-sample
extents directly, so the callers never expand heads or loop over samples.  The
work behind them is native (``csrc/torch_ops.cpp``).
"""
from __future__ import annotations

from typing import Optional

import torch

from . import _torch_ops  # noqa: F401  (registers torch.ops.natten_b200.*)

_OPS = torch.ops.natten_b200


def _require_cuda(*tensors: Optional[torch.Tensor]) -> None:
    for t in tensors:
        if t is not None and not t.is_cuda:
            raise RuntimeError(
                "natten_mps_b200 runs on CUDA tensors only (there is no CPU fallback); "
                f"got a tensor on {t.device}")


def fused_forward(q, k, v, kernel_size, stride, dilation, is_causal, scale: float,
                  extra_k=None, extra_v=None, extents=None):
    """-> (out [B,*O,Hq,Dv], lse [B,*O,Hq] float32/float64)."""
    _require_cuda(q, k, v, extra_k, extra_v)
    with torch.no_grad():
        return _OPS.na_fused(q, k, v, extra_k, extra_v, extents, kernel_size, stride, dilation, is_causal, scale)


def fused_backward(q, k, v, out, lse, dout, kernel_size, stride, dilation, is_causal, scale: float,
                   extra_k=None, extra_v=None, extents=None, dlse=None):
    """-> (dq, dk, dv, d_extra_k, d_extra_v)."""
    _require_cuda(q, k, v, out, lse, dout, extra_k, extra_v, dlse)
    with torch.no_grad():
        dq, dk, dv, dek, dev = _OPS.na_fused_bwd(q, k, v, extra_k, extra_v, extents, out, lse, dout, dlse, kernel_size,
                                                 stride, dilation, is_causal, scale)
    return (dq, dk, dv, None, None) if extra_k is None else (dq, dk, dv, dek, dev)


def qk_forward(q, k, kernel_size, dilation, stride, is_causal, scale: Optional[float]):
    _require_cuda(q, k)
    with torch.no_grad():
        return _OPS.na_qk(q, k, kernel_size, dilation, stride, is_causal, scale)


def qk_backward(dlogits, q, k, kernel_size, dilation, stride, is_causal, scale: Optional[float]):
    _require_cuda(dlogits, q, k)
    with torch.no_grad():
        return _OPS.na_qk_bwd(dlogits, q, k, kernel_size, dilation, stride, is_causal, scale)


def av_forward(attn, v, kernel_size, dilation, stride, is_causal):
    _require_cuda(attn, v)
    with torch.no_grad():
        return _OPS.na_av(attn, v, kernel_size, dilation, stride, is_causal)


def av_backward(dout, attn, v, kernel_size, dilation, stride, is_causal):
    _require_cuda(dout, attn, v)
    with torch.no_grad():
        return _OPS.na_av_bwd(dout, attn, v, kernel_size, dilation, stride, is_causal)


def qk_rpb_forward(q, k, rpb, kernel_size, dilation, scale: Optional[float]):
    """Logits with a relative position bias; ``rpb [H, 2*K_0-1, ...]``."""
    _require_cuda(q, k, rpb)
    with torch.no_grad():
        return _OPS.na_qk_rpb(q, k, rpb, kernel_size, dilation, scale)


def qk_rpb_backward(dlogits, q, k, rpb_shape, kernel_size, dilation, scale: Optional[float]):
    """-> (dq, dk, d_rpb)."""
    _require_cuda(dlogits, q, k)
    with torch.no_grad():
        return _OPS.na_qk_rpb_bwd(dlogits, q, k, rpb_shape, kernel_size, dilation, scale)
