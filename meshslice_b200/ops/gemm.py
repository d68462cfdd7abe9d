"""Local GEMM on the tcgen05 kernel: C = op(A) @ op(B), bf16 inputs, fp32 accumulation.

Layouts follow the reference cost model's naming (CostModel.py:74-98):
  'nn': A [M,K] @ B [K,N]      'nt': A [M,K] @ B[N,K]^T      'tn': A[K,M]^T @ B [K,N]
All operands are row-major; no operand is ever transposed in memory, the tensor-core
descriptors select the major-ness.
"""
from __future__ import annotations

import os

import torch

from .. import _native

_SM_COUNT = {}


def sm_count(device=None) -> int:
    dev = torch.cuda.current_device() if device is None else torch.device(device).index or 0
    if dev not in _SM_COUNT:
        _SM_COUNT[dev] = torch.cuda.get_device_properties(dev).multi_processor_count
    return _SM_COUNT[dev]


def _dims(a, b, layout):
    if layout == "nn":
        M, K = a.shape
        K2, N = b.shape
    elif layout == "nt":
        M, K = a.shape
        N, K2 = b.shape
    elif layout == "tn":
        K, M = a.shape
        K2, N = b.shape
    else:
        raise ValueError(f"unknown layout {layout!r}")
    if K != K2:
        raise ValueError(f"contraction mismatch: {tuple(a.shape)} x {tuple(b.shape)} ({layout})")
    return M, N, K


def _operands(a, b, layout, out, accumulate, out_dtype=torch.bfloat16):
    """Checks one product; returns its output and the thirteen values that the native calls take."""
    M, N, K = _dims(a, b, layout)
    if out is None:
        if accumulate:
            raise ValueError("accumulate=True needs an output tensor")
        out = torch.empty(M, N, dtype=out_dtype, device=a.device)
    (lda, sa), (ldb, sb), (ldc, sc) = a.stride(), b.stride(), out.stride()
    if a.dtype != torch.bfloat16 or b.dtype != torch.bfloat16 or sa != 1 or sb != 1:
        raise ValueError("GEMM operands must be bf16 with a contiguous last dimension")
    if out.shape != (M, N) or sc != 1:
        raise ValueError("bad output shape")
    return out, (M, N, K, a.data_ptr(), lda, 1 if layout == "tn" else 0, b.data_ptr(), ldb, 0 if layout == "nt" else 1,
                 out.data_ptr(), ldc, 1 if out.dtype == torch.float32 else 0, 1 if accumulate else 0)


def gemm(a, b, layout="nn", *, out=None, out_dtype=torch.bfloat16, accumulate=False, bias=None,
         act=None, pre_act=None, two_cta=None):
    """C = op(A) @ op(B) on the tensor cores of the current GPU.  ``two_cta`` selects the
    cta_group::2 kernel (default: on, MSB_TWO_CTA=0 turns it off)."""
    out, v = _operands(a, b, layout, out, accumulate, out_dtype)
    if act is not None and act != "gelu":
        raise ValueError("only act='gelu' is fused")
    _native.load().gemm_local(
        *v, 0 if bias is None else bias.data_ptr(), 0 if act is None else 1,
        0 if act is None or pre_act is None else pre_act.data_ptr(), -1 if two_cta is None else int(bool(two_cta)),
        _SM_COUNT.get(a.device.index) or sm_count(a.device), _native.status().dev, _native.stream_ptr())
    return out


def gemm_pair(a0, b0, layout0, out0, accumulate0, a1, b1, layout1, out1=None, accumulate1=False, gelu_pre=None):
    """Two independent products as ``gemm`` computes them, in one launch (the two gradients of a linear layer): returns
    both outputs.  Neither output may overlap an operand or the output of the other product.  ``gelu_pre`` (bf16, the shape
    of the second product): the second result is multiplied by the derivative of GeLU at it before it is rounded."""
    out0, v0 = _operands(a0, b0, layout0, out0, accumulate0)
    out1, v1 = _operands(a1, b1, layout1, out1, accumulate1)
    pre = 0
    if gelu_pre is not None:
        if gelu_pre.shape != out1.shape or gelu_pre.dtype != torch.bfloat16 or out1.dtype != torch.bfloat16:
            raise ValueError("gelu_pre must be bf16 and of the shape of the second product")
        if gelu_pre.stride() != out1.stride():
            if not out1.is_contiguous():
                raise ValueError("gelu_pre needs a contiguous output")
            gelu_pre = gelu_pre.contiguous()
        if gelu_pre.data_ptr() % 16 and os.environ.get("MSB_TWO_CTA") == "0":
            gelu_pre = gelu_pre.clone()      # a kernel of its own reads it there, 16 bytes at a time
        pre = gelu_pre.data_ptr()
    _native.load().gemm_pair(*v0, *v1, _SM_COUNT.get(a0.device.index) or sm_count(a0.device), _native.status().dev,
                             _native.stream_ptr(), pre)
    return out0, out1
