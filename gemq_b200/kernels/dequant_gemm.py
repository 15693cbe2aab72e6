"""Dequant-fused GEMM; same call signature as gemq/triton_kernels/dequant_gemm.py."""
from __future__ import annotations

from typing import Optional

import torch
from torch import Tensor

from .. import _capi
from ._ops import library_op
from ._runtime import (check_kernel_form, error_word, few_rows_ok, host_linear, linear_rows, one_row_streams, require, require_cuda, stream_ptr,
                       tc_gemm_ok)
from .dequant_gemv import dequant_gemv_rows

_ROW_BLOCK = 64


def _fake_gemm(x, w_q, scales, zeros, nbits, group_size):
    M, K = x.shape
    N = w_q.shape[1]
    tc = tc_gemm_ok(M, N, K, group_size) and x.dtype in (torch.float16, torch.bfloat16)
    return x.new_empty((M, N), dtype=x.dtype if tc else torch.float16)


def _gemm_tc(x: Tensor, w_q: Tensor, scales: Tensor, zeros: Tensor, nbits: int, group_size: int,
             bias: Optional[Tensor]) -> Tensor:
    """The tcgen05 GEMM; the arguments have been checked."""
    x = x.contiguous()
    M, K = x.shape
    N = w_q.shape[1]
    out = torch.empty((M, N), dtype=x.dtype, device=x.device)
    parts = _capi.lib.gemq_linear_gemm_scratch_bytes(M, N, K, nbits)
    scratch = torch.empty(parts, dtype=torch.uint8, device=x.device) if parts else None
    _capi.check("gemq_linear_gemm", _capi.lib.gemq_linear_gemm(
        x.data_ptr(), None, w_q.data_ptr(), scales.data_ptr(), zeros.data_ptr(), None, None, None, nbits,
        bias.data_ptr() if bias is not None else None, out.data_ptr(), M, N, K, group_size, int(x.dtype == torch.bfloat16),
        error_word(x.device).data_ptr(), scratch.data_ptr() if parts else None, parts, stream_ptr(x.device)))
    return out


@library_op("dequant_gemm", _fake_gemm, lambda *a: host_linear(*a, None, 3) if len(a) == 6 else None)
def dequant_gemm(x: Tensor, w_q: Tensor, scales: Tensor, zeros: Tensor, nbits: int, group_size: int) -> Tensor:
    """``output[M, N] = x[M, K] @ dequantize(w_q, scales, zeros)``, fp16
    (gemq/triton_kernels/dequant_gemm.py:150-193).  32 rows or more go to the tcgen05 GEMM when
    N % 32 == 0 and K % 64 == 0; otherwise rows are processed by the decode
    kernel, in calls of at most 64 rows to bound the split-K workspace."""
    require(x.dim() == 2, "x must be [M, K]")
    M, K = x.shape
    N = w_q.shape[1]
    if tc_gemm_ok(M, N, K, group_size) and x.dtype in (torch.float16, torch.bfloat16):
        require_cuda(x, w_q, scales, zeros)
        check_kernel_form(w_q, scales, zeros, K, N, nbits, group_size)
        return _gemm_tc(x, w_q, scales, zeros, nbits, group_size, None)
    rows = dequant_gemv_rows._init_fn  # the plain function behind the operator
    if M <= _ROW_BLOCK:
        return rows(x, w_q, scales, zeros, nbits, group_size)
    return torch.cat([rows(x[i:i + _ROW_BLOCK], w_q, scales, zeros, nbits, group_size)
                      for i in range(0, M, _ROW_BLOCK)])


@library_op("quant_linear",
            lambda x, w_q, scales, zeros, nbits, group_size, bias: x.new_empty((x.shape[0], w_q.shape[1])),
            lambda *a: host_linear(*a, 0) if len(a) == 7 else None)
def quant_linear(x: Tensor, w_q: Tensor, scales: Tensor, zeros: Tensor, nbits: int, group_size: int,
                 bias: Optional[Tensor]) -> Tensor:
    """``x [M, K] @ deq(w_q) + bias`` in x's dtype (fp16 or bf16): what ``QuantLinear`` computes, in one call
    of the tcgen05 GEMM or of the few-row kernel, whichever is estimated the faster; either reads x and writes
    y in their own dtype."""
    dev = require_cuda(x, w_q, scales, zeros)
    M, K = x.shape
    N = w_q.shape[1]
    half = x.dtype in (torch.float16, torch.bfloat16)
    few = few_rows_ok(w_q, scales, zeros, K, N, group_size) and not (x.dtype == torch.float16 and one_row_streams(M, N, K))
    tc = bool(_capi.lib.gemq_linear_takes_gemm(M, N, K, nbits)) if few else tc_gemm_ok(M, N, K, group_size)
    if half and (tc or few):
        check_kernel_form(w_q, scales, zeros, K, N, nbits, group_size)
        if bias is not None:
            bias = bias.to(device=dev, dtype=x.dtype).contiguous()
        if tc:
            return _gemm_tc(x, w_q, scales, zeros, nbits, group_size, bias)
        return linear_rows(x if x.stride(1) == 1 else x.contiguous(), w_q, scales, zeros, nbits, group_size, bias)
    small = M < 32 and x.dtype != torch.float16
    y = dequant_gemm._init_fn(x.to(torch.float16) if small else x, w_q, scales, zeros, nbits, group_size).to(x.dtype)
    return y if bias is None else y + bias.to(y.dtype)


dequant_gemm_triton = dequant_gemm
