"""Host-side plumbing shared by the op wrappers: argument checks, streams, workspace."""
from __future__ import annotations

import torch

from .. import _capi

_workspaces: dict = {}


def require_cuda(*tensors: torch.Tensor) -> torch.device:
    dev = None
    for t in tensors:
        if not isinstance(t, torch.Tensor):
            raise TypeError(f"expected a torch.Tensor, got {type(t).__name__}")
        if not t.is_cuda:
            raise RuntimeError("gemq_b200 ops run on CUDA tensors only (there is no CPU path)")
        if dev is None:
            dev = t.device
        elif t.device != dev:
            raise RuntimeError(f"tensors on different devices: {dev} and {t.device}")
    return dev


def require(cond: bool, msg: str) -> None:
    if not cond:
        raise ValueError(msg)


def stream_ptr(dev: torch.device) -> int:
    return torch.cuda.current_stream(dev).cuda_stream


def workspace(dev: torch.device, nbytes: int) -> torch.Tensor:
    """Zero-initialised uint8 scratch of at least ``nbytes`` on ``dev``.

    The arrival counters at its head are left at zero by every kernel, so the buffer is
    zeroed only when it is (re)allocated.  One buffer per device: calls that share it must
    be ordered on one stream.
    """
    key = (dev.type, dev.index if dev.index is not None else torch.cuda.current_device())
    ws = _workspaces.get(key)
    if ws is None or ws.numel() < nbytes:
        ws = torch.zeros(max(nbytes, 1 << 20), dtype=torch.uint8, device=dev)
        _workspaces[key] = ws
    return ws


def gemv_workspace(dev: torch.device, total_cols: int, max_k: int, tokens: int) -> torch.Tensor:
    return workspace(dev, _capi.lib.gemq_gemv_workspace_bytes(total_cols, max_k, tokens))


def check_kernel_form(wq, scales, zeros, K: int, N: int, nbits: int, group_size: int) -> None:
    require(nbits in (1, 2, 3, 4), f"unsupported bit-width {nbits}")
    require(wq.dtype == torch.int32 and wq.is_contiguous(), "w_q must be contiguous int32 [ceil(K/eps), N]")
    eps = 32 // nbits
    require(tuple(wq.shape) == (-(-K // eps), N), f"w_q shape {tuple(wq.shape)} != {(-(-K // eps), N)}")
    require(K % group_size == 0, "K must be a multiple of group_size")
    for name, t in (("scales", scales), ("zeros", zeros)):
        require(t.dtype == torch.float16 and t.is_contiguous(), f"{name} must be contiguous float16")
        require(tuple(t.shape) == (K // group_size, N), f"{name} shape {tuple(t.shape)} != {(K // group_size, N)}")


_err_words: dict = {}


def error_word(dev: torch.device) -> torch.Tensor:
    """One int32 per device that kernels with bounded waits set when a wait expires."""
    key = (dev.type, dev.index if dev.index is not None else torch.cuda.current_device())
    t = _err_words.get(key)
    if t is None:
        t = torch.zeros(1, dtype=torch.int32, device=dev)
        _err_words[key] = t
    return t


_err_ptrs: dict = {}


def host_linear(x, w_q, scales, zeros, nbits, group_size, bias, mode: int):
    """The native call (csrc/host.cpp) or None.  ``mode``: 0 dense layer, 1 rows operator, 2 one-row operator,
    3 GEMM operator."""
    i = x.get_device()
    p = _err_ptrs.get(i)
    if p is None:
        if i < 0:
            return None
        p = _err_ptrs[i] = error_word(x.device).data_ptr()
    return _capi.host.linear(x, w_q, scales, zeros, nbits, group_size, bias, p, mode)


def tc_gemm_ok(M: int, N: int, K: int, group_size: int) -> bool:
    """Shapes the tcgen05 GEMM takes; smaller row counts stay on the decode kernel."""
    return M >= 32 and N % 32 == 0 and K % 64 == 0 and group_size % 64 == 0 and K % group_size == 0


def one_row_streams(M: int, N: int, K: int) -> bool:
    """One row of a matrix that the split-K streaming kernel takes in less time than the few-row kernel."""
    return M == 1 and bool(_capi.lib.gemq_one_row_streams(N, K))


def few_rows_ok(w_q, scales, zeros, K: int, N: int, group_size: int) -> bool:
    """Matrices the few-row kernel takes (``gemq_linear_rows``)."""
    return (group_size == 128 and K % 128 == 0 and K <= 32768 and N % 32 == 0 and
            (w_q.data_ptr() | scales.data_ptr() | zeros.data_ptr()) & 15 == 0)


def linear_rows(x, w_q, scales, zeros, nbits: int, group_size: int, bias=None):
    """``x [M, K] @ deq(w_q) (+ bias)`` in x's dtype (fp16 or bf16) through the few-row kernel; the
    arguments have been checked."""
    dev = x.device
    M, K = x.shape
    N = w_q.shape[1]
    out = torch.empty((M, N), dtype=x.dtype, device=dev)
    _capi.check("gemq_linear_rows", _capi.lib.gemq_linear_rows(
        x.data_ptr(), x.stride(0), int(x.dtype == torch.bfloat16), w_q.data_ptr(), scales.data_ptr(), zeros.data_ptr(),
        bias.data_ptr() if bias is not None else None, out.data_ptr(), M, N, K, nbits, group_size,
        error_word(dev).data_ptr(), stream_ptr(dev)))
    return out
