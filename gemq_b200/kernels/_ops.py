"""Registration of the library calls as ``torch.library`` custom operators.

The reference runs its decode step under ``torch.compile(mode="reduce-overhead",
fullgraph=True)`` (gemq/benchmark_generate.py:158-160).  A ctypes call is opaque to dynamo, so
every public op is a custom operator with a fake (meta) implementation: tracing sees an
operator with known output shapes and dtypes, and the real implementation -- argument checks
plus the C-ABI call on the current stream -- runs at execution (and CUDA-graph capture) time.
"""
from __future__ import annotations

import functools

import torch
from torch.autograd import forward_ad
from torch.utils._device import DeviceContext

from .. import _capi

NAMESPACE = "gemq_b200"
_len_function_stack, _function_mode = torch._C._len_torch_function_stack, torch._C._get_function_stack_at
_len_dispatch_stack = torch._C._len_torch_dispatch_stack
_functorch_level = torch._C._functorch.peek_interpreter_stack
_tracing_state = torch._C._get_tracing_state


def plain_call(*args) -> bool:
    """Nobody but the caller looks at this call, so the operator registry has nothing to add to it: no compiler, tracer,
    dispatch or function mode (but for a default device) and no function transform is active, the tensors among the
    arguments are ordinary ones, and none of them asks for a gradient, which the operators refuse."""
    if torch.compiler.is_compiling():
        return False
    return bool(_capi.host.plain(*args)) or _plain(args)  # the native form is the fast yes: here these checks take 1 us


def _plain(args) -> bool:
    if _len_dispatch_stack() or _functorch_level() is not None or _tracing_state() is not None:
        return False
    n = _len_function_stack()
    if n and not all(type(_function_mode(i)) is DeviceContext for i in range(n)):
        return False
    grad = torch.is_grad_enabled()
    dual = forward_ad._current_level >= 0
    for a in args:
        if isinstance(a, torch.Tensor) and (type(a) not in (torch.Tensor, torch.nn.Parameter) or (grad and a.requires_grad) or
                                            (dual and forward_ad.unpack_dual(a).tangent is not None)):
            return False
    return True


def library_op(name: str, fake, fast=None):
    """``@library_op("name", fake_fn)``: register ``fn`` as ``gemq_b200::name`` (no argument is
    mutated, outputs are fresh tensors) with ``fake_fn`` as its shape/dtype propagation.

    A call in eager mode goes straight to ``fn``: the Python dispatch of a custom operator costs
    20-30 us of host time, more than the kernels of a small call take.  ``fast`` is tried before it with the
    positional arguments: native code that returns None for what it does not take.  Every other call
    (``plain_call``) is the operator."""
    def deco(fn):
        op = torch.library.custom_op(f"{NAMESPACE}::{name}", mutates_args=())(fn)
        op.register_fake(fake)
        overload = op._opoverload

        @functools.wraps(fn)
        def call(*args, **kwargs):
            if not plain_call(*args, *kwargs.values()):
                return overload(*args, **kwargs)
            if fast is not None and not kwargs:
                y = fast(*args)
                if y is not None:
                    return y
            return fn(*args, **kwargs)

        call._init_fn = fn
        for method in ("register_autograd", "register_fake", "register_kernel", "register_vmap"):
            setattr(call, method, getattr(op, method))
        return call
    return deco
