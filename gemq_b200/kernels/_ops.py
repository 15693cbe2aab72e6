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

NAMESPACE = "gemq_b200"


def plain_call(x) -> bool:
    """No compiler and no tracing mode is active and ``x`` is an ordinary tensor: nobody but the
    caller looks at this call, so the operator registry has nothing to add to it."""
    return (not torch.compiler.is_compiling() and torch._C._len_torch_dispatch_stack() == 0 and
            type(x) in (torch.Tensor, torch.nn.Parameter))


def library_op(name: str, fake, fast=None):
    """``@library_op("name", fake_fn)``: register ``fn`` as ``gemq_b200::name`` (no argument is
    mutated, outputs are fresh tensors) with ``fake_fn`` as its shape/dtype propagation.

    A call in eager mode goes straight to ``fn``: the Python dispatch of a custom operator costs
    20-30 us of host time, more than the kernels of a small call take.  ``fast`` is tried before it with the
    positional arguments: native code that returns None for what it does not take.  Under ``torch.compile`` and
    under tracing modes (fake tensors) the call is the operator."""
    def deco(fn):
        op = torch.library.custom_op(f"{NAMESPACE}::{name}", mutates_args=())(fn)
        op.register_fake(fake)
        overload = op._opoverload

        @functools.wraps(fn)
        def call(*args, **kwargs):
            if not args or not plain_call(args[0]):
                return overload(*args, **kwargs)
            if fast is not None and not kwargs:
                y = fast(*args)
                if y is not None:
                    return y
            return fn(*args, **kwargs)

        call._init_fn = fn
        return call
    return deco
