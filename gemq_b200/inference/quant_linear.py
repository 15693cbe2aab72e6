"""A quantised ``nn.Linear`` replacement on the MoE kernels.

The reference quantises attention and dense-MLP linears to 4 bits (``--attn_wbits 4
--dense_wbits 4``, gemq/quantize.py:333-343) and runs them with gemlite's kernels
(gemq/inference/patch.py:71-79).  The same packed format goes through this library's few-row
kernel or its tcgen05 GEMM, whichever is estimated the faster for the rows, any bit width from 1 to 4.
"""
from __future__ import annotations

import torch
import torch.nn as nn
from torch import Tensor

from ..kernels._ops import plain_call
from ..kernels._runtime import host_linear
from ..kernels.dequant_gemm import quant_linear
from .packed_linear import PackedLinear


class QuantLinear(nn.Module):
    def __init__(self, packed: PackedLinear, bias: Tensor = None):
        super().__init__()
        self.in_features, self.out_features = packed.in_features, packed.out_features
        self.W_nbits, self.group_size = packed.W_nbits, packed.group_size
        # plain attributes, like the reference's blocks keep their packed tensors
        self.W_q, self.scales, self.zeros = packed.W_q, packed.scales, packed.zeros
        self.bias = bias

    def forward(self, x: Tensor) -> Tensor:
        """``x [..., in]`` fp16 / bf16 -> ``[..., out]`` in the same dtype."""
        w_q, scales, zeros, bias = self.W_q, self.scales, self.zeros, self.bias
        plain = plain_call(x, w_q, scales, zeros, bias)
        if plain:
            y = host_linear(x, w_q, scales, zeros, self.W_nbits, self.group_size, bias, 0)
            if y is not None:
                return y
        lead = x.shape[:-1]
        y = quant_linear(x.reshape(-1, self.in_features), w_q, scales, zeros, self.W_nbits, self.group_size, bias if plain else None)
        if bias is not None and not plain:  # the same value; the addition has a gradient, the operator has none
            y = y + bias.to(y.dtype)
        return y.reshape(*lead, self.out_features)
