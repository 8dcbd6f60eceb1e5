"""Causal depthwise short convolution whose leading channels get SiLU: `conv_split_act_call`.

Same call, shapes, dtypes and packed-row semantics as the reference's cute_triadic_gdn/ops/conv_split_act.py:194-197
(conv_split_act_call) with its custom ops :143-173 and autograd glue :176-191; the device work is the CUDA library's
tgdn_conv_fwd / tgdn_conv_bwd instead of Triton kernels, the operators, their checks and their autograd are native
(csrc/tgdn_torch.cpp).
"""
from __future__ import annotations

import torch

from . import _lib


@torch.library.register_fake("tgdn_b200::conv_split_act_fwd")
def _conv_fwd_fake(x, weight, act_channels, cu_seqlens=None):
    return torch.empty_like(x, memory_format=torch.contiguous_format)


@torch.library.register_fake("tgdn_b200::conv_split_act_bwd")
def _conv_bwd_fake(x, dy, weight, act_channels, cu_seqlens=None):
    return torch.empty_like(x, memory_format=torch.contiguous_format), torch.empty_like(weight)


conv_split_act_fwd = torch.ops.tgdn_b200.conv_split_act_fwd
conv_split_act_bwd = torch.ops.tgdn_b200.conv_split_act_bwd


def conv_split_act_call(x, weight, act_channels, cu_seqlens=None):
    """Width-4 causal depthwise convolution over (B, T, C) bf16 `x` with taps `weight` (C, 4); the first `act_channels`
    channels pass through SiLU.  With `cu_seqlens` (offsets of the documents of one packed row, B = 1) the window starts
    afresh at every document.  Same call as the reference's conv_split_act_call (ops/conv_split_act.py:194-197)."""
    if not torch.compiler.is_compiling():
        return _lib.host.conv_call(x, weight, int(act_channels), cu_seqlens)
    return conv_split_act_fwd(x, weight.contiguous(), int(act_channels), cu_seqlens)


# ----------------------------------------------------------------------------------------------------------------------
# The layer glue fused into the convolution (beyond the reference's surface; it describes the glue at
# cute_triadic_gdn/ops/conv_split_act.py:3-5 and leaves it to its caller)
# ----------------------------------------------------------------------------------------------------------------------
@torch.library.register_fake("tgdn_b200::conv_split_norm_fwd")
def _norm_fwd_fake(x, weight, heads, slices, eps, cu_seqlens=None):
    B, T, _ = x.shape
    qkv = [x.new_empty((B, T, heads, 128)) for _ in range(3)]
    gates = [x.new_empty((B, T, heads, slices), dtype=torch.float32) for _ in range(2)]
    return (*qkv, *gates)


@torch.library.register_fake("tgdn_b200::conv_split_norm_bwd")
def _norm_bwd_fake(x, weight, dq, dk, dv, dk2, dq2, heads, slices, eps, cu_seqlens=None):
    return torch.empty_like(x, memory_format=torch.contiguous_format), torch.empty_like(weight)


conv_split_norm_fwd = torch.ops.tgdn_b200.conv_split_norm_fwd
conv_split_norm_bwd = torch.ops.tgdn_b200.conv_split_norm_bwd


def conv_split_norm_call(x, weight, heads, slices, cu_seqlens=None, eps=1e-6):
    """The convolution pre-pass with the layer glue fused in: x (B, T, C) bf16 with C = heads*(3*128 + 2*slices) channels
    laid out [q | k | v | k2 | q2] goes straight to what `gdn_joint_call` takes,

        q, k = l2norm(SiLU(conv(x)))  bf16 (B, T, heads, 128)      v = SiLU(conv(x))  bf16 (B, T, heads, 128)
        k2, q2 = l2norm(softplus(conv(x)))  f32 (B, T, heads, slices),     l2norm(s) = s * rsqrt(sum s^2 + eps),

    without the convolution's output ever being written.  Differentiable in x and weight; packed rows as in
    `conv_split_act_call`."""
    if not torch.compiler.is_compiling():
        return _lib.host.conv_norm_call(x, weight, int(heads), int(slices), float(eps), cu_seqlens)
    return conv_split_norm_fwd(x, weight.contiguous(), int(heads), int(slices), float(eps), cu_seqlens)
