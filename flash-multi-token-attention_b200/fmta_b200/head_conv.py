"""Head-mixing attention API, mirroring the reference's ``head_conv_attn`` package
(``head_conv_attn.py:11-116`` and the host functions of ``fwd_kernel.py:282``,
``bwd_dq_dw.py:373``, ``bwd_dk_dv.py:407``), plus the composed "key-query conv then grouped
head mix" operator of the head-mixing training configuration.

Groups of 2 to 16 heads at head dim 64 or 128 run on the tensor-core kernels (csrc/mix_tc.cuh).  Short
sequences, which the others finish sooner, and what those do not take -- 32 heads (without a conv, up to head dim 64), head
dim 32, little memory -- run on kernels that keep all heads of a group in one CTA or, behind a conv (there also more than seven
query taps), one head per CTA of a cluster, exchanging score tiles.  A dense [H,H] matrix is the single-group case G = H; grouped
mixing takes ``w`` as [H/G, G, G].
"""
import math
import os

import torch
import torch.nn as nn

from . import _native
from .conv_attn import _keep_limit


# What a head mix may take for itself.  On the tensor cores that is the scores' operands P and dC (4.5 GiB of them, or one
# group's, at a time) and, with a filter, the stacked keys; the kernels for the rest exchange the heads' score tiles through a
# global scratch (up to 4 GiB) instead of the cluster's shared memory.  FMTA_MIX_EXCHANGE_LIMIT_GB (here: this switch, in bytes)
# bounds either: fewer groups at a time, then the kernels without such buffers.  So does what the GPU has left.
_LIMIT_GB = os.environ.get("FMTA_MIX_EXCHANGE_LIMIT_GB")
MIX_EXCHANGE_LIMIT_BYTES = None if _LIMIT_GB is None else int(float(_LIMIT_GB) * (1 << 30))


def _limits():
    if MIX_EXCHANGE_LIMIT_BYTES is None:
        return 4 << 30, (1 << 63) - 1
    return MIX_EXCHANGE_LIMIT_BYTES, MIX_EXCHANGE_LIMIT_BYTES


def conv_headmix_forward(q, k, v, w, conv_kernel=None, scale=1.0, causal=False, out_dtype=None):
    """(o, l, m, lse): o in ``out_dtype`` (default: dtype of q), l = sum exp, m = max, fp32 [B,H,N]."""
    return _native.mix_forward(q, k, v, w, conv_kernel, scale, bool(causal), out_dtype, _limits())


def head_conv_attention_forward(q, k, v, w, scale=1.0, causal=False):
    """(o, l, m) -- fwd_kernel.py:282-364."""
    o, l, m, _ = conv_headmix_forward(q, k, v, w, None, scale, causal)
    return o, l, m


def _backward(q, k, v, w, o, do, l, m, conv_kernel, causal, scale, lse, want):
    return _native.mix_backward(q, k, v, w, o, do, l, m, conv_kernel, bool(causal), scale, lse, want, _limits())


def conv_headmix_bwd_dq_dw(q, k, v, w, o, do, l, m, conv_kernel=None, causal=False, scale=None):
    """(dq fp32, dw fp32 shaped like w, dtheta fp32 or None)."""
    g = _backward(q, k, v, w, o, do, l, m, conv_kernel, causal, scale, None, 1)
    return g[0], g[3], g[4]


def conv_headmix_bwd_dkdv(q, k, v, w, o, do, l, m, conv_kernel=None, causal=False, scale=None):
    """(dk fp32, dv fp32)."""
    g = _backward(q, k, v, w, o, do, l, m, conv_kernel, causal, scale, None, 2)
    return g[1], g[2]


def conv_headmix_backward(q, k, v, w, o, do, l, m, conv_kernel=None, causal=False, scale=None, lse=None):
    """(dq, dk, dv, dw shaped like w, dtheta or None), all fp32, from ONE call of the fused backward entry
    point: D = rowsum(dO * O) and the log-sum-exp are prepared once for both halves (the two host functions
    above, which mirror the reference's pair of calls, each prepare them again)."""
    return tuple(_backward(q, k, v, w, o, do, l, m, conv_kernel, causal, scale, lse, 3))


def head_conv_attention_bwd_dq_dw(q, k, v, w, o, do, l, m, causal=False, scale=None):
    """(dq in q's dtype, dw) -- bwd_dq_dw.py:373-460."""
    dq, dw, _ = conv_headmix_bwd_dq_dw(q, k, v, w, o, do, l, m, None, causal, scale)
    return dq.to(q.dtype), dw.to(w.dtype)


def head_conv_attention_bwd_dkdv(q, k, v, w, o, do, l, m, causal=False, scale=None):
    """(dk, dv) in the input dtypes -- bwd_dk_dv.py:407-485."""
    dk, dv = conv_headmix_bwd_dkdv(q, k, v, w, o, do, l, m, None, causal, scale)
    return dk.to(k.dtype), dv.to(v.dtype)


class HeadConvAttentionFunction(torch.autograd.Function):
    """Same argument list of ``apply`` as head_conv_attn.py:11-63; the autograd node is native (csrc_torch/fmta_torch.cpp),
    except under ``torch.jit.trace`` (see FlashConvAttentionCUDAFunction)."""

    @staticmethod
    def apply(q, k, v, w, causal=False, scale=None):
        if scale is None:
            scale = 1.0 / math.sqrt(q.shape[-1])
        if torch.jit.is_tracing():
            return super(HeadConvAttentionFunction, HeadConvAttentionFunction).apply(q, k, v, w, causal, scale)
        return _native.mix_attention(q, k, v, None, w, scale, bool(causal), False, _limits(), 0)

    @staticmethod
    def forward(ctx, q, k, v, w, causal, scale):
        o, l, m = head_conv_attention_forward(q, k, v, w, scale=scale, causal=causal)
        ctx.save_for_backward(q, k, v, w, o, l, m)
        ctx.causal, ctx.scale = causal, scale
        return o

    @staticmethod
    def backward(ctx, do):
        q, k, v, w, o, l, m = ctx.saved_tensors
        dq, dk, dv, dw, _ = conv_headmix_backward(q, k, v, w, o, do, l, m, None, ctx.causal, ctx.scale)
        return dq.to(q.dtype), dk.to(k.dtype), dv.to(v.dtype), dw.to(w.dtype), None, None


class HeadConvAttention(nn.Module):
    """Drop-in for head_conv_attn.py:66-98 (parameter ``head_conv_weights`` [H,H])."""

    def __init__(self, n_heads, dtype=torch.float16):
        super().__init__()
        self.n_heads = n_heads
        self.dtype = dtype
        self.head_conv_weights = nn.Parameter(torch.randn(n_heads, n_heads, dtype=dtype) / math.sqrt(n_heads))

    def forward(self, q, k, v, causal=False, scale=None):
        return HeadConvAttentionFunction.apply(q, k, v, self.head_conv_weights, causal, scale)


def head_conv_attention(q, k, v, w, causal=False, scale=None):
    """Functional form (head_conv_attn.py:101-116)."""
    return HeadConvAttentionFunction.apply(q, k, v, w, causal, scale)


class ConvHeadMixFunction(torch.autograd.Function):
    """Key-query conv followed by a grouped head mix (w [H/G,G,G]), then softmax and PV; fp32 output."""

    @staticmethod
    def apply(q, k, v, conv_kernel, w, causal, scale):
        if torch.jit.is_tracing():
            return super(ConvHeadMixFunction, ConvHeadMixFunction).apply(q, k, v, conv_kernel, w, causal, scale)
        return _native.mix_attention(q, k, v, conv_kernel, w, scale, bool(causal), True, _limits(), _keep_limit())

    @staticmethod
    def forward(ctx, q, k, v, conv_kernel, w, causal, scale):
        o, l, m, lse = conv_headmix_forward(q, k, v, w, conv_kernel, scale, causal, out_dtype=torch.float32)
        ctx.save_for_backward(q, k, v, conv_kernel, w, o, l, m, lse)
        ctx.causal, ctx.scale = causal, scale
        return o

    @staticmethod
    def backward(ctx, do):
        q, k, v, conv_kernel, w, o, l, m, lse = ctx.saved_tensors
        dq, dk, dv, dw, dth = conv_headmix_backward(q, k, v, w, o, do, l, m, conv_kernel, ctx.causal, ctx.scale, lse=lse)
        return dq.to(q.dtype), dk.to(k.dtype), dv.to(v.dtype), dth.to(conv_kernel.dtype), dw.to(w.dtype), None, None


def conv_headmix_attention(q, k, v, conv_kernel, w, causal=True, scale=None):
    if scale is None:
        scale = 1.0 / math.sqrt(q.shape[-1])
    return ConvHeadMixFunction.apply(q, k, v, conv_kernel, w, causal, scale)
