"""Rotary position embedding of the query and key projections as one kernel, forward and backward
(csrc/rotary.cu): what models.apply_rotary does with torch operations on bf16 projections that an
attention kernel reads in bf16 (nvfp4_train.py:91-98)."""
from __future__ import annotations

import torch

from . import _lib
from .quant import _stream


class RotaryFn(torch.autograd.Function):
    """(q [B, T, Hq, D], k [B, T, Hk, D], cos, sin [T, D / 2]) -> both rotated, bf16, same layout.  transposed: by the
    transposed rotation.  The operation is linear and its gradient is the other of the two, so it can be differentiated
    any number of times."""

    @staticmethod
    def forward(ctx, q, k, cos, sin, transposed):
        ctx.save_for_backward(cos, sin)
        ctx.transposed = transposed
        return _rotate(q, k, cos, sin, transposed)

    @staticmethod
    def backward(ctx, gq, gk):
        args = gq.to(torch.bfloat16), gk.to(torch.bfloat16), *ctx.saved_tensors, not ctx.transposed
        gq, gk = RotaryFn.apply(*args) if torch.is_grad_enabled() else _rotate(*args)
        return gq, gk, None, None, None


def _rotate(q, k, cos, sin, transposed):
    q, k = _rows(q), _rows(k)
    dev = _lib.cuda_device_of(q, k, cos, sin)
    B, T, hq, D = q.shape
    qo, ko = torch.empty_like(q), torch.empty_like(k)
    with torch.cuda.device(dev):                   # the C side launches on the current device
        code = _lib.lib().nvfp4_rotary_bf16(q.data_ptr(), qo.data_ptr(), hq, k.data_ptr(), ko.data_ptr(), k.shape[2], B * T,
                                            T, D, cos.data_ptr(), sin.data_ptr(), int(transposed), _stream(dev))
    _lib.check(code, "nvfp4_rotary_bf16")
    return qo, ko


def _rows(t):
    t = t.contiguous()
    return t if t.data_ptr() % 16 == 0 else t.clone()


def takes(q, k, cos, sin):
    """Does the kernel stand for the torch operations here?  They promote bf16 projections to the fp32 of the tables, and
    autocast rounds the result to bf16 in front of the attention: one rounding, as in the kernel.  Without autocast, or
    with another dtype, the attention would see fp32, so those calls keep the torch operations."""
    return (q.is_cuda and q.dtype == torch.bfloat16 and k.dtype == torch.bfloat16 and q.numel() > 0 and q.shape[-1] % 16 == 0
            and torch.is_autocast_enabled("cuda") and torch.get_autocast_dtype("cuda") == torch.bfloat16
            and all(t.dtype == torch.float32 and t.device == q.device and not t.requires_grad
                    and tuple(t.shape) == (1, 1, q.shape[1], q.shape[-1] // 2) for t in (cos, sin)))


def rotary(q, k, cos, sin):
    """q [B, T, Hq, D] and k [B, T, Hk, D] rotated by the tables [1, 1, T, D / 2]."""
    T, half = cos.shape[2:]
    return RotaryFn.apply(q, k, _rows(cos.reshape(T, half)), _rows(sin.reshape(T, half)), False)
