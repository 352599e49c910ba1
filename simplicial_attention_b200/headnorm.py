"""Per-head RMSNorm of a packed projection in one kernel (forward and backward).

The reference normalises q, k, k', v, v' with five ``RMSNorm(dim_head)`` modules
after splitting its fused projection (simplicial_attention/simplicial_mha.py:69-73,
124-127).  ``head_rmsnorm`` does the same arithmetic on the projection as a whole:
``x`` is ``(..., channels)``, every ``d`` consecutive channels are one head and
``weight`` holds one gain per channel.  The CUDA kernels sit behind the C ABI
(``sa2_headnorm_fwd`` / ``sa2_headnorm_bwd`` in ``include/sa2.h``); the autograd node is native
(``csrc/sa2_torch.cpp``).
"""
from __future__ import annotations

import torch

from . import _lib

_DTYPES = {torch.float32: _lib.SA2_F32, torch.bfloat16: _lib.SA2_BF16}


def head_rmsnorm(x, weight, d, eps, out_dtype=None):
    """``y[..., c] = x[..., c] * rsqrt(mean over c's head of x^2 + eps) * weight[c]``; ``weight`` has one
    entry per channel.  ``out_dtype`` defaults to ``x.dtype``."""
    out_dtype = x.dtype if out_dtype is None else out_dtype
    assert x.is_cuda and x.dtype in _DTYPES and out_dtype in _DTYPES
    y = _lib.ext().headnorm(x, weight, int(d), float(eps), out_dtype)
    if y is not None:
        return y
    # torch is recording or transforming the computation (the native call says when): the same arithmetic in its operators
    heads = x.float().unflatten(-1, (-1, int(d)))
    y = (heads * torch.rsqrt(heads.square().mean(-1, keepdim=True) + float(eps))).flatten(-2)
    return (y * weight.float()).to(out_dtype)


class RMSNorm(torch.nn.Module):
    """``torch.nn.RMSNorm(dim)`` with the same parameter (``weight``) and arithmetic, run by the fused kernel
    on CUDA when ``dim`` is 32 ... 512 (a power of two times 32); under autocast the result is produced in
    the autocast dtype directly - its consumers here are linear layers, which would round it anyway."""

    def __init__(self, dim, eps=None):
        super().__init__()
        self.dim, self.eps = dim, eps
        self.weight = torch.nn.Parameter(torch.ones(dim))

    def forward(self, x):
        fused = x.is_cuda and self.dim in (32, 64, 128, 256, 512) and x.dtype in _DTYPES
        if not fused:
            return torch.nn.functional.rms_norm(x, (self.dim,), self.weight, self.eps)
        autocast = torch.is_autocast_enabled()
        eps = self.eps if self.eps is not None else torch.finfo(torch.float32 if autocast else x.dtype).eps
        out_dtype = torch.get_autocast_dtype("cuda") if autocast else x.dtype
        if out_dtype not in _DTYPES:
            out_dtype = x.dtype
        return head_rmsnorm(x, self.weight, self.dim, eps, out_dtype)
