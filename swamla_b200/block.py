"""``x + ffn(ffn_norm(x))``: the feed-forward half of the reference's block (``models/mla_block.py:83-85, 159``) with
the RMSNorm (``models/normalization.py:25-39``) and the residual add as fused row kernels of ``liblmoe.so``.

``NormedResidualFFN(ffn, dim, eps)`` owns the norm weight under the reference's name (``ffn_norm.weight``) and wraps any
feed-forward module (here: ``LatentMoELayer`` / ``MoELayer``).  Forward: one kernel for the norm (one read of x, one
write), the layer, one kernel for the add.  Backward: ONE kernel for the adjoint of the norm and the residual branch
(``dx = norm_bwd(d_xn) + dy``), plus a deterministic two-stage sum for the weight gradient.  The residual stream keeps the
input's dtype: under the reference's autocast training it is fp32 (train.py:1195, normalization.py:25-39) and the residual
branch is never rounded to bf16 (the norm's input is, as it is read).  The autograd nodes are in ``csrc/torch_host.cpp``.  No CPU fallback.
"""
from __future__ import annotations

import torch
import torch.nn as nn

from .functional import _host
from .layer import LatentMoELayer, MoELayer, _drops, _hooked


class _NormAndPass:
    """``apply(x, weight, eps)`` -> (rmsnorm(x) * weight, x), both in x's dtype (a differentiable call)."""

    @staticmethod
    def apply(x, weight, eps: float):
        return tuple(_host().norm_and_pass(x, weight, float(eps), False))


class _NormWeight(nn.Module):
    """Holds ``weight`` [dim] (ones at init) under the reference's parameter name ``ffn_norm.weight``."""

    def __init__(self, dim: int, eps: float):
        super().__init__()
        self.eps = eps
        self.weight = nn.Parameter(torch.ones(dim))


class NormedResidualFFN(nn.Module):
    """``forward(x) = x + ffn(rmsnorm(x))`` for x[B, S, D]; output dtype = input dtype, arithmetic bf16/fp32.
    ``state_dict`` keys: ``ffn_norm.weight`` and ``ffn.*`` as in the reference block."""

    def __init__(self, ffn: nn.Module, dim: int, eps: float = 1e-6):
        super().__init__()
        if dim % 8 or dim > 2048:
            raise ValueError("kernel constraints: dim a multiple of 8, at most 2048")
        self.ffn_norm = _NormWeight(dim, eps)
        self.ffn = ffn

    def forward(self, x: torch.Tensor) -> torch.Tensor:
        _B, _S, _D = x.shape
        norm, ffn = self.ffn_norm, self.ffn
        if torch.compiler.is_compiling():
            xn, x_pass = _norm_opaque(x, norm.weight, norm.eps)
            return _add_opaque(x_pass, ffn(xn))
        host = _host()
        xn, x_pass = host.norm_and_pass(x, norm.weight, norm.eps, _takes_bf16(ffn))
        return host.residual_add(x_pass, ffn(xn))


def _takes_bf16(ffn) -> bool:
    """Whether the feed-forward module is handed bf16 and gives bf16 back, instead of a widened copy each way: this package's
    own layers compute in bf16 whatever they are given.  Not where something else sees or changes the tensors in the stream's
    precision: an active dropout, a hook, a replaced ``forward``."""
    return type(ffn) in (LatentMoELayer, MoELayer) and "forward" not in ffn.__dict__ and not _hooked(ffn) and not _drops(ffn.dropout)


# opaque to torch.compile (calls into the kernel library); the feed-forward module between them is compiled
@torch.compiler.disable
def _norm_opaque(x, weight, eps):
    return _NormAndPass.apply(x, weight, eps)


@torch.compiler.disable
def _add_opaque(a, b):
    return _host().residual_add(a, b)
