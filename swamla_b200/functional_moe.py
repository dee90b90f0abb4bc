"""The non-latent ``MoELayer`` of Orolol/swamla (``models/moe.py:294-559``) on the same sm_100a kernels.

Same routing, grouped GEMMs and row kernels as the latent layer, with the experts working at the model width:
there is no down/up projection, ``x`` itself is gathered into the padded expert layout and the weighted sum of the
expert outputs is added to the shared expert's output (``moe.py:366``).  The native host path (``csrc/torch_host.cpp``)
issues the generic entry points of ``include/lmoe.h``; no CPU fallback.
"""
from __future__ import annotations

import torch

from . import _testing, functional


def moe(x: torch.Tensor, w_gate, w_gate_up_s, w_down_s, w_gate_up, w_down_e, expert_bias, top_k: int, z_coef: float,
        evaluation: bool = False):
    """Functional form on a [..., D] activation.  Returns (y like x, aux_loss scalar, sel [T,K] int32, counts [E] int32);
    (y, aux_loss) only where ``evaluation`` takes the few-token path (see ``functional.latent_moe``)."""
    forced = _testing.FORCE_SEL
    if forced is not None:
        forced = forced.to(device=x.device, dtype=torch.int32).contiguous()
    return functional._host().moe(x, w_gate, w_gate_up_s, w_down_s, w_gate_up, w_down_e, expert_bias, top_k, z_coef, forced,
                                  evaluation)


# opaque to torch.compile: the layer runs as an eager call between compiled regions
moe_opaque = torch.compiler.disable(moe)
