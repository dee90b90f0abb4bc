"""``torch.library`` custom operators around the LatentMoE path, so that ``torch.compile`` keeps ONE graph across the
layer (the reference compiles the whole model by default, ``train.py:936-942``).

Two opaque operators, ``swamla_b200::latent_moe_fwd`` and ``swamla_b200::latent_moe_bwd``, each with a fake (shape-only)
implementation for tracing, tied together with ``register_autograd``.  Their real implementations are the two directions
of the native host path that the eager call runs too.  A third, ``swamla_b200::latent_moe_eval``, is the evaluated layer
without gradients, whose eager call may take the few-token kernels and keeps nothing for a backward.  So compiled and eager
execution give the same bits in every mode, and launch the same kernels but for a training-mode forward without gradients,
which keeps what a backward would read.

An operator's outputs may alias neither its inputs nor one another, so the forward operator returns only tensors it
creates (what the backward needs travels as one allocation) and the backward operator takes the layer's inputs
again and re-derives the bf16 operands from them (a no-op for a bf16 module).

Covers the single-GPU bf16 layer; FP8 experts and the expert-parallel modes stay opaque eager calls
(``torch.compiler.disable``) because they keep Python-side state (collectives, symmetric buffers, scale caches).
"""
from __future__ import annotations

import os
from typing import Optional, Tuple

import torch
from torch import Tensor

from . import functional as Fn


def _dims(x: Tensor, w_gate_up: Tensor, w_down_s: Tensor, top_k: int):
    T, D = x.shape
    E, L, F2 = w_gate_up.shape
    return T, D, L, E, int(top_k), F2 // 2, w_down_s.shape[1]


@torch.library.custom_op("swamla_b200::latent_moe_fwd", mutates_args=())
def latent_moe_fwd(x: Tensor, w_gate: Tensor, w_down: Tensor, w_up: Tensor, w_gate_up_s: Tensor, w_down_s: Tensor,
                   w_gate_up: Tensor, w_down_e: Tensor, expert_bias: Tensor, top_k: int, z_coef: float
                   ) -> Tuple[Tensor, Tensor, Tensor, Tensor, Tensor]:
    if os.environ.get("LMOE_TMA_GATHER", "0") == "1":
        raise RuntimeError("LMOE_TMA_GATHER is not available under torch.compile")
    y, z_loss, sel, counts, saved, _ = Fn._host().latent_fwd_raw(x, w_gate, w_down, w_up, w_gate_up_s, w_down_s, w_gate_up,
                                                                 w_down_e, expert_bias, top_k, z_coef, False, None, False)
    return y, z_loss, sel, counts, saved


@latent_moe_fwd.register_fake
def _(x, w_gate, w_down, w_up, w_gate_up_s, w_down_s, w_gate_up, w_down_e, expert_bias, top_k, z_coef):
    T, D, L, E, K, F, Fs = _dims(x, w_gate_up, w_down_s, top_k)
    new = lambda *shape, dtype: x.new_empty(shape, dtype=dtype)
    return (new(T, D, dtype=x.dtype), new(dtype=torch.float32), new(T, K, dtype=torch.int32), new(E, dtype=torch.int32),
            new(Fn.saved_bytes(T, D, L, E, K, F, Fs), dtype=torch.uint8))


@torch.library.custom_op("swamla_b200::latent_moe_bwd", mutates_args=())
def latent_moe_bwd(dy: Tensor, d_z: Optional[Tensor], x: Tensor, w_gate: Tensor, w_down: Tensor, w_up: Tensor,
                   w_gate_up_s: Tensor, w_down_s: Tensor, w_gate_up: Tensor, w_down_e: Tensor, sel: Tensor, saved: Tensor,
                   top_k: int, z_coef: float
                   ) -> Tuple[Tensor, Tensor, Tensor, Tensor, Tensor, Tensor, Tensor, Tensor]:
    grads, _ = Fn._host().latent_bwd_raw(dy, d_z, x, w_gate, w_down, w_up, w_gate_up_s, w_down_s, w_gate_up, w_down_e, sel,
                                         saved, top_k, z_coef, False, False)
    return tuple(grads)


@latent_moe_bwd.register_fake
def _(dy, d_z, x, w_gate, w_down, w_up, w_gate_up_s, w_down_s, w_gate_up, w_down_e, sel, saved, top_k, z_coef):
    return tuple(torch.empty_like(t) for t in (x, w_gate, w_down, w_up, w_gate_up_s, w_down_s, w_gate_up, w_down_e))


def _setup_context(ctx, inputs, output):
    (x, w_gate, w_down, w_up, w_gate_up_s, w_down_s, w_gate_up, w_down_e, _bias, top_k, z_coef) = inputs
    ctx.top_k, ctx.z_coef = int(top_k), float(z_coef)
    ctx.save_for_backward(x, w_gate, w_down, w_up, w_gate_up_s, w_down_s, w_gate_up, w_down_e, output[2], output[4])
    ctx.set_materialize_grads(False)


def _backward(ctx, *grads):
    dy, d_z = grads[0], grads[1]
    x = ctx.saved_tensors[0]
    if dy is None:
        dy = x.new_zeros(x.shape)
    out = torch.ops.swamla_b200.latent_moe_bwd(dy, d_z, *ctx.saved_tensors, ctx.top_k, ctx.z_coef)
    return (*out, None, None, None)


latent_moe_fwd.register_autograd(_backward, setup_context=_setup_context)


@torch.library.custom_op("swamla_b200::latent_moe_eval", mutates_args=())
def latent_moe_eval(x: Tensor, w_gate: Tensor, w_down: Tensor, w_up: Tensor, w_gate_up_s: Tensor, w_down_s: Tensor,
                    w_gate_up: Tensor, w_down_e: Tensor, expert_bias: Tensor, top_k: int, z_coef: float) -> Tuple[Tensor, Tensor]:
    out = Fn._host().latent_moe(x, w_gate, w_down, w_up, w_gate_up_s, w_down_s, w_gate_up, w_down_e, expert_bias, top_k, z_coef,
                                False, True)
    return out[0], out[1]


@latent_moe_eval.register_fake
def _(x, w_gate, w_down, w_up, w_gate_up_s, w_down_s, w_gate_up, w_down_e, expert_bias, top_k, z_coef):
    return x.new_empty(x.shape), x.new_empty((), dtype=torch.float32)


def latent_moe_eval_compiled(x2d, *args):
    """(y, aux_loss) of an evaluated layer without gradients; arguments of ``latent_moe_compiled``."""
    return torch.ops.swamla_b200.latent_moe_eval(x2d, *args)


def latent_moe_compiled(x2d, w_gate, w_down, w_up, w_gate_up_s, w_down_s, w_gate_up, w_down_e, expert_bias, top_k: int,
                        z_coef: float):
    """Same return values as ``functional.latent_moe`` through the custom operators (traceable without graph break)."""
    out = torch.ops.swamla_b200.latent_moe_fwd(x2d, w_gate, w_down, w_up, w_gate_up_s, w_down_s, w_gate_up, w_down_e,
                                               expert_bias, int(top_k), float(z_coef))
    return out[0], out[1], out[2], out[3]
