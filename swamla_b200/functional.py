"""Functional form of the LatentMoE path.  Forward and backward are assembled from the C-ABI entry points of ``liblmoe.so``
by the native host path (``csrc/torch_host.cpp`` -> ``_host.so``); PyTorch only provides device memory, the stream and
autograd.

Forward follows ``models/moe.py:702-734`` of the reference (``LatentMoELayer.forward``); the
backward is the adjoint of each cited line (the reference defines it only through autograd and
not at all for its grouped GEMM, ``models/moe_triton.py:200-242``).
"""
from __future__ import annotations

from typing import Optional

import torch

from . import _cabi, _testing
from ._cabi import Route, Shape, ptr

BF = torch.bfloat16

# LMOE_TMA_GATHER=1 (read by the native host path): the gate_up GEMMs (forward and weight gradient) read the latent rows
# through TMA gathers (tile::gather4) driven by the routing table, with no gather kernel and no x_sorted buffer (P*L*2
# bytes less memory).  Off by default: results are bit-identical but four-row gathers of 128-byte rows sustained only about
# 8 GB/s per SM.


def d_hidden_scratch(lib, P, L, F, **kw):
    """The routed dgrad stage needs no [P, F] scratch: the SwiGLU adjoint runs in the epilogue of the d_hidden GEMM
    (saved gate / up staged by TMA), or inside the chain kernel; d_hidden never reaches memory."""
    return None


def _host():
    """The native host path; ``liblmoe.so`` is loaded (and checked for) first."""
    global _native
    if _native is None:
        _cabi.load()
        try:
            from . import _host as native
        except ImportError as e:
            raise _cabi.LmoeError(f"swamla_b200/_host.so is missing or was built for another PyTorch or Python ({e}): build it with "
                                  "`python -m swamla_b200.build` (there is no CPU or PyTorch fallback for this path)") from e
        native.set_error_class(_cabi.LmoeError)
        _native = native
    return _native


_native = None


def _stream() -> int:
    return torch.cuda.current_stream().cuda_stream


def _as_bf16(t: torch.Tensor) -> torch.Tensor:
    """bf16 copy of a float tensor through the library's cast kernel (no-op for bf16)."""
    if t.dtype == BF:
        return t.contiguous()
    if t.dtype != torch.float32:
        t = t.float()
    t = t.contiguous()
    out = torch.empty(t.shape, dtype=BF, device=t.device)
    _cabi.call("lmoe_cast_f32_to_bf16", ptr(t), ptr(out), t.numel(), _stream())
    return out


def padded_rows_of(T: int, K: int, E: int) -> int:
    """Static row count of the padded expert layout (what ``lmoe_padded_rows`` returns)."""
    return (T * K + 127) // 128 * 128 + E * 128


class RouteTables:
    """Device buffers behind an ``lmoe_route`` struct: one int32 allocation (``storage``), sliced."""

    @staticmethod
    def storage_numel(T: int, K: int, E: int) -> int:
        P = padded_rows_of(T, K, E)
        return sum((n + 3) // 4 * 4 for n in (E, E + 1, E + 1, 1, P // 128, T * K, T * K, P))

    def __init__(self, shape: Shape, device, storage: Optional[torch.Tensor] = None,
                 counts: Optional[torch.Tensor] = None):
        T, K, E = shape.T, shape.K, shape.E
        self.padded_rows = padded_rows_of(T, K, E)
        i32 = dict(dtype=torch.int32, device=device)
        # one allocation, sliced; every slice starts 16-byte aligned
        sizes = dict(counts=E, offsets=E + 1, pad_offsets=E + 1, n_tiles=1, tile_expert=self.padded_rows // 128,
                     perm=T * K, pos=T * K, row_src=self.padded_rows)
        total = sum((n + 3) // 4 * 4 for n in sizes.values())
        self.storage = torch.empty(total, **i32) if storage is None else storage   # given: tables of an earlier forward
        off = 0
        for name, n in sizes.items():
            setattr(self, name, self.storage[off:off + n])
            off += (n + 3) // 4 * 4
        if counts is not None:      # the native host path keeps the histogram in a tensor of its own
            self.counts = counts
        self.struct = Route(**{k: ptr(getattr(self, k)) for k in sizes})


def make_shape(T, D, L, E, K, F, Fs, n_shared=1) -> Shape:
    return Shape(T=T, D=D, L=L, E=E, K=K, F=F, Fs=Fs, n_shared=n_shared)


def check_status(status: torch.Tensor) -> None:
    """Reads one device status word now (synchronises); raises if a kernel reported a failure.  The layers use the
    non-blocking monitor in ``status.py`` instead; this form serves tests and callers of the functional API."""
    code = int(status.item())
    if code != 0:
        raise _cabi.LmoeError(f"device status {code}: {_cabi.status_string(code)}")


class LatentMoEFunction(torch.autograd.Function):
    """The native host path's two directions under a Python autograd node that can hand out their intermediates and take
    a given selection: used while a parity test's hook is set (``_testing.py``)."""

    @staticmethod
    def forward(ctx, x, w_gate, w_down, w_up, w_gate_up_s, w_down_s, w_gate_up, w_down_e, expert_bias, top_k: int,
                z_coef: float, fp8: bool = False):
        forced = _testing.FORCE_SEL
        if forced is not None:
            forced = forced.to(device=x.device, dtype=torch.int32).contiguous()
        params = (x, w_gate, w_down, w_up, w_gate_up_s, w_down_s, w_gate_up, w_down_e)
        y, z_loss, sel, counts, saved, views = _host().latent_fwd_raw(*params, expert_bias, top_k, z_coef, fp8, forced,
                                                                      _testing.capturing())
        ctx.save_for_backward(*params, sel, saved)
        ctx.args = (top_k, z_coef, fp8)
        ctx.mark_non_differentiable(sel, counts)
        if views:
            E, L, F2 = w_gate_up.shape
            shape = make_shape(sel.shape[0], x.shape[-1], L, E, top_k, F2 // 2, w_down_s.shape[1])
            views["route"] = RouteTables(shape, x.device, storage=views.pop("route_storage"), counts=counts)
            _testing.capture(sel=sel, **views)
        return y, z_loss, sel, counts

    @staticmethod
    def backward(ctx, dy, d_z, _d_sel, _d_counts):
        *params, sel, saved = ctx.saved_tensors
        grads, views = _host().latent_bwd_raw(dy, d_z, *params, sel, saved, *ctx.args, _testing.capturing())
        _testing.capture(**views)
        return (*grads, None, None, None, None)


def latent_moe(x: torch.Tensor, w_gate, w_down, w_up, w_gate_up_s, w_down_s, w_gate_up, w_down_e, expert_bias, top_k: int,
               z_coef: float, fp8: bool = False, evaluation: bool = False):
    """Functional form on a [..., D] activation.  Returns (y like x, aux_loss scalar, sel [T,K] int32, counts [E] int32).
    ``fp8``: run the routed expert GEMMs in e4m3 with per-tensor scaling (latent and routed hidden dims % 128 == 0).
    ``evaluation``: without gradients and without ``fp8``, a few tokens may take the path of ``lmoe_few_forward`` (no
    routing tables: only (y, aux_loss) is returned then)."""
    if _testing.SINK is not None or _testing.FORCE_SEL is not None:
        return LatentMoEFunction.apply(x, w_gate, w_down, w_up, w_gate_up_s, w_down_s, w_gate_up, w_down_e, expert_bias,
                                       top_k, z_coef, fp8)
    return (_native or _host()).latent_moe(x, w_gate, w_down, w_up, w_gate_up_s, w_down_s, w_gate_up, w_down_e, expert_bias,
                                           top_k, z_coef, fp8, evaluation)


# opaque to torch.compile: the layer runs as an eager call between compiled regions
latent_moe_opaque = torch.compiler.disable(latent_moe)


def saved_bytes(T, D, L, E, K, F, Fs):
    """Bytes that one bf16 forward keeps for its backward (the native path's ``LatentLayout``), as shape arithmetic that
    also works on the symbolic sizes of a traced graph."""
    P = padded_rows_of(T, K, E)
    sizes = (T * E * 4, T * K * 4, T * 4, RouteTables.storage_numel(T, K, E) * 4, T * (L + Fs) * 2, T * 2 * Fs * 2, P * L * 2,
             P * 2 * F * 2, P * L * 2, P * F * 2)
    return sum((n + 255) // 256 * 256 for n in sizes)
