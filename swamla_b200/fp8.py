"""Routed experts in FP8 (e4m3) with per-tensor dynamic scaling.

Recipe: ``optimization/fp8_native.py:103-110`` ("tensorwise": one amax per tensor, scale = 448 / amax), which the
reference applies to ``nn.Linear`` modules through torchao; here it is applied to the six operands of the routed
expert GEMMs (x_sorted, gate_up weights, hidden, down weights in forward; d_y_sorted and d_h1 in backward).
Accumulation is fp32 in tensor memory and every GEMM output is bf16.  A tensor is quantised once and reused by
the forward, dgrad and wgrad GEMMs that read it.  The order of the stages is in ``csrc/torch_host.cpp``.
"""
from __future__ import annotations

import torch

from . import _cabi
from ._cabi import ptr

BF = torch.bfloat16


def quantize(t: torch.Tensor, rows: int, row_len: int, n_tiles, stream):
    """bf16 [rows, row_len] -> (e4m3 bytes [rows, row_len], deq [1] = amax / 448).  ``n_tiles``: optional device
    int32 scalar; only the first 128 * n_tiles rows are touched (padded routed layout)."""
    q = torch.empty(rows, row_len, dtype=torch.uint8, device=t.device)
    scal = torch.empty(2, dtype=torch.float32, device=t.device)      # [amax, deq]
    _cabi.call("lmoe_fp8_quantize", ptr(t), rows, row_len, ptr(n_tiles), ptr(q), ptr(scal[0:1]), ptr(scal[1:2]), stream)
    return q, scal[1:2]
