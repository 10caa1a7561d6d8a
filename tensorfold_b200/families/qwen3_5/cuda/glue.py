"""Row-wise glue that feeds the quantized matmuls: residual add + RMSNorm and SwiGLU, each returning the fp32 group sums
of its bf16 output (a matmul's ``xs``).  Mirrors ``add_rmsnorm`` and ``swiglu`` of the reference
(families/qwen3_5/cuda/glue.py:31-40,146-151); each row is computed on its own, in a fixed order of operations."""

from __future__ import annotations

import torch

from .... import _lib


def add_rmsnorm(x: torch.Tensor, r: torch.Tensor | None, w: torch.Tensor, eps: float, gs: int = 64):
    """h = x + r (bf16), y = rmsnorm(h) * w (bf16), xs = y's group sums (fp32).  Returns (h, y, xs); h is x when r is None."""

    return _lib.native().add_rmsnorm(x, r, w, eps, gs)


def swiglu(gate: torch.Tensor, up: torch.Tensor, gs: int = 64):
    """out = bf16(gate * sigmoid(gate) * up), xs = out's group sums (fp32).  Returns (out, xs)."""

    return _lib.native().swiglu(gate, up, gs)
