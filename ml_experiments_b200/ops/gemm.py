"""tcgen05/TMEM GEMM front end.

``gemm(a, b)`` computes ``epilogue(a @ b.T)`` on the fifth-generation tensor cores. Each operand may be given
K-major (``[rows, K]``, the default) or MN-major (``[K, rows]``, flag ``a_mn`` / ``b_mn``), which lets the three
products of a linear layer run on the stored tensors without a transpose pass:

* forward      ``y  = x @ W.T``   -> ``gemm(x, W)``
* data grad    ``dx = dy @ W``    -> ``gemm(dy, W, b_mn=True)``
* weight grad  ``dW = dy.T @ x``  -> ``gemm(dy, x, a_mn=True, b_mn=True)``

Counterpart of the cuBLAS / ``torch._scaled_mm`` / Triton ``tl.dot`` call sites of the reference
(modded-nanogpt/train_gpt.py:45-137,171-189,950,969; modded-nanogpt/triton_kernels.py:54-391).
"""
from __future__ import annotations

import torch

from .runtime import ops, status

EPI_NONE, EPI_RELU2, EPI_AXPBY, EPI_RELU2_BWD = 0, 1, 2, 3


def _overlap(x: torch.Tensor, y: torch.Tensor) -> bool:
    """True when the memory spans of two tensors intersect (conservative for strided views)."""
    if x.numel() == 0 or y.numel() == 0 or x.device != y.device:
        return False
    span = lambda t: (t.data_ptr(), t.data_ptr() + (sum((n - 1) * abs(st) for n, st in zip(t.shape, t.stride())) + 1) * t.element_size())
    (x0, x1), (y0, y1) = span(x), span(y)
    return x0 < y1 and y0 < x1


def gemm(a: torch.Tensor, b: torch.Tensor, *, out: torch.Tensor | None = None, out_dtype=None,
         a_mn: bool = False, b_mn: bool = False, epilogue: int = EPI_NONE, aux: torch.Tensor | None = None,
         alpha: float = 1.0, beta: float = 0.0, split_k: int = 1, accumulate: bool = False) -> torch.Tensor:
    """``out = epilogue(alpha * a @ b.T [+ beta * aux])``; 2-D or batched 3-D operands, bf16 or fp8 inputs."""
    m = a.shape[-1] if a_mn else a.shape[-2]
    n = b.shape[-1] if b_mn else b.shape[-2]
    if out is None:
        if out_dtype is None:
            out_dtype = torch.float32 if (split_k > 1 or accumulate) else torch.bfloat16
        out = torch.empty(*a.shape[:-2], m, n, dtype=out_dtype, device=a.device)
    elif _overlap(out, a) or _overlap(out, b):
        # an output tile is stored while other CTAs still read the operand panels: the result would depend on timing
        raise ValueError("gemm: `out` must not alias an operand")
    ops().gemm(a, b, out, aux, a_mn, b_mn, epilogue, alpha, beta, split_k, accumulate, status(a.device))
    return out


def auto_split_k(m: int, n: int, k: int, sms: int = 148) -> int:
    """Split factor of a weight gradient whose output has fewer tiles than the machine: as many parts as fill one round or, for a long
    ``k``, up to four rounds, by the work in the longest chain of tiles. A part costs its share of ``k`` and, where its result is added to
    the output, some 1700 more. 2304 x 768 x 49152 (54 tiles): 142 us in 2 parts, one round with 108 of 148 busy, 130 in 5; 3072 x 1024 x
    10000 (96 tiles) 67 in one, 56 in 3. Where this differs from as many as fill one round (22 of 200 weight gradients timed), all are faster.
    Three and more parts are added in any order: such a gradient repeats to the rounding of fp32 sums, not bit for bit."""
    bn = 256 if n > 128 else 128
    tiles = ((m + 127) // 128) * ((n + bn - 1) // bn)
    if tiles >= sms or k < 1024:
        return 1
    one = max(1, min(sms // tiles, k // 512))
    if k < 8192:
        return one
    return min([one] + list(range(one + 1, min(4 * sms // tiles, 16) + 1)),
               key=lambda s: -(-tiles * s // sms) * (-(-k // s) + (1700 if s > 1 else 400)))
