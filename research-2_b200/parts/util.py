"""How parts hold their weights: matrices in the compute dtype, vectors in float32."""

from __future__ import annotations

import torch

from .base import Runtime


def matrix(t: torch.Tensor, rt: Runtime) -> torch.Tensor:
    """A matrix or table on the device in the compute dtype (bfloat16 serving, or float32)."""
    return t.to(device=rt.device, dtype=rt.dtype).contiguous()


def product_matrix(t: torch.Tensor, rt: Runtime) -> tuple[torch.Tensor, bool]:
    """A matrix stored [in, out] in the order in which products read it: (matrix, whether it is now [out, in]). The bfloat16 products of
    few rows take a feature's weights side by side (16 bytes a lane go straight into the matrix instruction's registers); those of many
    rows take either order at the same speed, and the float32 ones keep [in, out]."""
    m = matrix(t, rt)
    return (m.t().contiguous(), True) if rt.dtype == torch.bfloat16 else (m, False)


def vector(t: torch.Tensor, rt: Runtime) -> torch.Tensor:
    """Biases and norm parameters stay float32: they enter sums that are kept in 32-bit."""
    return t.to(device=rt.device, dtype=torch.float32).contiguous()
