"""`dlblas.kernels.fp8` (dlblas/kernels/fp8.py:108-182 of the reference)."""
from typing import Optional, Tuple

import torch

from .._C import host


def per_token_group_quant_fp8(x: torch.Tensor, group_size: int, eps: float = 1e-10,
                              dtype: Optional[torch.dtype] = torch.float8_e4m3fn,
                              column_major_scales: bool = False) -> Tuple[torch.Tensor, torch.Tensor]:
    """Per-token-group FP8 quantisation: scale = max(absmax, eps) / 448, q = clamp(x / scale).
    Scales are [..., K/group] row-major, or for 2-D inputs a [M, G] view with strides (1, M)
    when `column_major_scales`."""
    assert dtype == torch.float8_e4m3fn, "only torch.float8_e4m3fn is supported"
    return host().group_quant_fp8(x, group_size, eps, column_major_scales)
