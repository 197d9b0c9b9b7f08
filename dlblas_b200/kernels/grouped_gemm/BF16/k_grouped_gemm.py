"""k_grouped_gemm (dlblas/kernels/grouped_gemm/BF16/k_grouped_gemm.py:126-176 and :254-330 of the reference):
C[g] = A[rows of g]^T @ B[rows of g] for contiguous row groups of sizes `size_per_group` along the shared leading
(reduction) dimension; A [K, M], B [K, N], C [G, M, N] in the operands' 16-bit type, fp32 accumulation.  This is the
weight-gradient GEMM of a grouped linear layer.

The tcgen05 kernel reads A and B where they lie, as MN-major operands (a row of memory holds one k): nothing is
transposed or copied.  Group offsets, the tile list and the order in which the CTAs take the tiles are built on the
device in a small workspace; nothing synchronises with the host.  An empty group yields a zero C[g]."""
import torch
from torch import Tensor

from ...._C import host


def k_grouped_gemm(A: Tensor, B: Tensor, size_per_group: torch.Tensor) -> Tensor:
    return host().k_grouped_gemm(A, B, size_per_group)
