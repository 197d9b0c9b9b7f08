"""m_grouped_gemm (dlblas/kernels/grouped_gemm/BF16/m_grouped_gemm.py:235-352 of the reference):
C[rows of group g] = A[rows of g] @ B[g] for contiguous row groups of sizes `size_per_group`.

B is read where it lies in both layouts: [G, N, K] (`trans_b=True`) as a K-major operand, [G, K, N] (`trans_b=False`,
the reference's default) as an MN-major operand of the tensor cores; only a K that is not a multiple of 64 makes the
second layout fall back to one transposition of B per call.  Tile list and group offsets are built on the device;
nothing synchronises with the host."""
import torch
from torch import Tensor

from ...._C import check_status, host  # noqa: F401


def m_grouped_gemm(A: Tensor, B: Tensor, size_per_group: torch.Tensor, trans_b: bool = False, numSM: int = -1) -> Tensor:
    return host().m_grouped_gemm(A, B, size_per_group, trans_b)
