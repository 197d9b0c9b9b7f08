"""`dlblas.kernels.moe_align_block_size` of the reference (vLLM's block-aligned token layout,
dlblas/kernels/moe_align_block_size.py:138-210).

Every expert's slots are laid out contiguously and padded to a multiple of `block_size`:
sorted_ids int32 [max padded] holds flat slot indices (t * top_k + j) grouped by expert in ascending slot
order, padding entries = topk_ids.numel(); expert_ids int32 [blocks] = expert of every block (0 for blocks
past the end); num_tokens_post_pad int32 [1].  The library's stable sort writes the layout itself (one kernel up to 4096 slots,
two up to 327680, three beyond; no host round trip).  Without slots everything is padding: zeros.
"""
from typing import Optional, Tuple

import torch

from .._C import host


def moe_align_block_size(topk_ids: torch.Tensor, block_size: int, num_experts: int, num_local_experts: int,
                         expert_map: Optional[torch.Tensor] = None,
                         pad_sorted_ids: bool = False) -> Tuple[torch.Tensor, torch.Tensor, torch.Tensor]:
    """Same contract as the reference, including its side effect: negative ids in `topk_ids` are replaced
    in place by `num_local_experts` (the "not on this rank" id, :178-180).  Ids >= num_experts are ignored."""
    return host().moe_align_block_size(topk_ids, block_size, num_experts, num_local_experts, expert_map, pad_sorted_ids)
