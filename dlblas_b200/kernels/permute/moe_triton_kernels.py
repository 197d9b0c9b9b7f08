"""Token permutation for MoE training, forward and backward
(dlblas/kernels/permute/moe_triton_kernels.py of the reference; the autograd wrappers follow
tests/kernels/permute/triton_ops.py).

permute:    rows of `input` are replicated top_k times and ordered by expert (stable: ascending flat slot
            index inside an expert; slots routed to -1 are dropped).  `row_id_map` int32 [top_k * tokens],
            k-major, gives the destination row of every (token, slot), -1 for dropped slots.
unpermute:  out[t] = sum_k prob[t, k] * permuted[row_id_map[k, t]], rounded to the tensor type after every
            product and add (the reference accumulates in the tensor type).
The module keeps its reference name although nothing here is Triton: the kernels are the library's sort,
fan-out copy and un-permute kernels, the host side and the autograd functions are in csrc/host.cpp.
"""
from typing import List, Optional, Tuple

import torch

from ..._C import check, host, lib, ptr, require_cuda, stream


def moe_permute_topk_op_triton(input_tensor: torch.Tensor, indices: torch.Tensor, num_out_tokens: int,
                               workspace: List[torch.Tensor], max_expanded_token_num: int,
                               num_negative_one_in_indices: int, permuted_output: torch.Tensor,
                               row_id_map: torch.Tensor):
    """Reference signature (:62-137).  Fills `permuted_output` [num_out_tokens, H] and `row_id_map`; returns
    (permuted_output, row_id_map, sorted_row_id, workspace).  Entries of row_id_map for dropped slots are set
    to -1 (the reference leaves them unwritten)."""
    require_cuda(input_tensor, indices)
    t, k = indices.shape
    h = input_tensor.shape[1]
    if num_out_tokens <= 0:
        num_out_tokens = t * k - num_negative_one_in_indices
    assert permuted_output.shape == (num_out_tokens, h), "permuted_output shape mismatch"
    assert row_id_map.numel() == t * k, "row_id_map size mismatch"
    sidx, dest, rmap, _, _ = host().permute_plan(indices, num_out_tokens)
    x = input_tensor.contiguous()
    row_bytes = h * x.element_size()
    check(lib().dlb_permute_rows(ptr(x), row_bytes, 0, 0, t, ptr(dest), k, ptr(permuted_output), 0, stream(x.device)))
    row_id_map.view(-1).copy_(rmap)
    return permuted_output, row_id_map, sidx, workspace


def moe_recover_topk_op_triton(input_tensor: torch.Tensor, row_id_map: torch.Tensor, prob: Optional[torch.Tensor],
                               num_tokens: int, num_topK: int) -> torch.Tensor:
    """Weighted gather back to token order (:274-301); prob None = plain sum."""
    return host().unpermute_rows(input_tensor, row_id_map, prob, num_tokens, num_topK)


def moe_permute_topk_bwd_op(permuted_act_grad: torch.Tensor, sorted_row_id: torch.Tensor, original_shape, num_topK: int):
    """Gradient of permute (:190-213): act_grad[t] = sum over the token's slots of permuted_act_grad[row].
    `sorted_row_id` lists the flat slot of every permuted row (rows of dropped slots must not be included)."""
    require_cuda(permuted_act_grad)
    t = original_shape[0]
    rows = permuted_act_grad.shape[0]
    sid = sorted_row_id.to(torch.int64)[-rows:] if sorted_row_id.numel() > rows else sorted_row_id.to(torch.int64)
    rmap = torch.full((num_topK * t,), -1, dtype=torch.int32, device=permuted_act_grad.device)
    rmap[(sid % num_topK) * t + sid // num_topK] = torch.arange(rows, dtype=torch.int32, device=rmap.device)
    return moe_recover_topk_op_triton(permuted_act_grad, rmap, None, t, num_topK)


def moe_recover_topk_bwd_op_triton(input_bwd: torch.Tensor, input_fwd: torch.Tensor, row_id_map: torch.Tensor,
                                   prob: torch.Tensor) -> Tuple[torch.Tensor, torch.Tensor]:
    """Gradient of unpermute (:480-528): (act_grad fp32 [rows, H], prob_grad fp32 [tokens, top_k])."""
    return host().unpermute_backward(input_bwd, input_fwd, row_id_map, prob, torch.float32)


def permute(input_act: torch.Tensor, indices: torch.Tensor):
    """(permuted activations [routed slots, H], row_id_map); differentiable in `input_act`."""
    return host().permute(input_act, indices)


def unpermute(input_act: torch.Tensor, row_id_map: torch.Tensor, probs: Optional[torch.Tensor] = None):
    """Weighted combine back to token order; differentiable in `input_act` and `probs`."""
    return host().unpermute(input_act, row_id_map, probs)
