// Internal interface of the stable token-by-expert sort (sort.cu), shared with the
// permutation, gating and expert-layer entry points.
#pragma once
#include <cuda_runtime.h>
#include <stddef.h>

namespace dlb {
// What one sort writes; every pointer may be null.
struct SortOut {
  long long* sorted_idx;
  long long* exp_start;
  long long* exp_end;
  int* slot_pos;
  int* rank_in_expert;
  int* counts;
  // tiles of tile_rows slots (0: none) of experts [expert_offset, expert_offset + num_local): the list that the grouped
  // GEMMs read
  int tile_rows, expert_offset, num_local;
  int4* tiles;
  int max_tiles;
  // ... or the block-aligned layout, every expert padded to whole tiles: slots in aligned[aligned_len] (pad_slot where
  // there is none), the expert of every block, slots of the padded experts
  int* aligned;
  long long aligned_len;
  int* block_expert;
  int num_blocks;
  int* padded_total;
  int pad_slot;
  // ids < 0 count as this id and are overwritten with it (< 0: they stay what they are)
  int negative_as = -1;
  void* ids_rw;
  int top_k;
  // routing weights divided by their sum over a token's top_k slots
  const float* w_in;
  float* w_out;
  // place of slot f among the routed slots, -1 if it has no expert or the place is not below dest_limit: [slots], and
  // the same with the slots of a token top_k-major
  int* dest;
  int* row_map;
  long long dest_limit;
  // {largest id (-1 if there is none), ids equal to -1, ids < 0}, written once; stats_event (a cudaEvent_t, may be null) is
  // recorded as soon as the kernel that writes them is enqueued
  int* stats;
  void* stats_event;
};
size_t sort_workspace_size(long long n, int num_experts);
int sort_by_expert(const void* ids, int ids_dtype, long long n, int num_experts, const SortOut& o, void* ws,
                   size_t ws_bytes, cudaStream_t st);
// Any output pointer may be null.  See dlb_sort_by_expert in include/dlblas_b200.h.
int sort_by_expert(const void* ids, int ids_dtype, long long n, int num_experts, long long* sorted_idx,
                   long long* exp_start, long long* exp_end, int* slot_pos, int* rank_in_expert, int* counts,
                   void* ws, size_t ws_bytes, cudaStream_t st);
}  // namespace dlb
