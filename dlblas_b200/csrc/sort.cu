// Stable token-by-expert counting sort and the tile lists of the grouped GEMMs.
//
// Replaces `argsort` + `_start_end_kernel` of the reference
// (dlblas/layers/moe/kernels/fused_moe.py:27-51, 83-88): O(S) instead of a radix sort plus
// an O(E*S) scan, and a defined (stable) order inside each expert segment.
//
// Buckets: 0 holds ids < 0 ("not routed here", sorted first like argsort does with -1),
// 1..E hold experts 0..E-1, E+1 holds ids >= E (sorted last, never part of a segment).
// Every warp owns a contiguous run of the flat id array, which keeps the order stable; the rank of an id inside its
// warp's run is taken once, while the run is counted, and kept in a register until the bucket bases are known.
//
// One launch up to ONE_BLOCK_SLOTS ids (the launch count is what such a sort costs), two launches (histograms per chunk;
// every block then sums the histograms of the chunks before its own, bases, scatter) up to DIRECT_CHUNKS chunks, and a
// scan kernel in between beyond that, where summing all histograms in every block would read more than the ids.
#include <mutex>

#include "common.cuh"
#include "sort.cuh"

namespace dlb {
namespace {

constexpr int ONE_BLOCK_SLOTS = 4096;
constexpr int ONE_BLOCK_MAX_SLOTS = 16384;   // still one block when the histograms of more experts than the chunked
                                             // path takes have to fit
constexpr int MAX_WARPS = 32;
constexpr int CHUNK_ITEMS = 2;               // ids per lane and pass of the chunked path
constexpr int CHUNK_STEP = MAX_WARPS * 32 * CHUNK_ITEMS;   // 2048
constexpr int DIRECT_CHUNKS = 160;
constexpr int SMEM_LIMIT = 220 * 1024;
// Without cudaFuncSetAttribute a block has 48 KB, and its static arrays (warp_sums, stats_s: 272 bytes) count towards them.
constexpr int SMEM_DEFAULT = 48 * 1024 - 512;

// Largest id and numbers of ids equal to -1 and below 0 seen by one thread (SortOut::stats).
struct IdStats {
  int largest = -1, minus_one = 0, negative = 0;
};

template <typename IdT, bool STATS = false>
__device__ __forceinline__ int bucket_of(const IdT* __restrict__ ids, unsigned f, unsigned end, int num_experts,
                                         int negative_as, IdStats* st = nullptr) {
  if (f >= end) return num_experts + 2;  // spare slot for idle lanes
  long long v = (long long)ids[f];
  if constexpr (STATS) {
    st->largest = max(st->largest, (int)min(v, 0x7fffffffll));
    st->minus_one += v == -1;
    st->negative += v < 0;
  }
  if (v < 0) {
    if (negative_as < 0) return 0;
    v = negative_as;
  }
  if (v >= num_experts) return num_experts + 1;
  return (int)v + 1;
}

// Adds a thread's statistics to the block's in shared memory (called by all threads; stats_s is zero / -1 before).
__device__ __forceinline__ void add_stats(IdStats st, int* stats_s) {
  st.largest = __reduce_max_sync(0xffffffffu, st.largest);
  st.minus_one = __reduce_add_sync(0xffffffffu, st.minus_one);
  st.negative = __reduce_add_sync(0xffffffffu, st.negative);
  if ((threadIdx.x & 31) == 0) {
    atomicMax(stats_s, st.largest);
    atomicAdd(stats_s + 1, st.minus_one);
    atomicAdd(stats_s + 2, st.negative);
  }
}

// Histograms of the warps' runs: 16-bit counters (a run and the runs before it in one pass hold at most 16384 ids), so that
// 32 warps x 256 experts take 17 KB of shared memory instead of 33.
using Count = uint16_t;
__host__ __device__ constexpr int hist_stride(int num_experts) {   // 32-bit words of two counters: E + 2 buckets + a spare
  return ((num_experts + 3 + 1) / 2) | 1;
}

// One step of the stable in-warp ranking: the number of ids of the same bucket before this one in the warp's run.
// The lanes with the same bucket are found with one ballot per bit of the bucket number: a match instruction takes its
// distinct values one after another, and with some thirty different experts in a warp that was most of the kernel.
__device__ __forceinline__ int warp_rank_step(Count* hist, int bucket, int lane, int bits) {
  unsigned peers = 0xffffffffu;
#pragma unroll 4
  for (int i = 0; i < bits; ++i) {
    const unsigned one = (bucket >> i) & 1u;
    peers &= __ballot_sync(0xffffffffu, one) ^ (one - 1u);
  }
  const int rank = __popc(peers & ((1u << lane) - 1u));
  const int old = hist[bucket];
  __syncwarp();
  if (rank == 0) hist[bucket] = (Count)(old + __popc(peers));
  __syncwarp();
  return old + rank;
}

// Turns the warps' counts of two neighbouring buckets (word p of every warp's histogram) into exclusive prefixes over the
// warps; returns the totals, one in each half.
template <int WARPS>
__device__ __forceinline__ uint32_t prefix_over_warps(uint32_t* hist, int stride, int warps, int p) {
  uint32_t run = 0;
  for (int w0 = 0; w0 < warps; w0 += WARPS) {
    uint32_t v[WARPS];
#pragma unroll
    for (int i = 0; i < WARPS; ++i) v[i] = w0 + i < warps ? hist[(w0 + i) * stride + p] : 0u;
#pragma unroll
    for (int i = 0; i < WARPS; ++i) {
      if (w0 + i < warps) hist[(w0 + i) * stride + p] = run;
      run += v[i];                  // no carry between the halves: each stays at or below 16384
    }
  }
  return run;
}

// Exclusive sums of the bucket totals (base[]) and of the buckets' tiles (tile_first[], when a tile list is wanted), by
// the whole block; block `part` of `parts` then writes its share of the segments and of the tile list.  total[], base[]
// and tile_first[] have nb = E + 2 entries in shared memory.
__device__ __forceinline__ void scan_and_write_segments(const int* total, int* base, int* tile_first, int num_experts,
                                                        const SortOut& o, int part, int parts) {
  __shared__ unsigned long long warp_sums[MAX_WARPS];
  const int nb = num_experts + 2;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, warps = blockDim.x >> 5;
  unsigned long long carry = 0;      // high half: tiles, low half: slots
  for (int b0 = 0; b0 < nb; b0 += blockDim.x) {
    const int busy = min(warps, (nb - b0 + 31) / 32);   // warps that hold buckets of this pass
    const int b = b0 + threadIdx.x;
    unsigned long long v = 0, inc = 0;
    if (warp < busy) {
      if (b < nb) {
        v = (unsigned)total[b];
        const int e = b - 1 - o.expert_offset;
        if (o.tile_rows > 0 && e >= 0 && e < o.num_local && b < nb - 1)
          v |= (unsigned long long)((unsigned)(total[b] + o.tile_rows - 1) / (unsigned)o.tile_rows) << 32;
      }
      inc = v;
#pragma unroll
      for (int d = 1; d < 32; d <<= 1) {
        const unsigned long long y = __shfl_up_sync(0xffffffffu, inc, d);
        if (lane >= d) inc += y;
      }
      if (lane == 31) warp_sums[warp] = inc;
    }
    __syncthreads();
    // the sums of the (at most 32) warps, added up by every warp for itself
    const unsigned long long s = lane < busy ? warp_sums[lane] : 0ull;
    unsigned long long incl = s;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
      if (d >= busy) break;
      const unsigned long long y = __shfl_up_sync(0xffffffffu, incl, d);
      if (lane >= d) incl += y;
    }
    const unsigned long long before = carry + __shfl_sync(0xffffffffu, incl - s, min(warp, busy - 1)) + inc - v;
    if (b < nb) {
      base[b] = (int)(unsigned)before;
      if (o.tile_rows > 0) tile_first[b] = (int)(before >> 32);
    }
    carry += __shfl_sync(0xffffffffu, incl, busy - 1);
    __syncthreads();
  }
  for (int e = part * blockDim.x + threadIdx.x; e < num_experts; e += parts * blockDim.x) {
    const int c = total[e + 1];
    const long long s = c > 0 ? (long long)base[e + 1] : 0ll;   // empty expert: start = end = 0
    if (o.exp_start) o.exp_start[e] = s;
    if (o.exp_end) o.exp_end[e] = s + c;
    if (o.counts) o.counts[e] = c;
  }
  const int num_tiles = (int)(carry >> 32);
  if (o.tiles != nullptr) {
    if (part == 0 && threadIdx.x == 0) o.tiles[0] = make_int4(min(num_tiles, o.max_tiles), 0, 0, 0);
    for (int e = part * warps + warp; e < o.num_local; e += parts * warps) {
      const int b = e + o.expert_offset + 1;
      if (b >= nb - 1) break;
      const int rows = total[b], first = tile_first[b], row0 = base[b];
      for (int i = lane; i * o.tile_rows < rows && first + i < o.max_tiles; i += 32)
        o.tiles[1 + first + i] =
            make_int4(e, row0 + i * o.tile_rows, min(o.tile_rows, rows - i * o.tile_rows), 0);
    }
  }
  if (o.aligned != nullptr) {
    if (part == 0 && threadIdx.x == 0) *o.padded_total = num_tiles * o.tile_rows;
    for (int e = part * warps + warp; e < num_experts; e += parts * warps) {
      const int rows = total[e + 1], first = tile_first[e + 1];
      const int blocks = (rows + o.tile_rows - 1) / o.tile_rows;
      for (int i = lane; i < blocks; i += 32) o.block_expert[first + i] = e;
      for (long long i = (long long)first * o.tile_rows + rows + lane; i < (long long)(first + blocks) * o.tile_rows; i += 32)
        o.aligned[i] = o.pad_slot;
    }
    for (int i = num_tiles + part * blockDim.x + threadIdx.x; i < o.num_blocks; i += parts * blockDim.x)
      o.block_expert[i] = 0;
    for (long long i = (long long)num_tiles * o.tile_rows + part * blockDim.x + threadIdx.x; i < o.aligned_len;
         i += parts * blockDim.x)
      o.aligned[i] = o.pad_slot;
  }
}

// Sum of a token's weights.  The expert-parallel path divides by torch's sum over the last dimension; the result here has the
// same bits: the upper half of the slots is added to the lower one until one is left (slots that do not exist count as zero).
__device__ __forceinline__ float slot_weight_sum(const float* __restrict__ w, int top_k) {
  auto at = [&](int j) { return j < top_k ? __ldg(w + j) : 0.f; };
  float v[8];
#pragma unroll
  for (int i = 0; i < 8; ++i) v[i] = at(i);
  if (top_k > 8) {
#pragma unroll
    for (int i = 0; i < 8; ++i) v[i] = (v[i] + at(i + 16)) + (at(i + 8) + at(i + 24));
    for (int j0 = 32; j0 < top_k; j0 += 8)
#pragma unroll
      for (int i = 0; i < 8; ++i) v[i] += at(j0 + i);
  }
  return ((v[0] + v[4]) + (v[2] + v[6])) + ((v[1] + v[5]) + (v[3] + v[7]));
}

// Output of slot f, which is at place `pos` of the sorted order.
template <typename IdT>
__device__ __forceinline__ void write_slot(unsigned f, unsigned n, int bucket, int pos, const int* base,
                                           const int* tile_first, int num_experts, const SortOut& o) {
  const bool expert = bucket >= 1 && bucket <= num_experts;
  if (o.sorted_idx) o.sorted_idx[pos] = f;
  if (o.slot_pos) o.slot_pos[f] = expert ? pos : -(pos + 1);
  if (o.rank_in_expert) o.rank_in_expert[f] = expert ? pos - base[bucket] : -1;
  if (o.aligned && expert) o.aligned[(long long)tile_first[bucket] * o.tile_rows + pos - base[bucket]] = (int)f;
  if (o.negative_as >= 0) {
    IdT* id = reinterpret_cast<IdT*>(o.ids_rw) + f;   // this thread has read it; nobody else in this kernel does
    if (*id < 0) *id = (IdT)o.negative_as;
  }
  if (o.dest) {
    const int d = pos - base[1];                      // base[1]: slots without an expert, which sort first
    const int out = expert && d < o.dest_limit ? d : -1;
    o.dest[f] = out;
    const unsigned t = f / (unsigned)o.top_k, j = f - t * (unsigned)o.top_k;
    o.row_map[j * (n / (unsigned)o.top_k) + t] = out;
  }
  if (o.w_out) {
    const float sum = slot_weight_sum(o.w_in + f / (unsigned)o.top_k * (unsigned)o.top_k, o.top_k);
    o.w_out[f] = __ldg(o.w_in + f) / sum;
  }
}

// ---- one block ---------------------------------------------------------------------
template <typename IdT, int ITEMS>
__global__ void __launch_bounds__(MAX_WARPS * 32) sort_one_block_kernel(const IdT* __restrict__ ids, unsigned n,
                                                                        int num_experts, SortOut o) {
  if (!wait_for_predecessor()) return;
  extern __shared__ int sm[];
  const int nb = num_experts + 2;
  const int stride = hist_stride(num_experts);
  const int warps = blockDim.x >> 5;
  uint32_t* hist = reinterpret_cast<uint32_t*>(sm);   // [warps][stride]
  int* total = sm + warps * stride;        // [nb]
  int* base = total + nb;                  // [nb]
  int* tile_first = base + nb;             // [nb]
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int bits = 32 - __clz(nb);         // buckets 0 ... nb, the last one for idle lanes
  const unsigned begin = warp * ITEMS * 32;
  int bucket[ITEMS], before[ITEMS];
  IdStats st;
#pragma unroll
  for (int i = 0; i < ITEMS; ++i)
    bucket[i] = bucket_of<IdT, true>(ids, begin + i * 32 + lane, n, num_experts, o.negative_as, &st);
  for (int i = threadIdx.x; i < warps * stride; i += blockDim.x) hist[i] = 0u;
  __shared__ int stats_s[3];
  if (threadIdx.x < 3) stats_s[threadIdx.x] = threadIdx.x == 0 ? -1 : 0;
  __syncthreads();
  if (o.stats != nullptr) add_stats(st, stats_s);
  Count* my = reinterpret_cast<Count*>(hist + warp * stride);
#pragma unroll
  for (int i = 0; i < ITEMS; ++i) before[i] = warp_rank_step(my, bucket[i], lane, bits);
  __syncthreads();
  for (int p = threadIdx.x; 2 * p < nb; p += blockDim.x) {
    const uint32_t both = prefix_over_warps<8>(hist, stride, warps, p);
    total[2 * p] = (int)(both & 0xffffu);
    if (2 * p + 1 < nb) total[2 * p + 1] = (int)(both >> 16);
  }
  __syncthreads();
  if (o.stats != nullptr && threadIdx.x < 3) o.stats[threadIdx.x] = stats_s[threadIdx.x];
  scan_and_write_segments(total, base, tile_first, num_experts, o, 0, 1);
#pragma unroll
  for (int i = 0; i < ITEMS; ++i) {
    const unsigned f = begin + i * 32 + lane;
    if (f < n)
      write_slot<IdT>(f, n, bucket[i], base[bucket[i]] + my[bucket[i]] + before[i], base, tile_first, num_experts, o);
  }
}

// ---- chunks ------------------------------------------------------------------------
// stats: the caller's {largest, equal to -1, below 0}; run[0..2] holds the running values and run[3] counts the blocks
// that are done (the last one, which waits for nobody, hands the values over), all of it {-1, 0, 0, 0} before the launch.
template <typename IdT>
__global__ void __launch_bounds__(512) sort_count_kernel(const IdT* __restrict__ ids, unsigned n, int num_experts,
                                                         unsigned chunk, int negative_as, int* __restrict__ cnt,
                                                         int* __restrict__ stats, int* __restrict__ run) {
  if (!wait_for_predecessor()) return;
  extern __shared__ int sm[];
  __shared__ int stats_s[3];
  const int nb = num_experts + 2;
  for (int b = threadIdx.x; b < nb + 1; b += blockDim.x) sm[b] = 0;
  if (threadIdx.x < 3) stats_s[threadIdx.x] = threadIdx.x == 0 ? -1 : 0;
  __syncthreads();
  const unsigned begin = blockIdx.x * chunk, end = min(begin + chunk, n);   // n < 2^31
  IdStats st;
  for (unsigned f0 = begin; f0 < end; f0 += 4 * 512) {
    int b[4];
#pragma unroll
    for (int i = 0; i < 4; ++i)
      b[i] = bucket_of<IdT, true>(ids, f0 + i * 512 + threadIdx.x, end, num_experts, negative_as, &st);
#pragma unroll
    for (int i = 0; i < 4; ++i)
      if (b[i] < nb) atomicAdd(sm + b[i], 1);
  }
  if (stats != nullptr) add_stats(st, stats_s);
  __syncthreads();
  if (stats != nullptr && threadIdx.x == 0) {
    atomicMax(run, stats_s[0]);
    atomicAdd(run + 1, stats_s[1]);
    atomicAdd(run + 2, stats_s[2]);
    __threadfence();
    if (atomicAdd(run + 3, 1) == (int)gridDim.x - 1) {
      __threadfence();
      for (int i = 0; i < 3; ++i) stats[i] = atomicAdd(run + i, 0);
    }
  }
  for (int b = threadIdx.x; b < nb; b += blockDim.x) cnt[(long long)blockIdx.x * nb + b] = sm[b];
}

// One CTA per bucket: exclusive prefix over chunks (in place) and the bucket total.
__global__ void __launch_bounds__(256) sort_scan_chunks_kernel(int* cnt, int num_chunks, int nb, int* total) {
  if (!wait_for_predecessor()) return;
  __shared__ int warp_sums[8];
  __shared__ int carry_s;
  const int b = blockIdx.x;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  if (threadIdx.x == 0) carry_s = 0;
  __syncthreads();
  for (int c0 = 0; c0 < num_chunks; c0 += 256) {
    const int c = c0 + threadIdx.x;
    const int v = c < num_chunks ? cnt[(long long)c * nb + b] : 0;
    int inc = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int y = __shfl_up_sync(0xffffffffu, inc, o);
      if (lane >= o) inc += y;
    }
    if (lane == 31) warp_sums[warp] = inc;
    __syncthreads();
    int woff = 0;
    for (int w = 0; w < warp; ++w) woff += warp_sums[w];
    const int carry = carry_s;
    if (c < num_chunks) cnt[(long long)c * nb + b] = carry + woff + inc - v;
    __syncthreads();
    if (threadIdx.x == 255) carry_s = carry + woff + inc;
    __syncthreads();
  }
  if (threadIdx.x == 0) total[b] = carry_s;
}

// total != nullptr: cnt already holds prefixes over the chunks (sort_scan_chunks_kernel); otherwise plain histograms.
template <typename IdT>
__global__ void __launch_bounds__(MAX_WARPS * 32) sort_scatter_kernel(const IdT* __restrict__ ids, unsigned n,
                                                                      int num_experts, unsigned chunk,
                                                                      const int* __restrict__ cnt,
                                                                      const int* __restrict__ total_in, SortOut o) {
  if (!wait_for_predecessor()) return;
  extern __shared__ int sm[];
  const int nb = num_experts + 2, stride = hist_stride(num_experts);
  uint32_t* hist = reinterpret_cast<uint32_t*>(sm);   // [MAX_WARPS][stride]
  int* total = sm + MAX_WARPS * stride;        // [nb]
  int* base = total + nb;                      // [nb]
  int* tile_first = base + nb;                 // [nb]
  int* mine = tile_first + nb;                 // [nb] slots of the bucket before the current pass of this chunk
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int bits = 32 - __clz(nb);
  const int c = blockIdx.x;
  if (total_in != nullptr) {
    for (int b = threadIdx.x; b < nb; b += blockDim.x) {
      total[b] = __ldg(total_in + b);
      mine[b] = __ldg(cnt + (long long)c * nb + b);
    }
  } else {
    for (int b = threadIdx.x; b < nb; b += blockDim.x) total[b] = mine[b] = 0;
    __syncthreads();
    // the chunks are split over as many groups of nb threads as the block holds
    const int groups = max(1, (int)blockDim.x / nb);
    const int g = threadIdx.x / nb;
    for (int b = groups > 1 ? threadIdx.x - g * nb : threadIdx.x; b < nb && g < groups; b += groups > 1 ? nb : blockDim.x) {
      int before = 0, all = 0;
#pragma unroll 8
      for (int r = groups > 1 ? g : 0; r < (int)gridDim.x; r += groups) {
        const int v = __ldg(cnt + (long long)r * nb + b);
        all += v;
        if (r < c) before += v;
      }
      atomicAdd(total + b, all);
      atomicAdd(mine + b, before);
    }
  }
  __syncthreads();
  scan_and_write_segments(total, base, tile_first, num_experts, o, c, gridDim.x);
  const unsigned begin = c * chunk, end = min(begin + chunk, n);
  Count* my = reinterpret_cast<Count*>(hist + warp * stride);
  for (unsigned p0 = begin; p0 < end; p0 += CHUNK_STEP) {
    const unsigned first = p0 + warp * CHUNK_ITEMS * 32;
    int bucket[CHUNK_ITEMS], before[CHUNK_ITEMS];
#pragma unroll
    for (int i = 0; i < CHUNK_ITEMS; ++i)
      bucket[i] = bucket_of(ids, first + i * 32 + lane, end, num_experts, o.negative_as);
    for (int i = lane; i < stride; i += 32) hist[warp * stride + i] = 0u;
    __syncwarp();
#pragma unroll
    for (int i = 0; i < CHUNK_ITEMS; ++i) before[i] = warp_rank_step(my, bucket[i], lane, bits);
    __syncthreads();
    uint32_t pass_total = 0;
    if (2 * threadIdx.x < nb) pass_total = prefix_over_warps<MAX_WARPS>(hist, stride, MAX_WARPS, threadIdx.x);
    __syncthreads();
#pragma unroll
    for (int i = 0; i < CHUNK_ITEMS; ++i) {
      const unsigned f = first + i * 32 + lane;
      const int b = bucket[i];
      if (f < end) write_slot<IdT>(f, n, b, base[b] + mine[b] + my[b] + before[i], base, tile_first, num_experts, o);
    }
    if (p0 + CHUNK_STEP < end) {
      __syncthreads();
      for (int b = 2 * threadIdx.x, i = 0; i < 2; ++i, ++b)
        if (b < nb) mine[b] += (int)((pass_total >> (16 * i)) & 0xffffu);
      __syncthreads();
    }
  }
}

struct Plan {
  bool one_block;
  int warps, items;   // of the one-block path
  size_t smem;
  long long chunk;
  int num_chunks;
  size_t total_off, run_off, bytes;
};

Plan make_plan(long long n, int num_experts) {
  Plan p;
  const int nb = num_experts + 2;
  auto one_block_smem = [&](int warps) { return (size_t)(warps * hist_stride(num_experts) + 3 * nb) * 4; };
  p.smem = (size_t)(MAX_WARPS * hist_stride(num_experts) + 4 * nb) * 4;
  const bool chunked_fits = nb <= 2048;   // a thread of the scatter kernel looks after two buckets
  p.one_block = n <= ONE_BLOCK_SLOTS || (n <= ONE_BLOCK_MAX_SLOTS && !chunked_fits);
  if (p.one_block) {
    p.items = n <= 1024 ? 1 : n <= 2048 ? 2 : n <= 4096 ? 4 : n <= 8192 ? 8 : 16;
    p.warps = (int)((n + 32 * p.items - 1) / (32 * p.items));
    if (p.warps < 8) p.warps = 8;
    // thousands of experts: fewer warps, more ids for each
    while (one_block_smem(p.warps) > (size_t)SMEM_LIMIT && p.items < 16) {
      p.items *= 2;
      p.warps = (int)((n + 32 * p.items - 1) / (32 * p.items));
    }
    p.smem = one_block_smem(p.warps);
  }
  long long chunk = (n + 1023) / 1024;
  p.chunk = (chunk + CHUNK_STEP - 1) / CHUNK_STEP * CHUNK_STEP;
  p.num_chunks = (int)((n + p.chunk - 1) / p.chunk);
  p.total_off = ((size_t)p.num_chunks * nb * 4 + 255) / 256 * 256;
  p.run_off = p.total_off + ((size_t)nb * 4 + 255) / 256 * 256;
  p.bytes = p.run_off + 256;
  return p;
}

int allow_smem(const void* kernel, bool (&configured)[64], const char* what) {
  int dev = 0;
  cudaGetDevice(&dev);
  if (dev >= 0 && dev < 64 && configured[dev]) return DLB_OK;
  int rc = check_cuda(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM_LIMIT), what);
  if (rc == DLB_OK && dev >= 0 && dev < 64) configured[dev] = true;
  return rc;
}

template <typename IdT, int ITEMS>
int launch_one_block(const IdT* ids, long long n, int num_experts, const SortOut& o, const Plan& p, cudaStream_t st) {
  if (p.smem > (size_t)SMEM_DEFAULT) {
    static bool configured[64] = {};
    int rc = allow_smem(reinterpret_cast<const void*>(sort_one_block_kernel<IdT, ITEMS>), configured,
                        "cudaFuncSetAttribute(sort_one_block_kernel)");
    if (rc != DLB_OK) return rc;
  }
  after_predecessor(sort_one_block_kernel<IdT, ITEMS>, 1, p.warps * 32, p.smem, st)(ids, (unsigned)n, num_experts, o);
  count_launch();
  DLB_CHECK_LAUNCH("sort_one_block_kernel");
  if (o.stats_event != nullptr) return check_cuda(cudaEventRecord((cudaEvent_t)o.stats_event, st), "cudaEventRecord");
  return DLB_OK;
}

template <typename IdT>
int run_sort(const IdT* ids, long long n, int num_experts, const SortOut& o, void* ws, size_t ws_bytes,
             cudaStream_t st) {
  const int nb = num_experts + 2;
  const Plan p = make_plan(n, num_experts);
  DLB_REQUIRE(p.smem <= (size_t)SMEM_LIMIT && (p.one_block || nb <= 2048), DLB_ERR_UNSUPPORTED, "sort_by_expert: %d experts are too many for %lld slots",
              num_experts, n);
  if (p.one_block) {
    switch (p.items) {
      case 1: return launch_one_block<IdT, 1>(ids, n, num_experts, o, p, st);
      case 2: return launch_one_block<IdT, 2>(ids, n, num_experts, o, p, st);
      case 4: return launch_one_block<IdT, 4>(ids, n, num_experts, o, p, st);
      case 8: return launch_one_block<IdT, 8>(ids, n, num_experts, o, p, st);
      default: return launch_one_block<IdT, 16>(ids, n, num_experts, o, p, st);
    }
  }
  DLB_REQUIRE(ws != nullptr && ws_bytes >= p.bytes, DLB_ERR_WORKSPACE,
              "sort_by_expert: workspace of %zu bytes needed, %zu given", p.bytes, ws_bytes);
  int* cnt = reinterpret_cast<int*>(ws);
  int* total = reinterpret_cast<int*>(reinterpret_cast<char*>(ws) + p.total_off);
  int* run = reinterpret_cast<int*>(reinterpret_cast<char*>(ws) + p.run_off);
  if (o.stats != nullptr) {
    cudaMemsetAsync(run, 0xff, 4, st);
    cudaMemsetAsync(run + 1, 0, 12, st);
  }
  after_predecessor(sort_count_kernel<IdT>, p.num_chunks, 512, (size_t)(nb + 1) * 4, st)(
      ids, (unsigned)n, num_experts, (unsigned)p.chunk, o.negative_as, cnt, o.stats, run);
  count_launch();
  DLB_CHECK_LAUNCH("sort_count_kernel");
  if (o.stats_event != nullptr) {
    int rc = check_cuda(cudaEventRecord((cudaEvent_t)o.stats_event, st), "cudaEventRecord");
    if (rc != DLB_OK) return rc;
  }
  const bool scan = p.num_chunks > DIRECT_CHUNKS;
  if (scan) {
    after_predecessor(sort_scan_chunks_kernel, nb, 256, 0, st)(cnt, p.num_chunks, nb, total);
    count_launch();
    DLB_CHECK_LAUNCH("sort_scan_chunks_kernel");
  }
  if (p.smem > (size_t)SMEM_DEFAULT) {
    static bool configured[64] = {};
    int rc = allow_smem(reinterpret_cast<const void*>(sort_scatter_kernel<IdT>), configured,
                        "cudaFuncSetAttribute(sort_scatter_kernel)");
    if (rc != DLB_OK) return rc;
  }
  after_predecessor(sort_scatter_kernel<IdT>, p.num_chunks, MAX_WARPS * 32, p.smem, st)(
      ids, (unsigned)n, num_experts, (unsigned)p.chunk, cnt, scan ? total : nullptr, o);
  count_launch();
  DLB_CHECK_LAUNCH("sort_scatter_kernel");
  return DLB_OK;
}

// ---- tile lists -------------------------------------------------------------------
// tiles[0] = {num_tiles, 0, 0, 0}; tiles[1 + i] = {expert, first row, valid rows, 0}.
__global__ void __launch_bounds__(1024) build_tiles_kernel(const long long* exp_start, const long long* exp_end,
                                                           const int* masked_m, int expert_offset, int num_local,
                                                           int rows_per_expert, int tile_rows, int4* tiles,
                                                           int max_tiles) {
  if (!wait_for_predecessor()) return;
  __shared__ int warp_sums[32];
  __shared__ int carry_s;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  if (threadIdx.x == 0) carry_s = 0;
  __syncthreads();
  for (int e0 = 0; e0 < num_local; e0 += blockDim.x) {
    const int e = e0 + threadIdx.x;
    long long start = 0;
    int rows = 0;
    if (e < num_local) {
      if (masked_m != nullptr) {
        rows = min(max(masked_m[e], 0), rows_per_expert);
        start = (long long)e * rows_per_expert;
      } else {
        start = exp_start[e + expert_offset];
        rows = (int)(exp_end[e + expert_offset] - start);
        if (rows < 0) rows = 0;
      }
    }
    const int nt = (rows + tile_rows - 1) / tile_rows;
    int inc = nt;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int y = __shfl_up_sync(0xffffffffu, inc, o);
      if (lane >= o) inc += y;
    }
    if (lane == 31) warp_sums[warp] = inc;
    __syncthreads();
    int woff = 0;
    for (int w = 0; w < warp; ++w) woff += warp_sums[w];
    const int carry = carry_s;
    const int first = carry + woff + inc - nt;
    for (int i = 0; i < nt; ++i) {
      const int idx = first + i;
      if (idx < max_tiles)
        tiles[1 + idx] = make_int4(e, (int)(start + (long long)i * tile_rows), min(tile_rows, rows - i * tile_rows), 0);
    }
    __syncthreads();
    if (threadIdx.x == blockDim.x - 1) carry_s = carry + woff + inc;
    __syncthreads();
  }
  if (threadIdx.x == 0) tiles[0] = make_int4(min(carry_s, max_tiles), 0, 0, 0);
}


// The same list from the sizes of consecutive row groups (clipped to `total_rows` rows in all).
template <typename SizeT>
__global__ void __launch_bounds__(1024) build_tiles_sizes_kernel(const SizeT* __restrict__ sizes, int groups,
                                                                 long long total_rows, int tile_rows,
                                                                 int4* __restrict__ tiles, int max_tiles) {
  if (!wait_for_predecessor()) return;
  __shared__ long long warp_rows[32];
  __shared__ int warp_tiles[32];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, warps = blockDim.x >> 5;
  long long rows_before = 0;     // of the groups of earlier passes
  int tiles_before = 0;
  for (int g0 = 0; g0 < groups; g0 += blockDim.x) {
    const int g = g0 + threadIdx.x;
    const long long size = g < groups ? max((long long)sizes[g], 0ll) : 0ll;
    long long inc = size;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
      const long long y = __shfl_up_sync(0xffffffffu, inc, d);
      if (lane >= d) inc += y;
    }
    if (lane == 31) warp_rows[warp] = inc;
    __syncthreads();
    long long start = rows_before + inc - size;
    for (int w = 0; w < warps; ++w) {
      if (w < warp) start += warp_rows[w];
      rows_before += warp_rows[w];
    }
    const int rows = (int)max(0ll, min(size, total_rows - start));
    const int nt = (rows + tile_rows - 1) / tile_rows;
    int tinc = nt;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
      const int y = __shfl_up_sync(0xffffffffu, tinc, d);
      if (lane >= d) tinc += y;
    }
    if (lane == 31) warp_tiles[warp] = tinc;
    __syncthreads();
    int first = tiles_before + tinc - nt;
    for (int w = 0; w < warps; ++w) {
      if (w < warp) first += warp_tiles[w];
      tiles_before += warp_tiles[w];
    }
    // one warp writes the tiles of its 32 groups, a group at a time
    for (int l = 0; l < 32; ++l) {
      const int l_nt = __shfl_sync(0xffffffffu, nt, l);
      if (l_nt == 0) continue;
      const int l_first = __shfl_sync(0xffffffffu, first, l), l_rows = __shfl_sync(0xffffffffu, rows, l);
      const int l_start = (int)__shfl_sync(0xffffffffu, start, l);
      for (int i = lane; i < l_nt && l_first + i < max_tiles; i += 32)
        tiles[1 + l_first + i] =
            make_int4(g0 + warp * 32 + l, l_start + i * tile_rows, min(tile_rows, l_rows - i * tile_rows), 0);
    }
    __syncthreads();
  }
  if (threadIdx.x == 0) tiles[0] = make_int4(min(tiles_before, max_tiles), 0, 0, 0);
}

}  // namespace

size_t sort_workspace_size(long long n, int num_experts) { return make_plan(n, num_experts).bytes; }

int sort_by_expert(const void* ids, int ids_dtype, long long n, int num_experts, long long* sorted_idx,
                   long long* exp_start, long long* exp_end, int* slot_pos, int* rank_in_expert, int* counts,
                   void* ws, size_t ws_bytes, cudaStream_t st) {
  SortOut o = {};
  o.sorted_idx = sorted_idx;
  o.exp_start = exp_start;
  o.exp_end = exp_end;
  o.slot_pos = slot_pos;
  o.rank_in_expert = rank_in_expert;
  o.counts = counts;
  return sort_by_expert(ids, ids_dtype, n, num_experts, o, ws, ws_bytes, st);
}

int sort_by_expert(const void* ids, int ids_dtype, long long n, int num_experts, const SortOut& o, void* ws,
                   size_t ws_bytes, cudaStream_t st) {
  DLB_REQUIRE(n >= 0 && n < (1ll << 31) && num_experts > 0, DLB_ERR_INVALID,
              "sort_by_expert: bad sizes num_slots=%lld num_experts=%d", n, num_experts);
  DLB_REQUIRE(ids_dtype == DLB_I32 || ids_dtype == DLB_I64, DLB_ERR_INVALID, "sort_by_expert: ids must be int32/int64");
  if (n == 0) {
    // no slots: every expert is empty, and so is the block-aligned layout (padding only: its filling is the number of slots)
    auto clear = [&](void* p, size_t bytes) {
      return p == nullptr || bytes == 0 ? DLB_OK : check_cuda(cudaMemsetAsync(p, 0, bytes, st), "cudaMemsetAsync(sort_by_expert)");
    };
    const struct { void* p; size_t bytes; } outputs[] = {
        {o.exp_start, sizeof(long long) * num_experts}, {o.exp_end, sizeof(long long) * num_experts},
        {o.counts, sizeof(int) * num_experts}, {o.tiles, sizeof(int4)}, {o.aligned, sizeof(int) * o.aligned_len},
        {o.block_expert, sizeof(int) * o.num_blocks}, {o.padded_total, sizeof(int)}};
    for (const auto& out : outputs) {
      const int rc = clear(out.p, out.bytes);
      if (rc != DLB_OK) return rc;
    }
    return DLB_OK;
  }
  DLB_REQUIRE(ids != nullptr, DLB_ERR_INVALID, "sort_by_expert: null ids");
  if (ids_dtype == DLB_I32) return run_sort<int>(reinterpret_cast<const int*>(ids), n, num_experts, o, ws, ws_bytes, st);
  return run_sort<long long>(reinterpret_cast<const long long*>(ids), n, num_experts, o, ws, ws_bytes, st);
}

}  // namespace dlb

using namespace dlb;

extern "C" size_t dlb_sort_by_expert_workspace_size(int64_t num_slots, int num_experts) {
  if (num_slots <= 0 || num_experts <= 0) return 0;
  return sort_workspace_size(num_slots, num_experts);
}

extern "C" int dlb_sort_by_expert(const void* ids, int ids_dtype, int64_t num_slots, int num_experts,
                                  int64_t* sorted_idx, int64_t* exp_start, int64_t* exp_end, int32_t* slot_pos,
                                  int32_t* rank_in_expert, int32_t* counts, void* workspace, size_t workspace_bytes,
                                  void* stream) {
  return sort_by_expert(ids, ids_dtype, num_slots, num_experts, reinterpret_cast<long long*>(sorted_idx),
                        reinterpret_cast<long long*>(exp_start), reinterpret_cast<long long*>(exp_end), slot_pos,
                        rank_in_expert, counts, workspace, workspace_bytes, (cudaStream_t)stream);
}

// ---- variant of the sort that never allocates -----------------------------------------
// Some callers cannot hand over a workspace: an inference engine that reserved all device
// memory for its own pool at start-up has nothing left for cudaMalloc to give, and code that
// runs where an allocation's implicit device-wide synchronisation is not acceptable must not
// call the allocator at all.  For them the chunk histograms live in a fixed array that is
// part of the loaded module (every GPU that loads the library holds these bytes until exit).
namespace {
constexpr size_t STATIC_SCRATCH_BYTES = (size_t)4 * 1024 * 1024 + 16 * 1024;
static __device__ __align__(256) unsigned char g_sort_scratch[STATIC_SCRATCH_BYTES];

// In host code `g_sort_scratch` is only a handle for the runtime, not a device address; the
// address the kernels need is looked up once per device, with that device current.
void* g_scratch_ptr[64] = {};
std::mutex g_scratch_mutex;

int static_scratch(void** out) {
  int dev = 0;
  int rc = check_cuda(cudaGetDevice(&dev), "cudaGetDevice");
  if (rc != DLB_OK) return rc;
  DLB_REQUIRE(dev >= 0 && dev < 64, DLB_ERR_UNSUPPORTED, "sort_by_expert_static: device index %d out of range", dev);
  std::lock_guard<std::mutex> lock(g_scratch_mutex);
  if (g_scratch_ptr[dev] == nullptr) {
    void* p = nullptr;
    rc = check_cuda(cudaGetSymbolAddress(&p, g_sort_scratch), "cudaGetSymbolAddress(g_sort_scratch)");
    if (rc != DLB_OK) return rc;
    DLB_REQUIRE(p != nullptr, DLB_ERR_CUDA, "sort_by_expert_static: the scratch array has no device address");
    g_scratch_ptr[dev] = p;
  }
  *out = g_scratch_ptr[dev];
  return DLB_OK;
}
}  // namespace

extern "C" size_t dlb_sort_by_expert_static_capacity(void) { return STATIC_SCRATCH_BYTES; }

extern "C" int dlb_sort_by_expert_static(const void* ids, int ids_dtype, int64_t num_slots, int num_experts,
                                         int64_t* sorted_idx, int64_t* exp_start, int64_t* exp_end,
                                         int32_t* slot_pos, int32_t* rank_in_expert, int32_t* counts, void* stream) {
  DLB_REQUIRE(num_slots >= 0 && num_experts > 0, DLB_ERR_INVALID,
              "sort_by_expert_static: bad sizes num_slots=%lld num_experts=%d", (long long)num_slots, num_experts);
  const size_t need = num_slots > 0 ? sort_workspace_size(num_slots, num_experts) : 0;
  DLB_REQUIRE(need <= STATIC_SCRATCH_BYTES, DLB_ERR_WORKSPACE,
              "sort_by_expert_static: num_slots=%lld with num_experts=%d needs %zu bytes of scratch, the built-in "
              "array holds %zu; use dlb_sort_by_expert with a caller-provided workspace",
              (long long)num_slots, num_experts, need, STATIC_SCRATCH_BYTES);
  void* scratch = nullptr;
  int rc = static_scratch(&scratch);
  if (rc != DLB_OK) return rc;
  // Every word of the scratch that the kernels read is written earlier in the same call (the
  // count kernel fills the whole histogram matrix), so leftovers of a previous call are harmless.
  return sort_by_expert(ids, ids_dtype, num_slots, num_experts, reinterpret_cast<long long*>(sorted_idx),
                        reinterpret_cast<long long*>(exp_start), reinterpret_cast<long long*>(exp_end), slot_pos,
                        rank_in_expert, counts, scratch, STATIC_SCRATCH_BYTES, (cudaStream_t)stream);
}

extern "C" int dlb_moe_build_tiles(const int64_t* exp_start, const int64_t* exp_end, int expert_offset,
                                   int num_local_experts, int32_t* tiles, int max_tiles, void* stream) {
  DLB_REQUIRE(exp_start && exp_end && tiles, DLB_ERR_INVALID, "build_tiles: null pointer");
  DLB_REQUIRE(num_local_experts > 0 && expert_offset >= 0 && max_tiles >= 0, DLB_ERR_INVALID, "build_tiles: bad sizes");
  DLB_REQUIRE((uintptr_t)tiles % 16 == 0, DLB_ERR_INVALID, "build_tiles: tiles must be 16-byte aligned");
  after_predecessor(build_tiles_kernel, 1, 1024, 0, (cudaStream_t)stream)(reinterpret_cast<const long long*>(exp_start),
                                                           reinterpret_cast<const long long*>(exp_end), nullptr,
                                                           expert_offset, num_local_experts, 0, 128,
                                                           reinterpret_cast<int4*>(tiles), max_tiles);
  count_launch();
  DLB_CHECK_LAUNCH("build_tiles_kernel");
  return DLB_OK;
}

extern "C" int dlb_moe_build_tiles_rows(const int64_t* exp_start, const int64_t* exp_end, int expert_offset,
                                        int num_local_experts, int tile_rows, int32_t* tiles, int max_tiles,
                                        void* stream) {
  DLB_REQUIRE(exp_start && exp_end && tiles, DLB_ERR_INVALID, "build_tiles_rows: null pointer");
  DLB_REQUIRE(num_local_experts > 0 && expert_offset >= 0 && max_tiles >= 0, DLB_ERR_INVALID,
              "build_tiles_rows: bad sizes");
  DLB_REQUIRE(tile_rows == 128 || tile_rows == 256, DLB_ERR_INVALID, "build_tiles_rows: tile_rows must be 128 or 256");
  DLB_REQUIRE((uintptr_t)tiles % 16 == 0, DLB_ERR_INVALID, "build_tiles_rows: tiles must be 16-byte aligned");
  after_predecessor(build_tiles_kernel, 1, 1024, 0, (cudaStream_t)stream)(reinterpret_cast<const long long*>(exp_start),
                                                           reinterpret_cast<const long long*>(exp_end), nullptr,
                                                           expert_offset, num_local_experts, 0, tile_rows,
                                                           reinterpret_cast<int4*>(tiles), max_tiles);
  count_launch();
  DLB_CHECK_LAUNCH("build_tiles_kernel");
  return DLB_OK;
}

extern "C" int dlb_moe_build_tiles_masked(const int32_t* masked_m, int num_local_experts, int rows_per_expert,
                                          int32_t* tiles, int max_tiles, void* stream) {
  DLB_REQUIRE(masked_m && tiles, DLB_ERR_INVALID, "build_tiles_masked: null pointer");
  DLB_REQUIRE(num_local_experts > 0 && rows_per_expert > 0 && max_tiles >= 0, DLB_ERR_INVALID,
              "build_tiles_masked: bad sizes");
  DLB_REQUIRE((uintptr_t)tiles % 16 == 0, DLB_ERR_INVALID, "build_tiles_masked: tiles must be 16-byte aligned");
  after_predecessor(build_tiles_kernel, 1, 1024, 0, (cudaStream_t)stream)(nullptr, nullptr, masked_m, 0, num_local_experts,
                                                           rows_per_expert, 128, reinterpret_cast<int4*>(tiles),
                                                           max_tiles);
  count_launch();
  DLB_CHECK_LAUNCH("build_tiles_kernel");
  return DLB_OK;
}

extern "C" int dlb_moe_build_tiles_sizes(const void* sizes, int sizes_dtype, int num_groups, int64_t total_rows,
                                         int tile_rows, int32_t* tiles, int max_tiles, void* stream) {
  DLB_REQUIRE(sizes && tiles, DLB_ERR_INVALID, "build_tiles_sizes: null pointer");
  DLB_REQUIRE(num_groups > 0 && total_rows >= 0 && total_rows < (1ll << 31) && max_tiles >= 0, DLB_ERR_INVALID,
              "build_tiles_sizes: bad sizes");
  DLB_REQUIRE(tile_rows == 128 || tile_rows == 256, DLB_ERR_INVALID, "build_tiles_sizes: tile_rows must be 128 or 256");
  DLB_REQUIRE(sizes_dtype == DLB_I32 || sizes_dtype == DLB_I64, DLB_ERR_INVALID,
              "build_tiles_sizes: sizes must be int32 or int64");
  DLB_REQUIRE((uintptr_t)tiles % 16 == 0, DLB_ERR_INVALID, "build_tiles_sizes: tiles must be 16-byte aligned");
  const int threads = num_groups >= 1024 ? 1024 : (num_groups + 31) / 32 * 32;
  int4* out = reinterpret_cast<int4*>(tiles);
  if (sizes_dtype == DLB_I32)
    after_predecessor(build_tiles_sizes_kernel<int>, 1, threads, 0, (cudaStream_t)stream)(
        reinterpret_cast<const int*>(sizes), num_groups, total_rows, tile_rows, out, max_tiles);
  else
    after_predecessor(build_tiles_sizes_kernel<long long>, 1, threads, 0, (cudaStream_t)stream)(
        reinterpret_cast<const long long*>(sizes), num_groups, total_rows, tile_rows, out, max_tiles);
  count_launch();
  DLB_CHECK_LAUNCH("build_tiles_sizes_kernel");
  return DLB_OK;
}

extern "C" int dlb_moe_plan(const void* ids, int ids_dtype, int64_t tokens, int top_k, int num_experts, int expert_offset,
                            int num_local_experts, int tile_rows, int64_t* sorted_idx, int32_t* slot_pos, int32_t* tiles,
                            int max_tiles, const float* weights, float* normalised, void* workspace, size_t workspace_bytes,
                            void* stream) {
  DLB_REQUIRE(tokens >= 0 && top_k > 0 && num_local_experts > 0 && expert_offset >= 0 && max_tiles >= 0, DLB_ERR_INVALID,
              "moe_plan: bad sizes");
  DLB_REQUIRE(tiles != nullptr && (uintptr_t)tiles % 16 == 0, DLB_ERR_INVALID, "moe_plan: tiles must be 16-byte aligned");
  DLB_REQUIRE(tile_rows == 128 || tile_rows == 256, DLB_ERR_INVALID, "moe_plan: tile_rows must be 128 or 256");
  DLB_REQUIRE((weights == nullptr) == (normalised == nullptr), DLB_ERR_INVALID, "moe_plan: weights without a result");
  SortOut o = {};
  o.sorted_idx = reinterpret_cast<long long*>(sorted_idx);
  o.slot_pos = slot_pos;
  o.tile_rows = tile_rows;
  o.expert_offset = expert_offset;
  o.num_local = num_local_experts;
  o.tiles = reinterpret_cast<int4*>(tiles);
  o.max_tiles = max_tiles;
  o.top_k = top_k;
  o.w_in = weights;
  o.w_out = normalised;
  return sort_by_expert(ids, ids_dtype, tokens * top_k, num_experts, o, workspace, workspace_bytes, (cudaStream_t)stream);
}

extern "C" int dlb_moe_align_block_size(void* ids, int ids_dtype, int64_t num_slots, int num_experts, int negative_as,
                                        int block_size, int32_t* sorted_ids, int64_t sorted_len, int32_t* expert_ids,
                                        int num_blocks, int32_t* num_padded, void* workspace, size_t workspace_bytes,
                                        void* stream) {
  DLB_REQUIRE(block_size > 0 && negative_as >= 0 && sorted_len >= 0 && num_blocks >= 0, DLB_ERR_INVALID,
              "moe_align_block_size: bad sizes");
  DLB_REQUIRE(num_slots >= 0 && num_experts > 0 && sorted_len >= num_slots + (int64_t)num_experts * (block_size - 1) &&
                  sorted_len < (1ll << 31) && (int64_t)num_blocks * block_size >= sorted_len,
              DLB_ERR_INVALID, "moe_align_block_size: outputs too small");
  DLB_REQUIRE((sorted_ids || sorted_len == 0) && (expert_ids || num_blocks == 0) && num_padded, DLB_ERR_INVALID,
              "moe_align_block_size: null pointer");
  SortOut o = {};
  o.tile_rows = block_size;
  o.num_local = num_experts;
  o.aligned = sorted_ids;
  o.aligned_len = sorted_len;
  o.block_expert = expert_ids;
  o.num_blocks = num_blocks;
  o.padded_total = num_padded;
  o.pad_slot = (int)num_slots;
  o.negative_as = negative_as;
  o.ids_rw = ids;
  return sort_by_expert(ids, ids_dtype, num_slots, num_experts, o, workspace, workspace_bytes, (cudaStream_t)stream);
}

extern "C" int dlb_permute_plan(const void* ids, int ids_dtype, int64_t tokens, int top_k, int num_experts,
                                int64_t dest_limit, int64_t* sorted_idx, int32_t* dest, int32_t* row_id_map, int32_t* stats,
                                void* stats_event, void* workspace, size_t workspace_bytes, void* stream) {
  DLB_REQUIRE(tokens > 0 && top_k > 0 && dest && row_id_map, DLB_ERR_INVALID, "permute_plan: bad arguments");
  SortOut o = {};
  o.sorted_idx = reinterpret_cast<long long*>(sorted_idx);
  o.top_k = top_k;
  o.dest = dest;
  o.row_map = row_id_map;
  o.dest_limit = dest_limit;
  o.stats = stats;
  o.stats_event = stats_event;
  return sort_by_expert(ids, ids_dtype, tokens * top_k, num_experts, o, workspace, workspace_bytes, (cudaStream_t)stream);
}
