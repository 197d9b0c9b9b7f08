// Block-scaled FP8 (e4m3) GEMMs for sm_100a: dense and grouped over ragged expert
// segments.  One persistent, warp-specialised kernel:
//
//   warp 8  (1 thread)  TMA producer: A tile [128 x 128B] and B tile [BN x 128B] per
//                       128-wide K block into a ring of 128B-swizzled smem stages.
//   warp 9  (1 thread)  issues tcgen05.mma kind::f8f6f4 (128 x BN x 32, four per K block)
//                       into a ring of TMEM accumulators, one accumulator per K block.
//   warps 0-7           promotion: tcgen05.ld each K block's partial product,
//                       acc += partial * a_scale[row, kb] * b_scale[nblk, kb] on the CUDA
//                       cores (the scales are arbitrary fp32, so the hardware block-scale
//                       path, which wants UE8M0 scales, does not apply).  At the end of a tile
//                       they round the accumulators to the 16-bit output type, park them in a
//                       shared-memory staging tile and go straight on to the next tile.
//   warps 10-11         epilogue: rows of the staging tile leave with one bulk copy each
//                       (store / scatter), or are turned into silu(gate)*up, quantised per 128
//                       columns and stored as e4m3 (fused w13 epilogue), while the other roles
//                       already work on the next tile.  (Tiles of 64 and 128 columns are emptied by the
//                       promotion warps, see store_rows.  With fp32 output the tile does not fit
//                       the staging buffer and the promotion warps store it themselves.)
//
// (A 16-warp variant, four promotion warps per scheduler partition with 64 accumulator columns
// each, was measured too: 5 % faster on large dense problems, but its 96-register budget spills
// in the fused silu*up epilogue and it was 15 % slower on the grouped w13 GEMM, so the 8-warp
// layout below is the one kept.)
//
// Register budget: an accumulator tile is 128 x BN fp32 = half of the register file at
// BN = 256, and hiding the TMEM load latency needs 64 more staging registers per promotion
// thread, so the promotion warpgroups run at 232 registers and the third warpgroup at 40.
//
// The arithmetic follows dlblas/kernels/fp8_gemm.py:50-59 and
// dlblas/layers/moe/kernels/blocked_fp8_fused_moe.py:95-156 of the reference: fp32
// accumulation over K blocks in increasing order, one rounding to the output type.
//
// All mbarrier waits are bounded (about 2 s of SM clock cycles): a wait that exceeds its limit raises a CTA-wide
// abort flag, every role leaves its loop, the status word is set to DLB_STATUS_TIMEOUT
// and the kernel returns after draining what it issued.
#include "tile_width.h"
#include "umma.cuh"

namespace dlb {
namespace {

constexpr int BM = 128;
constexpr int BK = 128;              // bytes == elements (e4m3)
constexpr int A_STAGE_BYTES = BM * BK;
constexpr int EPI_WARPS = 8;         // two warpgroups
constexpr int PRODUCER_WARP = 8;
constexpr int MMA_WARP = 9;
constexpr int STORE_WARP0 = 10;       // warps 10 and 11: epilogue out of the staging tile
constexpr int STORE_WARPS = 2;
constexpr int NUM_THREADS = 384;      // three warpgroups
constexpr int REGS_PROMOTION = 232;    // 256 * 232 + 128 * 40 = 384 * 168
constexpr int REGS_OTHER = 40;
constexpr int TMEM_COLS = 512;

// Tiles of at most SWAP_ROWS rows (256-wide, 16-bit output, one CTA per tile) exchange the operands: the 128 rows of the
// tensor core's tile are columns of C, its columns the rows of A, 16 at a time.  A tile with a handful of rows otherwise
// multiplies and promotes 128 all the same; the weights' way from DRAM bounds such a launch, and in repeated passes that
// work costs the clocks and with them the memory rate.  (Up to 64 rows per tile this way: 2 % slower on those steps.)
// Registers: the promotion warps hold both forms without a spill, but for 24 bytes of stores and 72 of loads in the fused
// epilogue, where the kernel without the exchanged form spills 24 / 64 (ptxas).
constexpr int SWAP_ROWS = 32;
constexpr int CHUNK = 16;                    // rows of A per box and per step of N
constexpr int CHUNKS = SWAP_ROWS / CHUNK;

struct GemmArgs {
  const float* a_s;
  long long a_s_rs, a_s_ks;   // a_s[row * rs + kb * ks]
  const float* b_s;
  long long b_s_es;           // per-expert stride; inside: [nblk * kblocks + kb]
  void* c;
  long long ldc;
  float* q_scale;             // SWIGLU_QUANT: [rows, n_half/128]
  int quant_mode;
  float quant_eps;
  const int4* tiles;          // nullptr: dense, M tiles derived from m
  int m, n, k;
  int n_half;                 // SWIGLU_QUANT: intermediate size (n / 2)
  int num_m_tiles_static;
  int num_n_tiles;
  int m_band;    // order of the tiles, see tile_at
  int n_tile0;   // first n tile of the launch (a launch may cover a window of the columns; 0 otherwise)
  const long long* sorted_idx;
  const float* weights;
  int* status;
  unsigned long long timeout_cycles;
  int withhold_loads;         // self-test of the time-out path: the producer issues no load
};

// kind::f8f6f4, A and B e4m3 K-major, fp32 accumulate, M = 128, N = bn.
__host__ __device__ constexpr uint32_t make_idesc(int bn, int ctas = 1) {
  return (1u << 4) | ((uint32_t)(bn >> 3) << 17) | ((uint32_t)((ctas * BM) >> 4) << 24);
}

// CTAS = 2: pairs of CTAs on 256-row tiles (tcgen05 cta_group::2); every CTA then stages only half of the B tile
template <int BN, int CTAS = 1> struct Cfg {
  static constexpr int B_STAGE_BYTES = (BN / CTAS) * BK;
  static constexpr int STAGE_BYTES = A_STAGE_BYTES + B_STAGE_BYTES;
  static constexpr int STAGES = (BN == 256) ? (CTAS == 2 ? 4 : 3) : (BN == 128 ? 5 : 8);
  static constexpr int TMEM_BUFS = TMEM_COLS / BN;
  // accumulators are handed back in order, so the last of RUN free ones says that all of them are
  static constexpr int RUN = TMEM_BUFS / 2;
  static constexpr int COLS = BN / 2;  // columns per promotion thread: the first warpgroup has the first half
  // Staging tile of the epilogue: BM rows of BN 16-bit values.  Rows are padded by 16 bytes so
  // that the 16-byte stores of 32 threads holding 32 different rows spread over all banks.
  static constexpr int STAGING_ROW_BYTES = BN * 2 + 16;
  static constexpr int STAGING_BYTES = BM * STAGING_ROW_BYTES;
  // dynamic smem: stages | staging tile | barriers (full, done, tmem_empty, drain, staged, staging_free) | misc
  static constexpr int STAGING_OFF = STAGES * STAGE_BYTES;
  static constexpr int BAR_OFF = STAGING_OFF + STAGING_BYTES;
  // One commit per K block: its barrier (the stage's) tells the producer that the stage is free and the promotion warps that
  // the accumulator is full.  (A commit holds the MMA warp for about 45 cycles, and a question for a barrier for as long:
  // narrow tiles ask about the accumulators once in RUN K blocks.)  The promotion warps wait by parity, so none may miss a
  // phase.  K block it + STAGES uses the stage next; its MMAs are issued only after every promotion warp has drained K block
  // it + STAGES - TMEM_BUFS, and with it, STAGES being no less than TMEM_BUFS, K block it, whose phase it waited for.
  static_assert(STAGES >= TMEM_BUFS, "a promotion warp could miss a phase of the stage's barrier");
  static constexpr int NUM_BARS = 2 * STAGES + TMEM_BUFS + 3;
  static constexpr int MISC_OFF = BAR_OFF + NUM_BARS * 8;
  static constexpr int SMEM_BYTES = MISC_OFF + 16 + 1024;  // + slack for 1024 B alignment
};

struct Tile {
  int e, row0, rows, n0;
};

// The part of tile t that CTA `rank` of a pair works on (CTAS = 2: rows [rank * 128, rank * 128 + 128) of the
// 256-row tile; its `rows` is 0 when the tile ends before them).
template <int BN, int MODE, int CTAS = 1>
__device__ __forceinline__ Tile decode_tile(const GemmArgs& g, int num_m_tiles, int t, int rank = 0) {
  Tile ti;
  int m_tile, n_tile;
  tile_at(t, num_m_tiles, g.num_n_tiles, g.m_band, m_tile, n_tile);
  if (g.tiles != nullptr) {
    const int4 v = __ldg(g.tiles + 1 + m_tile);
    ti.e = v.x;
    ti.row0 = v.y;
    ti.rows = v.z;
  } else {
    ti.e = 0;
    ti.row0 = m_tile * CTAS * BM;
    ti.rows = min(CTAS * BM, g.m - ti.row0);
  }
  if constexpr (CTAS == 2) {
    ti.row0 += rank * BM;
    ti.rows = min(BM, max(0, ti.rows - rank * BM));
  }
  ti.n0 = (n_tile + g.n_tile0) * (MODE == DLB_EPI_SWIGLU_QUANT ? BN / 2 : BN);
  return ti;
}

template <typename OutT> struct Pack;
template <> struct Pack<__nv_bfloat16> {
  static __device__ __forceinline__ uint32_t two(float a, float b) {
    __nv_bfloat162 v = __floats2bfloat162_rn(a, b);
    return *reinterpret_cast<uint32_t*>(&v);
  }
};
template <> struct Pack<__half> {
  static __device__ __forceinline__ uint32_t two(float a, float b) {
    __half2 v = __floats2half2_rn(a, b);
    return *reinterpret_cast<uint32_t*>(&v);
  }
};

// Stores NCOLS accumulators (a compile-time count, multiple of 8) of one row; only the first
// `valid` columns exist.  dst is 16-byte aligned.  Fully unrolled so `acc` stays in registers.
template <typename OutT, int NCOLS>
__device__ __forceinline__ void store_row(OutT* dst, const float (&acc)[NCOLS], int valid) {
  if constexpr (sizeof(OutT) == 4) {
#pragma unroll
    for (int j = 0; j < NCOLS; j += 4) {
      if (j < valid)
        *reinterpret_cast<float4*>(reinterpret_cast<float*>(dst) + j) =
            make_float4(acc[j], acc[j + 1], acc[j + 2], acc[j + 3]);
    }
  } else {
#pragma unroll
    for (int j = 0; j < NCOLS; j += 8) {
      if (j < valid) {
        uint4 v;
        v.x = Pack<OutT>::two(acc[j], acc[j + 1]);
        v.y = Pack<OutT>::two(acc[j + 2], acc[j + 3]);
        v.z = Pack<OutT>::two(acc[j + 4], acc[j + 5]);
        v.w = Pack<OutT>::two(acc[j + 6], acc[j + 7]);
        *reinterpret_cast<uint4*>(dst + j) = v;
      }
    }
  }
}

__device__ __forceinline__ void tmem_ld16(uint32_t taddr, uint32_t (&v)[16]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 "
      "{%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
      : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]), "=r"(v[8]),
        "=r"(v[9]), "=r"(v[10]), "=r"(v[11]), "=r"(v[12]), "=r"(v[13]), "=r"(v[14]), "=r"(v[15])
      : "r"(taddr)
      : "memory");
}
__device__ __forceinline__ void tmem_ld_wait16(uint32_t (&a)[16]) {
  asm volatile("tcgen05.wait::ld.sync.aligned;"
               : "+r"(a[0]), "+r"(a[1]), "+r"(a[2]), "+r"(a[3]), "+r"(a[4]), "+r"(a[5]), "+r"(a[6]), "+r"(a[7]),
                 "+r"(a[8]), "+r"(a[9]), "+r"(a[10]), "+r"(a[11]), "+r"(a[12]), "+r"(a[13]), "+r"(a[14]), "+r"(a[15])
               :
               : "memory");
}

template <int BN, int MODE, typename OutT, int CTAS, bool SWAP>
__global__ void __launch_bounds__(NUM_THREADS, 1)
gemm_fp8_kernel(const __grid_constant__ CUtensorMap tmap_a, const __grid_constant__ CUtensorMap tmap_a16,
                const __grid_constant__ CUtensorMap tmap_b, const GemmArgs g) {
  using C = Cfg<BN, CTAS>;
  constexpr bool PAIR = CTAS == 2;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  const uint32_t smem_base = smem_u32(smem);
  const uint32_t bar_base = smem_base + C::BAR_OFF;
  auto full_bar = [&](int s) { return bar_base + 8u * s; };
  auto done_bar = [&](int s) { return bar_base + 8u * (C::STAGES + s); };   // stage free, its K block's accumulator full
  auto tempty_bar = [&](int b) { return bar_base + 8u * (2 * C::STAGES + b); };
  const uint32_t drain_bar = bar_base + 8u * (2 * C::STAGES + C::TMEM_BUFS);
  const uint32_t staged_bar = drain_bar + 8u;   // promotion warps -> epilogue warps: tile is in the staging buffer
  const uint32_t sfree_bar = drain_bar + 16u;   // epilogue warps -> promotion warps: staging buffer may be reused
  uint8_t* staging = smem + C::STAGING_OFF;
  constexpr bool STAGED = sizeof(OutT) == 2;
  constexpr bool SELF_DRAIN = STAGED && BN < 256;   // the promotion warps empty the staging tile
  static_assert(!SWAP || (BN == 256 && !PAIR && STAGED), "the exchanged form fills the staging tile of one CTA");
  auto swapped = [](const Tile& ti) { return SWAP && ti.rows <= SWAP_ROWS; };
  auto chunks_of = [](const Tile& ti) { return max(1, (ti.rows + CHUNK - 1) / CHUNK); };   // of a swapped tile
  volatile uint32_t* tmem_holder = reinterpret_cast<volatile uint32_t*>(smem + C::MISC_OFF);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(smem + C::MISC_OFF + 4);

  const int warp = threadIdx.x >> 5;
  const int lane = threadIdx.x & 31;
  const uint32_t rank = PAIR ? cluster_ctarank() : 0u;   // 0 = leader of a pair: it issues the MMAs
  const int worker = blockIdx.x / CTAS;                   // CTA or pair index
  const int workers = gridDim.x / CTAS;
  const int kblocks = g.k / BK;
  const unsigned long long limit = g.timeout_cycles;

  if (threadIdx.x == 0) {
    for (int s = 0; s < C::STAGES; ++s) {
      mbar_init(full_bar(s), 1);
      mbar_init(done_bar(s), 1);
    }
    for (int b = 0; b < C::TMEM_BUFS; ++b)
      mbar_init(tempty_bar(b), CTAS * EPI_WARPS);   // pair: the promotion warps of both CTAs release the leader's
    mbar_init(drain_bar, 1);
    mbar_init(staged_bar, EPI_WARPS);
    mbar_init(sfree_bar, SELF_DRAIN ? EPI_WARPS : STORE_WARPS);
    abort_flag[0] = 0;
    abort_flag[1] = 0;   // private flag of the drain waits
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  }
  if (warp == PRODUCER_WARP && elect_one()) {
    prefetch_map(&tmap_a);
    prefetch_map(&tmap_b);
    if constexpr (SWAP) prefetch_map(&tmap_a16);
  }
  if (warp == MMA_WARP) {
    if constexpr (PAIR) {
      asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(
                       smem_u32(const_cast<uint32_t*>(tmem_holder))),
                   "r"(TMEM_COLS)
                   : "memory");
      asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
    } else {
      asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(
                       smem_u32(const_cast<uint32_t*>(tmem_holder))),
                   "r"(TMEM_COLS)
                   : "memory");
      asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
  }
  tc_fence_before();
  __syncthreads();
  if constexpr (PAIR) cluster_sync();   // both CTAs' barriers exist before anything remote touches them
  tc_fence_after();
  const uint32_t tmem_base = *tmem_holder;
  if (!wait_for_predecessor(false)) return;
  const int num_m_tiles = g.tiles != nullptr ? __ldg(reinterpret_cast<const int*>(g.tiles)) : g.num_m_tiles_static;
  const int total_tiles = num_m_tiles * g.num_n_tiles;

  // Narrow tiles are chosen for launches that probably have one tile per CTA, so nothing follows that could hide the staging
  // tile's way out: the promotion warps empty it themselves with ordinary 16-byte stores, warp w of EPI_WARPS its share of the
  // rows.  (A bulk copy per row holds its lane for some 70 cycles: 100 rows of 64 columns took two warps 5100 of the kernel's
  // 18300 cycles; 100 x 7168 x 2048 alone 11.1 -> 9.0 us by these stores, 128 x 12288 x 2048 12.2 -> 10.8.  256 columns keep
  // the two epilogue warps and the bulk copies, which run beside the next tile: with these lines for the last tile only,
  // 8192 x 4096 x 7168 lost 3 %.)
  auto store_rows = [&](const Tile& ti, int w) {
    constexpr int VECS = BN / 8, ROWS = 32 / VECS;       // vectors of a row, rows of a pass
    const int vec = lane % VECS, in_pass = lane / VECS;
    const bool there = ti.n0 + vec * 8 < g.n;            // n % 8 == 0
#pragma unroll 4
    for (int row = w * ROWS + in_pass; row < ti.rows; row += EPI_WARPS * ROWS) {
      long long crow = (long long)ti.row0 + row;
      if constexpr (MODE == DLB_EPI_SCATTER_WEIGHT) crow = __ldg(g.sorted_idx + crow);
      if (there)
        *reinterpret_cast<uint4*>(reinterpret_cast<OutT*>(g.c) + crow * g.ldc + ti.n0 + vec * 8) =
            *reinterpret_cast<const uint4*>(staging + row * C::STAGING_ROW_BYTES + vec * 16);
    }
  };

  if (warp >= EPI_WARPS) {
    // third warpgroup: give registers away, then run the producer / MMA roles
    reg_dec<REGS_OTHER>();
  // The producer and MMA warps run their loops with all 32 lanes converged and elect one lane
  // only around the TMA / tcgen05 instructions: addresses, descriptors and barrier operands then
  // live in uniform registers.  With a single lane running the whole loop the same instructions
  // were issued from per-thread registers and each tcgen05.mma held the warp's scheduler
  // partition for ~120 cycles, starving the two promotion warps that share it.
  if (warp == PRODUCER_WARP) {
    {
      uint32_t it = 0;
      bool ok = true;
      for (int t = worker; t < total_tiles && ok; t += workers) {
        const Tile ti = decode_tile<BN, MODE, CTAS>(g, num_m_tiles, t, (int)rank);
        const int boxes = swapped(ti) ? chunks_of(ti) : 0;
        for (int kb = 0; kb < kblocks; ++kb, ++it) {
          const int s = it % C::STAGES;
          const uint32_t ph = (it / C::STAGES) & 1u;
          if (!mbar_wait(done_bar(s), ph ^ 1u, abort_flag, limit)) {
            ok = false;
            break;
          }
          const uint32_t a_dst = smem_base + s * C::STAGE_BYTES;
          const uint32_t b_dst = a_dst + A_STAGE_BYTES;
          if (g.withhold_loads) {
            // nothing is loaded: the consumers' waits run into their limit
          } else if constexpr (PAIR) {
            // each CTA fetches its 128 rows of A and its half of the B tile (the gate slab in the leader, the up
            // slab in its partner for the fused w13 epilogue); all of it is counted on the leader's barrier
            const uint32_t lead_full = mapa(full_bar(s), 0);
            if (elect_one()) {
              if (rank == 0) mbar_expect_tx(full_bar(s), 2 * C::STAGE_BYTES);
              tma_load_2d_pair(a_dst, &tmap_a, kb * BK, ti.row0, lead_full);
              const int b_row = (MODE == DLB_EPI_SWIGLU_QUANT) ? ti.e * g.n + (int)rank * g.n_half + ti.n0
                                                                : ti.e * g.n + ti.n0 + (int)rank * (BN / 2);
              tma_load_2d_pair(b_dst, &tmap_b, kb * BK, b_row, lead_full);
            }
          } else if (elect_one()) {
            if (boxes == 0) {
              mbar_expect_tx(full_bar(s), C::STAGE_BYTES);
              tma_load_2d(a_dst, &tmap_a, kb * BK, ti.row0, full_bar(s));
            } else {
              mbar_expect_tx(full_bar(s), C::B_STAGE_BYTES + boxes * (CHUNK * BK));
              for (int i = 0; i < boxes; ++i)
                tma_load_2d(a_dst + i * (CHUNK * BK), &tmap_a16, kb * BK, ti.row0 + i * CHUNK, full_bar(s));
            }
            if constexpr (MODE == DLB_EPI_SWIGLU_QUANT) {
              // gate rows [n0, n0+128) and up rows [n_half + n0, ...+128) of expert e
              tma_load_2d(b_dst, &tmap_b, kb * BK, ti.e * g.n + ti.n0, full_bar(s));
              tma_load_2d(b_dst + 128 * BK, &tmap_b, kb * BK, ti.e * g.n + g.n_half + ti.n0, full_bar(s));
            } else {
#pragma unroll
              for (int h = 0; h < (BN + 127) / 128; ++h)   // boxes of min(BN, 128) rows
                tma_load_2d(b_dst + h * 128 * BK, &tmap_b, kb * BK, ti.e * g.n + ti.n0 + h * 128, full_bar(s));
            }
          }
          __syncwarp();
        }
      }
      if (!ok && !g.withhold_loads) {
        // drain: give the loads of the last STAGES iterations a bounded chance to land
        const uint32_t first = it > (uint32_t)C::STAGES ? it - C::STAGES : 0u;
        for (uint32_t i = first; i < it; ++i)
          mbar_wait(full_bar(i % C::STAGES), (i / C::STAGES) & 1u, abort_flag + 1, 40000000ull);
      }
    }
  } else if (warp == MMA_WARP) {
    {
      constexpr uint32_t idesc = make_idesc(BN, CTAS);
      uint32_t s = 0, s_phase = 0, b = 0, b_phase = 1;   // stage and accumulator of the next K block
      bool ready = false;                                // both are known to be there
      // One lane issues; elected once, as the warp is whole wherever it acts.  (Two elections per K block and lanes that
      // branch on their own answers: 64 x 4096 x 7168 18.3 us, votes with two elections 18.6, votes and this 17.1.)
      const bool lead = elect_one();
      bool ok = true;
      for (int t = worker; t < total_tiles && ok && rank == 0; t += workers) {
        uint32_t idesc_swap = 0;
        if constexpr (SWAP) {
          const Tile ti = decode_tile<BN, MODE, CTAS>(g, num_m_tiles, t, (int)rank);
          if (swapped(ti)) idesc_swap = make_idesc(CHUNK * chunks_of(ti));
        }
        for (int kb = 0; kb < kblocks; ++kb) {
          const bool new_run = b % C::RUN == 0;
          if (!ready && (!mbar_wait(full_bar(s), s_phase, abort_flag, limit) ||
                         (new_run && !mbar_wait(tempty_bar(b + C::RUN - 1), b_phase, abort_flag, limit)))) {
            ok = false;
            break;
          }
          tc_fence_after();
          const uint32_t a_addr = smem_base + s * C::STAGE_BYTES;
          const uint64_t a_desc = make_smem_desc(a_addr);
          const uint64_t b_desc = make_smem_desc(a_addr + A_STAGE_BYTES);
          const uint32_t d_tmem = tmem_base + b * BN;
          const uint32_t done = done_bar(s);
          if (++s == C::STAGES) { s = 0; s_phase ^= 1u; }
          if (++b == C::TMEM_BUFS) { b = 0; b_phase ^= 1u; }
          // +32 bytes along K inside the 128 B swizzle row == +2 in the (addr >> 4) field
          auto mma = [&](int kk) {
            if constexpr (PAIR) tc_mma_f8_pair(d_tmem, a_desc + 2u * kk, b_desc + 2u * kk, idesc, kk > 0 ? 1u : 0u);
            else tc_mma_f8(d_tmem, a_desc + 2u * kk, b_desc + 2u * kk, idesc, kk > 0 ? 1u : 0u);
          };
          const bool swap = SWAP && idesc_swap != 0;
          if (lead) {
            if (swap) {
#pragma unroll
              for (int kk = 0; kk < BK / 32; ++kk)
                tc_mma_f8(d_tmem, b_desc + 2u * kk, a_desc + 2u * kk, idesc_swap, kk > 0 ? 1u : 0u);
            } else {
              mma(0);
              mma(1);
            }
          }
          // The tensor core's queue holds two to three instructions: the next K block's barriers are asked about while
          // those of this one are in it.  Asked after the last, the answers left the pipe idle for some 300 cycles a block.
          ready = mbar_test(full_bar(s), s_phase);
          if (b % C::RUN == 0) ready = mbar_test(tempty_bar(b + C::RUN - 1), b_phase) && ready;
          if (lead) {
            if (swap) {
              const uint64_t b2_desc = make_smem_desc(a_addr + A_STAGE_BYTES + BM * BK);
#pragma unroll
              for (int kk = 0; kk < BK / 32; ++kk)
                tc_mma_f8(d_tmem + BM, b2_desc + 2u * kk, a_desc + 2u * kk, idesc_swap, kk > 0 ? 1u : 0u);
            } else {
              mma(2);
              mma(3);
            }
            if constexpr (PAIR) {
              tc_commit_pair(done);   // both CTAs
            } else {
              tc_commit(done);   // once these MMAs retire
            }
          }
          ready = __all_sync(WHOLE_WARP, ready);
        }
      }
      if (!ok) {
        if (lead) {
          if constexpr (PAIR)
            asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(drain_bar)
                         : "memory");
          else
            tc_commit(drain_bar);
        }
        __syncwarp();
        mbar_wait(drain_bar, 0, abort_flag + 1, 40000000ull);
      }
    }
  } else if (STAGED && !SELF_DRAIN) {
    // ---- epilogue warps: empty the staging tile while the next tile is being computed ----
    const int ew = warp - STORE_WARP0;
    uint32_t tile_no = 0;
    bool ok = true;
    for (int t = worker; t < total_tiles && ok; t += workers, ++tile_no) {
      const Tile ti = decode_tile<BN, MODE, CTAS>(g, num_m_tiles, t, (int)rank);
      if constexpr (MODE == DLB_EPI_SWIGLU_QUANT) {
        // A staging row holds the tile's 128 gate columns, then its 128 up columns, already
        // rounded to OutT.  Reference rounding points: silu(gate)*up -> OutT, then
        // scale = absmax * (1/448), q = h / scale (dlblas/kernels/moe.py:398-417), or the
        // max(absmax, eps) / 448 form of dlblas/kernels/fp8.py:9-182.  Same arithmetic as
        // silu_mul_quant_kernel, bit for bit.
        if (!mbar_wait(staged_bar, tile_no & 1u, abort_flag, limit)) {
          ok = false;
          break;
        }
        const long long groups = g.n_half / 128;
        // half a warp per row, eight columns per lane: two rows per pass, eight independent
        // chains per lane to cover the exp / divide latencies
        const int sub = lane >> 4;
        const int cl = lane & 15;
        for (int row0 = ew * 2; row0 < ti.rows; row0 += 2 * STORE_WARPS) {
          const int row = row0 + sub;
          const bool act = row < ti.rows;
          const uint8_t* srow = staging + (act ? row : row0) * C::STAGING_ROW_BYTES;
          const uint4 gv = *reinterpret_cast<const uint4*>(srow + cl * 16);
          const uint4 uv = *reinterpret_cast<const uint4*>(srow + BN + cl * 16);
          const OutT* gp = reinterpret_cast<const OutT*>(&gv);
          const OutT* up = reinterpret_cast<const OutT*>(&uv);
          float h[8];
          float amax = 0.f;
#pragma unroll
          for (int j = 0; j < 8; ++j) {
            const float gt = to_f32<OutT>(gp[j]);
            h[j] = to_f32<OutT>(from_f32<OutT>(silu_fast(gt) * to_f32<OutT>(up[j])));
            amax = fmaxf(amax, fabsf(h[j]));
          }
#pragma unroll
          for (int o = 8; o > 0; o >>= 1) amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, o));
          const float scale =
              g.quant_mode == DLB_QUANT_RECIP_MUL ? amax * (1.0f / 448.0f) : fmaxf(amax, g.quant_eps) / 448.0f;
          if (act) {
            const long long p = (long long)ti.row0 + row;
            const uint2 q = quant8_rcp(h, 1.0f / scale);
            *reinterpret_cast<uint2*>(reinterpret_cast<uint8_t*>(g.c) + p * g.ldc + ti.n0 + cl * 8) = q;
            if (cl == 0) g.q_scale[p * groups + ti.n0 / 128] = scale;
          }
        }
      } else {
        // this lane sends rows ew*64 + lane and ew*64 + 32 + lane
        long long crow[2];
        bool valid[2];
#pragma unroll
        for (int i = 0; i < 2; ++i) {
          const int row = ew * 64 + i * 32 + lane;
          valid[i] = row < ti.rows;
          crow[i] = (long long)ti.row0 + row;
          if constexpr (MODE == DLB_EPI_SCATTER_WEIGHT) {
            if (valid[i]) crow[i] = g.sorted_idx[crow[i]];
          }
        }
        if (!mbar_wait(staged_bar, tile_no & 1u, abort_flag, limit)) {
          ok = false;
          break;
        }
        const uint32_t bytes = (uint32_t)min(BN, g.n - ti.n0) * 2u;   // n % 8 == 0
#pragma unroll
        for (int i = 0; i < 2; ++i) {
          if (valid[i]) {
            const int row = ew * 64 + i * 32 + lane;
            bulk_store(reinterpret_cast<OutT*>(g.c) + crow[i] * g.ldc + ti.n0,
                       smem_u32(staging + row * C::STAGING_ROW_BYTES), bytes);
          }
        }
        bulk_commit();
        bulk_wait_read();
      }
      __syncwarp();
      if (lane == 0) mbar_arrive(sfree_bar);
    }
    bulk_wait_all();
  }
  } else {
    // ---- promotion + epilogue warps ------------------------------------------
    reg_inc<REGS_PROMOTION>();
    const int wg = warp >> 2;                 // 0 or 1
    const int quad = warp & 3;                // TMEM lane quadrant of this warp
    const int r = quad * 32 + lane;           // row inside the tile
    constexpr int COLS = C::COLS;
    const int col0 = wg * COLS;               // this thread's columns of the tile (SWIGLU: gate | up)
    const uint32_t lane_addr = tmem_base + ((uint32_t)(quad * 32) << 16);
    uint32_t it = 0;
    uint32_t tile_no = 0;
    bool ok = true;
    for (int t = worker; t < total_tiles && ok; t += workers, ++tile_no) {
      const Tile ti = decode_tile<BN, MODE, CTAS>(g, num_m_tiles, t, (int)rank);
      const bool row_ok = r < ti.rows;
      const long long p = (long long)ti.row0 + r;          // row of A / sorted position
      // threads without a row read the scales of a row that exists (a pair's second CTA can hold an empty
      // half tile whose first row lies beyond the end of A)
      const float* as_ptr = g.a_s + (row_ok ? p : (long long)min(ti.row0, g.m - 1)) * g.a_s_rs;
      // scale block of this thread's columns
      const float* bs_ptr;
      {
        const int nb = MODE == DLB_EPI_SWIGLU_QUANT ? (wg * g.n_half + ti.n0) / 128
                                                    : min((ti.n0 + col0) / 128, (g.n + 127) / 128 - 1);
        bs_ptr = g.b_s + (long long)ti.e * g.b_s_es + (long long)nb * kblocks;
      }
      if constexpr (SWAP) {
        if (swapped(ti)) {
          // lane = column: the first warpgroup has the first 128 columns of the tile (SWIGLU: gate), the second the others.
          // Lanes 0-15 (and 16-31 again) fetch the scales of a chunk's 16 rows, two K blocks ahead.  The products and their
          // order are those of the other form.
          const int chunks = chunks_of(ti);
          const float* bs = bs_ptr;
          const float* as = g.a_s + (long long)min(ti.row0, g.m - 1) * g.a_s_rs;
          int a_off[CHUNKS];                       // less than SWAP_ROWS rows' worth of scales
          float a0[CHUNKS], a1[CHUNKS], a2[CHUNKS];
          float b0 = __ldg(bs), b1 = kblocks > 1 ? __ldg(bs + 1) : 0.f, b2 = 0.f;
#pragma unroll
          for (int i = 0; i < CHUNKS; ++i) {
            const int row = i * CHUNK + (lane & 15);
            a_off[i] = min(row, max(ti.rows - 1, 0)) * (int)g.a_s_rs;
            a0[i] = i < chunks ? __ldg(as + a_off[i]) : 0.f;
            a1[i] = i < chunks && kblocks > 1 ? __ldg(as + a_off[i] + g.a_s_ks) : 0.f;
            a2[i] = 0.f;
          }
          uint64_t acc[CHUNKS][CHUNK / 2];
#pragma unroll
          for (int i = 0; i < CHUNKS; ++i)
#pragma unroll
            for (int j = 0; j < CHUNK / 2; ++j) acc[i][j] = 0ull;
          for (int kb = 0; kb < kblocks; ++kb, ++it) {
            const int b = it % C::TMEM_BUFS;
            if (kb + 2 < kblocks) {
#pragma unroll
              for (int i = 0; i < CHUNKS; ++i)
                if (i < chunks) a2[i] = __ldg(as + (long long)(kb + 2) * g.a_s_ks + a_off[i]);
              b2 = __ldg(bs + kb + 2);
            }
            if (!mbar_wait(done_bar(it % C::STAGES), (it / C::STAGES) & 1u, abort_flag, limit)) {
              ok = false;
              break;
            }
            tc_fence_after();
#pragma unroll
            for (int i0 = 0; i0 < CHUNKS; i0 += 2) {   // two chunks in flight
              uint32_t v[2][CHUNK];
#pragma unroll
              for (int i = 0; i < 2; ++i)
                if (i0 + i < chunks) tmem_ld16(lane_addr + (uint32_t)(b * BN + wg * BM + (i0 + i) * CHUNK), v[i]);
#pragma unroll
              for (int i = 0; i < 2; ++i)
                if (i0 + i < chunks) tmem_ld_wait16(v[i]);
              if (i0 + 2 >= CHUNKS) {
                tc_fence_before();
                __syncwarp();
                if (lane == 0) mbar_arrive(tempty_bar(b));
              }
#pragma unroll
              for (int i = 0; i < 2; ++i) {
                if (i0 + i < chunks) {
                  const float sc = a0[i0 + i] * b0;
#pragma unroll
                  for (int j = 0; j < CHUNK / 2; ++j)
                    fma2(acc[i0 + i][j], v[i][2 * j], v[i][2 * j + 1],
                         pack2(__shfl_sync(0xffffffffu, sc, 2 * j), __shfl_sync(0xffffffffu, sc, 2 * j + 1)));
                }
              }
            }
#pragma unroll
            for (int i = 0; i < CHUNKS; ++i) {
              a0[i] = a1[i];
              a1[i] = a2[i];
            }
            b0 = b1;
            b1 = b2;
          }
          // the staging tile looks as in the other form; the epilogue warps do not know the difference
          if (!ok || !mbar_wait(sfree_bar, (tile_no & 1u) ^ 1u, abort_flag, limit)) {
            ok = false;
            break;
          }
          OutT* scol = reinterpret_cast<OutT*>(staging) + wg * BM + r;
#pragma unroll
          for (int i = 0; i < CHUNKS; ++i) {
            if (i < chunks) {
              float row_w = 1.f;
              if constexpr (MODE == DLB_EPI_SCATTER_WEIGHT) {
                const int row = i * CHUNK + (lane & 15);
                if (row < ti.rows) row_w = g.weights[g.sorted_idx[ti.row0 + row]];
              }
#pragma unroll
              for (int j = 0; j < CHUNK; ++j) {
                float lo, hi;
                unpack2(acc[i][j / 2], lo, hi);
                float x = j & 1 ? hi : lo;
                if constexpr (MODE == DLB_EPI_SCATTER_WEIGHT) x *= __shfl_sync(0xffffffffu, row_w, j);
                scol[(i * CHUNK + j) * (C::STAGING_ROW_BYTES / 2)] = from_f32<OutT>(x);
              }
            }
          }
          asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
          __syncwarp();
          if (lane == 0) mbar_arrive(staged_bar);
          continue;
        }
      }
      uint64_t acc2[COLS / 2];            // COLS fp32 accumulators, packed in pairs
#pragma unroll
      for (int j = 0; j < COLS / 2; ++j) acc2[j] = 0ull;
      // row / weight of the scatter epilogue, fetched now so that the two dependent loads are
      // long done when the tile's last K block arrives
      long long crow = p;
      float row_w = 1.f;
      if constexpr (MODE == DLB_EPI_SCATTER_WEIGHT) {
        if (row_ok) {
          crow = g.sorted_idx[p];
          row_w = g.weights[crow];
        }
      }

      // scales are fetched two K blocks ahead: under full TMA load an L2 round trip can take
      // longer than one K block
      float a_sc = __ldg(as_ptr), b_sc = __ldg(bs_ptr);
      float a_n1 = 0.f, b_n1 = 0.f;
      if (kblocks > 1) {
        a_n1 = __ldg(as_ptr + g.a_s_ks);
        b_n1 = __ldg(bs_ptr + 1);
      }
      // Two 32-column staging buffers: while one is folded into the accumulators, the load of the next 32 columns (or of
      // the next K block's first 32) is in flight into the other.  This and the early questions for the barriers (here and
      // in the MMA warp) took 8192 x 4096 x 7168 from 287 to 257 us in repeated passes at the power limit (1675 -> 1869
      // TFLOP/s, 1600 -> 1480 MHz), 4096 x 7168 x 2048 from 84 to 76, 8192 x 24576 x 1536 from 405 to 369; the promotion
      // warp's question alone is two thirds of that.  (With whole-warp answers 247, 73 and 362.)
      constexpr int CH = COLS / 32;      // 32-column chunks per thread and K block (1, 2 or 4)
      uint32_t stage[2][32];
      bool pending = false;              // first chunk of the current K block already issued
      for (int kb = 0; kb < kblocks && ok; ++kb, ++it) {
        const int b = it % C::TMEM_BUFS;
        const uint32_t buf_addr = lane_addr + (uint32_t)(b * BN + col0);
        float a_n2 = 0.f, b_n2 = 0.f;
        if (kb + 2 < kblocks) {
          a_n2 = __ldg(as_ptr + (long long)(kb + 2) * g.a_s_ks);
          b_n2 = __ldg(bs_ptr + kb + 2);
        }
        if (!pending) {
          if (!mbar_wait(done_bar(it % C::STAGES), (it / C::STAGES) & 1u, abort_flag, limit)) {
            ok = false;
            break;
          }
          tc_fence_after();
          tmem_ld32(buf_addr, stage[0]);
        }
        pending = false;
        const float scf = a_sc * b_sc;
        const uint64_t sc = pack2(scf, scf);
        const int nb = (it + 1) % C::TMEM_BUFS;
        const uint32_t next_done = done_bar((it + 1) % C::STAGES), next_phase = ((it + 1) / C::STAGES) & 1u;
        bool next_full = false;
#pragma unroll
        for (int q = 0; q < CH; ++q) {
          tmem_ld_wait(stage[q & 1]);
          if (q < CH - 1) {
            tmem_ld32(buf_addr + (q + 1) * 32, stage[(q + 1) & 1]);
            // the next K block's accumulator is asked about under the FMAs below
            if (q == CH - 2) next_full = mbar_test(next_done, next_phase);
          } else {
            // every column of this accumulator is in registers: hand it back to the MMA warp
            tc_fence_before();
            __syncwarp();
            if (lane == 0) {
              if (rank == 0) mbar_arrive(tempty_bar(b));
              else mbar_arrive_cluster_relaxed(mapa(tempty_bar(b), 0));
            }
            if (CH > 1 && kb + 1 < kblocks) {
              if (!__all_sync(WHOLE_WARP, next_full) && !mbar_wait(next_done, next_phase, abort_flag, limit)) {
                ok = false;
              } else {
                tc_fence_after();
                tmem_ld32(lane_addr + (uint32_t)(nb * BN + col0), stage[0]);
                pending = true;
              }
            }
          }
#pragma unroll
          for (int j = 0; j < 16; ++j) fma2(acc2[q * 16 + j], stage[q & 1][2 * j], stage[q & 1][2 * j + 1], sc);
        }
        if (!ok) {
          tmem_ld_wait_plain();
          break;
        }
        a_sc = a_n1;
        b_sc = b_n1;
        a_n1 = a_n2;
        b_n1 = b_n2;
      }
      if (!ok) break;

      // ---- hand the tile over ------------------------------------------------
      float acc[COLS];
#pragma unroll
      for (int j = 0; j < COLS / 2; ++j) unpack2(acc2[j], acc[2 * j], acc[2 * j + 1]);
      if constexpr (MODE == DLB_EPI_SCATTER_WEIGHT) {
#pragma unroll
        for (int j = 0; j < COLS; ++j) acc[j] *= row_w;
      }
      if constexpr (STAGED) {
        // the staging tile must have been emptied by the epilogue warps (previous tile)
        if (!mbar_wait(sfree_bar, (tile_no & 1u) ^ 1u, abort_flag, limit)) {
          ok = false;
          break;
        }
        uint8_t* srow = staging + r * C::STAGING_ROW_BYTES + col0 * 2;
#pragma unroll
        for (int j = 0; j < COLS; j += 8) {
          uint4 v;
          v.x = Pack<OutT>::two(acc[j], acc[j + 1]);
          v.y = Pack<OutT>::two(acc[j + 2], acc[j + 3]);
          v.z = Pack<OutT>::two(acc[j + 4], acc[j + 5]);
          v.w = Pack<OutT>::two(acc[j + 6], acc[j + 7]);
          *reinterpret_cast<uint4*>(srow + j * 2) = v;
        }
        // the rows leave through the async proxy (bulk copies): order these writes before it
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        __syncwarp();
        if (lane == 0) mbar_arrive(staged_bar);
        if constexpr (SELF_DRAIN) {
          if (!mbar_wait(staged_bar, tile_no & 1u, abort_flag, limit)) break;   // all promotion warps' parts are there
          store_rows(ti, warp);
          __syncwarp();
          if (lane == 0) mbar_arrive(sfree_bar);
        }
      } else {
        if (row_ok) {
          OutT* dst = reinterpret_cast<OutT*>(g.c) + crow * g.ldc + ti.n0 + col0;
          store_row<OutT, COLS>(dst, acc, min(COLS, g.n - ti.n0 - col0));   // n % 8 == 0
        }
      }
    }
  }

  // ---- teardown ----------------------------------------------------------------
  start_successor();
  tc_fence_before();
  __syncthreads();
  if constexpr (PAIR) cluster_sync();   // no CTA leaves while its partner may still signal its barriers
  if (threadIdx.x == 0 && *abort_flag != 0 && g.status != nullptr) atomicExch(g.status, DLB_STATUS_TIMEOUT);
  if (warp == MMA_WARP) {
    __syncwarp();
    tc_fence_after();
    if constexpr (PAIR)
      asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(TMEM_COLS) : "memory");
    else
      asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(TMEM_COLS) : "memory");
  }
}

template <int BN, int MODE, typename OutT, int CTAS = 1, bool SWAP = false>
int launch_one(const CUtensorMap& ma, const CUtensorMap& ma16, const CUtensorMap& mb, const GemmArgs& g, int grid,
               cudaStream_t st) {
  auto kern = gemm_fp8_kernel<BN, MODE, OutT, CTAS, SWAP>;
  constexpr int SMEM = Cfg<BN, CTAS>::SMEM_BYTES;
  static bool configured[64] = {};
  int dev = 0;
  cudaGetDevice(&dev);
  if (dev < 64 && !configured[dev]) {
    int rc = check_cuda(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM),
                        "cudaFuncSetAttribute(gemm_fp8_kernel)");
    if (rc != DLB_OK) return rc;
    configured[dev] = true;
  }
  after_predecessor(kern, grid, NUM_THREADS, SMEM, st, CTAS)(ma, ma16, mb, g);
  DLB_CHECK_LAUNCH("gemm_fp8_kernel");
  count_launch();
  return DLB_OK;
}

template <int MODE>
int launch_typed(int bn, int ctas, bool swap, int c_dtype, const CUtensorMap& ma, const CUtensorMap& ma16,
                 const CUtensorMap& mb, const GemmArgs& g, int grid, cudaStream_t st) {
  if (ctas == 2) {
    // pairs exist for 256-wide tiles with a 16-bit output (the ones that go through the staging tile)
    if (bn == 256 && c_dtype == DLB_BF16) return launch_one<256, MODE, __nv_bfloat16, 2>(ma, ma16, mb, g, grid, st);
    if (bn == 256 && c_dtype == DLB_F16) return launch_one<256, MODE, __half, 2>(ma, ma16, mb, g, grid, st);
    return fail(DLB_ERR_INVALID, "256-row tiles need 256-wide tiles and a 16-bit output");
  }
  if (bn == 256) {
    if (swap && c_dtype == DLB_BF16) return launch_one<256, MODE, __nv_bfloat16, 1, true>(ma, ma16, mb, g, grid, st);
    if (swap && c_dtype == DLB_F16) return launch_one<256, MODE, __half, 1, true>(ma, ma16, mb, g, grid, st);
    if (c_dtype == DLB_BF16) return launch_one<256, MODE, __nv_bfloat16>(ma, ma16, mb, g, grid, st);
    if (c_dtype == DLB_F16) return launch_one<256, MODE, __half>(ma, ma16, mb, g, grid, st);
    if constexpr (MODE != DLB_EPI_SWIGLU_QUANT)
      if (c_dtype == DLB_F32) return launch_one<256, MODE, float>(ma, ma16, mb, g, grid, st);
  } else {
    if constexpr (MODE != DLB_EPI_SWIGLU_QUANT) {
      if (bn == 64 && c_dtype == DLB_BF16) return launch_one<64, MODE, __nv_bfloat16>(ma, ma16, mb, g, grid, st);
      if (bn == 64 && c_dtype == DLB_F16) return launch_one<64, MODE, __half>(ma, ma16, mb, g, grid, st);
      if (c_dtype == DLB_BF16) return launch_one<128, MODE, __nv_bfloat16>(ma, ma16, mb, g, grid, st);
      if (c_dtype == DLB_F16) return launch_one<128, MODE, __half>(ma, ma16, mb, g, grid, st);
      if (c_dtype == DLB_F32) return launch_one<128, MODE, float>(ma, ma16, mb, g, grid, st);
    }
  }
  return fail(DLB_ERR_INVALID, "unsupported output dtype %d for this GEMM epilogue", c_dtype);
}

}  // namespace
}  // namespace dlb

using namespace dlb;

extern "C" int dlb_fp8_gemm(const void* a, const void* b, const float* a_s, int64_t a_s_row_stride,
                            int64_t a_s_kb_stride, const float* b_s, void* c, int c_dtype, int64_t m, int64_t n,
                            int64_t k, int tile_rows, int32_t* status, void* stream) {
  DLB_REQUIRE(m >= 0 && n > 0 && k > 0, DLB_ERR_INVALID, "fp8_gemm: bad sizes m=%lld n=%lld k=%lld", (long long)m,
              (long long)n, (long long)k);
  DLB_REQUIRE(k % 128 == 0, DLB_ERR_INVALID, "fp8_gemm: k=%lld must be a multiple of 128", (long long)k);
  DLB_REQUIRE(n % 8 == 0, DLB_ERR_INVALID, "fp8_gemm: n=%lld must be a multiple of 8", (long long)n);
  DLB_REQUIRE(m < (1ll << 31) && n < (1ll << 31) && k < (1ll << 31), DLB_ERR_INVALID, "fp8_gemm: size too large");
  if (m == 0) return DLB_OK;
  DLB_REQUIRE(a && b && a_s && b_s && c, DLB_ERR_INVALID, "fp8_gemm: null pointer");
  DLB_REQUIRE(((uintptr_t)a % 16 == 0) && ((uintptr_t)b % 16 == 0) && ((uintptr_t)c % 16 == 0), DLB_ERR_INVALID,
              "fp8_gemm: a, b and c must be 16-byte aligned");
  int rc = check_device();
  if (rc != DLB_OK) return rc;
  CUtensorMap ma, mb;
  if ((rc = make_map(&ma, a, (uint64_t)m, (uint64_t)k)) != DLB_OK) return rc;
  DLB_REQUIRE(tile_rows == 0 || tile_rows == 128 || tile_rows == 256, DLB_ERR_INVALID,
              "fp8_gemm: tile_rows must be 0 (choose), 128 or 256");
  const int sms = sm_count();
  // Pairs of CTAs only on request: they move a third less through L2 and shared memory, but what bounds a K block is the
  // hand-over between the MMA warp and the promotion warps, which crosses CTAs there: 8192 x 4096 x 7168 252 us against 247,
  // 4096 x 7168 x 2048 75 against 73, 64 groups of about 256 rows 943 against 830 (tiles of 256 rows fill worse).
  const int ctas = tile_rows == 256 ? 2 : 1;
  const int m_tiles = (int)ceil_div(m, (int64_t)(ctas * BM));
  int bn = 256;
  if (ctas == 1) bn = fp8_tile_width(m_tiles, m_tiles, n, sms, c_dtype != DLB_F32);
  if ((rc = make_map_box(&mb, b, (uint64_t)n, (uint64_t)k, bn < 128 ? bn : 128)) != DLB_OK) return rc;
  GemmArgs g = {};
  g.a_s = a_s;
  g.a_s_rs = a_s_row_stride;
  g.a_s_ks = a_s_kb_stride;
  g.b_s = b_s;
  g.b_s_es = 0;
  g.c = c;
  g.ldc = n;
  g.tiles = nullptr;
  g.m = (int)m;
  g.n = (int)n;
  g.k = (int)k;
  g.num_m_tiles_static = m_tiles;
  g.num_n_tiles = (int)ceil_div(n, bn);
  g.status = status;
  g.timeout_cycles = wait_limit_cycles(DEFAULT_TIMEOUT_CYCLES);
  g.withhold_loads = withhold_loads() ? 1 : 0;
  g.m_band = tile_band(BM * ctas, g.num_n_tiles);
  const long long total = (long long)m_tiles * g.num_n_tiles;
  const int workers = sms / ctas;
  const int grid = ctas * (int)(total < workers ? total : workers);
  return launch_typed<DLB_EPI_STORE>(bn, ctas, false, c_dtype, ma, ma, mb, g, grid, (cudaStream_t)stream);
}

// n_begin, n_count: the window of output columns this launch computes (whole tiles of 256; 0, n = everything);
// sm_margin: SMs left free for kernels of other streams (0 = use them all).
static int moe_grouped_gemm(const void* a, const float* a_s, int64_t rows_a, const void* b, const float* b_s,
                            int num_local_experts, int64_t n, int64_t k, const int32_t* tiles, int max_tiles,
                            int tile_rows, int epilogue, void* c, int c_dtype, int64_t ldc, float* q_scale,
                            int quant_mode, float quant_eps, const int64_t* sorted_idx, const float* weights,
                            int32_t* status, void* stream, int64_t n_begin, int64_t n_count, int sm_margin) {
  DLB_REQUIRE(rows_a >= 0 && n > 0 && k > 0 && num_local_experts > 0 && max_tiles >= 0, DLB_ERR_INVALID,
              "grouped_gemm: bad sizes rows=%lld n=%lld k=%lld experts=%d", (long long)rows_a, (long long)n,
              (long long)k, num_local_experts);
  DLB_REQUIRE(k % 128 == 0, DLB_ERR_INVALID, "grouped_gemm: k=%lld must be a multiple of 128", (long long)k);
  DLB_REQUIRE(n % 128 == 0, DLB_ERR_INVALID, "grouped_gemm: n=%lld must be a multiple of 128", (long long)n);
  DLB_REQUIRE(rows_a < (1ll << 31) && (long long)num_local_experts * n < (1ll << 31) && k < (1ll << 31),
              DLB_ERR_INVALID, "grouped_gemm: size too large");
  if (rows_a == 0 || max_tiles == 0) return DLB_OK;
  DLB_REQUIRE(a && a_s && b && b_s && c && tiles, DLB_ERR_INVALID, "grouped_gemm: null pointer");
  DLB_REQUIRE(((uintptr_t)a % 16 == 0) && ((uintptr_t)b % 16 == 0) && ((uintptr_t)c % 16 == 0) &&
                  ((uintptr_t)tiles % 16 == 0),
              DLB_ERR_INVALID, "grouped_gemm: a, b, c and tiles must be 16-byte aligned");
  int rc = check_device();
  if (rc != DLB_OK) return rc;
  CUtensorMap ma, ma16, mb;
  if ((rc = make_map(&ma, a, (uint64_t)rows_a, (uint64_t)k)) != DLB_OK) return rc;
  const bool window = n_begin != 0 || n_count != n;
  DLB_REQUIRE(n_begin >= 0 && n_count > 0 && n_begin + n_count <= n && n_begin % 256 == 0 &&
                  (n_count % 256 == 0 || n_begin + n_count == n),
              DLB_ERR_INVALID, "grouped_gemm: column window [%lld, +%lld) of n=%lld must consist of whole 256-column tiles",
              (long long)n_begin, (long long)n_count, (long long)n);
  DLB_REQUIRE(!window || epilogue != DLB_EPI_SWIGLU_QUANT, DLB_ERR_INVALID,
              "grouped_gemm: the swiglu epilogue pairs gate and up columns and takes no column window");
  DLB_REQUIRE(sm_margin >= 0 && sm_margin < sm_count(), DLB_ERR_INVALID, "grouped_gemm: sm_margin=%d", sm_margin);
  const int sms = sm_count() - sm_margin;
  GemmArgs g = {};
  g.a_s = a_s;
  g.a_s_rs = k / 128;
  g.a_s_ks = 1;
  g.b_s = b_s;
  g.b_s_es = (n / 128) * (k / 128);
  g.c = c;
  g.ldc = ldc;
  g.q_scale = q_scale;
  g.quant_mode = quant_mode;
  g.quant_eps = quant_eps;
  g.tiles = reinterpret_cast<const int4*>(tiles);
  g.m = (int)rows_a;
  g.n = (int)n;
  g.k = (int)k;
  g.n_half = (int)(n / 2);
  g.sorted_idx = reinterpret_cast<const long long*>(sorted_idx);
  g.weights = weights;
  g.status = status;
  g.timeout_cycles = wait_limit_cycles(DEFAULT_TIMEOUT_CYCLES);
  g.withhold_loads = withhold_loads() ? 1 : 0;
  DLB_REQUIRE(tile_rows == 128 || tile_rows == 256, DLB_ERR_INVALID, "grouped_gemm: tile_rows must be 128 or 256");
  const int ctas = tile_rows / BM;
  int bn = 256;
  if (epilogue == DLB_EPI_SWIGLU_QUANT) {
    DLB_REQUIRE(n % 256 == 0, DLB_ERR_INVALID, "grouped_gemm: swiglu epilogue needs n %% 256 == 0 (n=%lld)",
                (long long)n);
    DLB_REQUIRE(q_scale != nullptr, DLB_ERR_INVALID, "grouped_gemm: swiglu epilogue needs q_scale");
    DLB_REQUIRE(ldc % 16 == 0, DLB_ERR_INVALID, "grouped_gemm: ldc must be a multiple of 16 for e4m3 output");
    g.num_n_tiles = (int)(n / 256);
  } else {
    DLB_REQUIRE(epilogue == DLB_EPI_STORE || epilogue == DLB_EPI_SCATTER_WEIGHT, DLB_ERR_INVALID,
                "grouped_gemm: unknown epilogue %d", epilogue);
    if (epilogue == DLB_EPI_SCATTER_WEIGHT)
      DLB_REQUIRE(sorted_idx && weights, DLB_ERR_INVALID, "grouped_gemm: scatter epilogue needs sorted_idx and weights");
    DLB_REQUIRE(ldc % 8 == 0, DLB_ERR_INVALID, "grouped_gemm: ldc must be a multiple of 8");
    if (!window && ctas == 1)
      bn = fp8_tile_width(max_tiles, likely_tiles(rows_a, num_local_experts, max_tiles), n, sms, c_dtype != DLB_F32);
    g.num_n_tiles = (int)ceil_div(n_count, bn);
    g.n_tile0 = (int)(n_begin / bn);
  }
  if ((rc = make_map_box(&mb, b, (uint64_t)num_local_experts * (uint64_t)n, (uint64_t)k, bn < 128 ? bn : 128)) != DLB_OK)
    return rc;
  // A rule on the average, the experts' counts are on the device.  Decode step of 128 tokens, 256 experts, 7168 x 2048, 540 ->
  // 449 us, of 32 experts (32 rows each on average), 4096 x 2048, 210 -> 198; layer of 200
  // tokens, 64 experts, top-4, 115 -> 108, of one token, 8 experts 54 -> 50.  At 62 rows on average the plain kernel is 6 %
  // ahead, and a kernel that can do both is 7 % slower on large problems that never do.
  // rows_a is the number of rows of A, which in the masked layout is the layout's size and not the few rows in use: the split
  // decode steps (several ranks, FusedMoELowLatency.experts) therefore run the plain kernel.
  const bool swap = bn == 256 && ctas == 1 && c_dtype != DLB_F32 && rows_a <= 32ll * num_local_experts;
  ma16 = ma;
  if (swap && (rc = make_map_box(&ma16, a, (uint64_t)rows_a, (uint64_t)k, CHUNK)) != DLB_OK) return rc;
  g.m_band = tile_band(BM * ctas, g.num_n_tiles);
  const long long total = (long long)max_tiles * g.num_n_tiles;
  const int workers = sms / ctas;
  const int grid = ctas * (int)(total < workers ? total : workers);
  cudaStream_t st = (cudaStream_t)stream;
  if (epilogue == DLB_EPI_STORE) return launch_typed<DLB_EPI_STORE>(bn, ctas, swap, c_dtype, ma, ma16, mb, g, grid, st);
  if (epilogue == DLB_EPI_SCATTER_WEIGHT)
    return launch_typed<DLB_EPI_SCATTER_WEIGHT>(bn, ctas, swap, c_dtype, ma, ma16, mb, g, grid, st);
  return launch_typed<DLB_EPI_SWIGLU_QUANT>(bn, ctas, swap, c_dtype, ma, ma16, mb, g, grid, st);
}

extern "C" int dlb_moe_grouped_gemm(const void* a, const float* a_s, int64_t rows_a, const void* b, const float* b_s,
                                    int num_local_experts, int64_t n, int64_t k, const int32_t* tiles, int max_tiles,
                                    int tile_rows, int epilogue, void* c, int c_dtype, int64_t ldc, float* q_scale,
                                    int quant_mode, float quant_eps,
                                    const int64_t* sorted_idx, const float* weights, int32_t* status, void* stream) {
  return moe_grouped_gemm(a, a_s, rows_a, b, b_s, num_local_experts, n, k, tiles, max_tiles, tile_rows, epilogue, c,
                          c_dtype, ldc, q_scale, quant_mode, quant_eps, sorted_idx, weights, status, stream, 0, n, 0);
}

extern "C" int dlb_moe_grouped_gemm_window(const void* a, const float* a_s, int64_t rows_a, const void* b,
                                           const float* b_s, int num_local_experts, int64_t n, int64_t k,
                                           const int32_t* tiles, int max_tiles, int tile_rows, int epilogue, void* c,
                                           int c_dtype, int64_t ldc, float* q_scale, int quant_mode, float quant_eps,
                                           const int64_t* sorted_idx, const float* weights, int32_t* status,
                                           void* stream, int64_t n_begin, int64_t n_count, int sm_margin) {
  return moe_grouped_gemm(a, a_s, rows_a, b, b_s, num_local_experts, n, k, tiles, max_tiles, tile_rows, epilogue, c,
                          c_dtype, ldc, q_scale, quant_mode, quant_eps, sorted_idx, weights, status, stream, n_begin,
                          n_count, sm_margin);
}
