// Shared pieces of the tcgen05 GEMM kernels (sm_100a): mbarrier / TMA / tcgen05 PTX wrappers with bounded
// waits, shared-memory operand descriptors, tensor-map construction.
#pragma once
#include <cuda.h>

#include "common.cuh"

namespace dlb {
namespace {

constexpr int UMMA_BK_BYTES = 128;   // one K block = one 128-byte swizzle row per operand row

// ---- PTX wrappers ------------------------------------------------------------
__device__ __forceinline__ uint32_t smem_u32(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }

__device__ __forceinline__ void mbar_init(uint32_t bar, uint32_t count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bar), "r"(count) : "memory");
}
__device__ __forceinline__ void mbar_expect_tx(uint32_t bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
}
__device__ __forceinline__ void mbar_arrive(uint32_t bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory");
}
// One poll of the barrier.  The suspend-time hint lets the hardware park the warp until the
// phase completes (or the hint, in ns, runs out) instead of spinning: a spinning role would
// take issue slots from the promotion warps that share its scheduler.
__device__ __forceinline__ uint32_t mbar_try_wait(uint32_t bar, uint32_t parity) {
  uint32_t ok;
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2, %3;\n\t"
      "selp.u32 %0, 1, 0, p;\n\t}"
      : "=r"(ok)
      : "r"(bar), "r"(parity), "r"(1000000u)
      : "memory");
  return ok;
}
// The same without waiting: whether the phase has completed, as this lane sees it.  A role asks for its next barrier while it
// still has work of the current one to issue, so that the answer's latency (100 to 300 cycles beside TMA writes and operand
// reads) is hidden; only where the answer was no does it wait.  Lanes may get different answers, so a warp votes on them
// where it acts as a whole (not here: a vote waits for the answer, 100 x 7168 x 2048 9.0 -> 9.7 us).
__device__ __forceinline__ bool mbar_test(uint32_t bar, uint32_t parity) {
  uint32_t ok;
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "mbarrier.test_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
      "selp.u32 %0, 1, 0, p;\n\t}"
      : "=r"(ok)
      : "r"(bar), "r"(parity)
      : "memory");
  return ok != 0;
}
constexpr uint32_t WHOLE_WARP = 0xffffffffu;
// Bounded wait of a whole warp.  Returns false when the CTA is aborting (set by this or another thread).
// All lanes get the same answer and leave together: tcgen05.ld and its like must find the warp converged, which lanes that
// each went on by their own poll, or by their own look at the abort flag, need not be.  Votes in the place of branches per
// lane: 8192 x 4096 x 7168 246 -> 240 us, expert layer of 4096 tokens, 8 experts, 4096 x 14336, 2052 -> 2022, decode step of
// 128 tokens and 256 experts 458 -> 448 (the promotion warps spill less, too).
// The time limit is counted in SM clock cycles (clock64 is a register read; the global
// nanosecond timer costs hundreds of cycles per read and these waits sit on the critical path
// of every K block).
__device__ __forceinline__ bool mbar_wait(uint32_t bar, uint32_t parity, volatile int* abort_flag,
                                          unsigned long long limit_cycles) {
  if (__all_sync(WHOLE_WARP, mbar_try_wait(bar, parity))) return true;
  long long t0 = 0;
  while (!__all_sync(WHOLE_WARP, mbar_try_wait(bar, parity))) {
    bool stop = *abort_flag != 0;
    const long long now = clock64();
    if (t0 == 0) {
      t0 = now;
    } else if ((unsigned long long)(now - t0) > limit_cycles) {
      *abort_flag = 1;
      stop = true;
    }
    if (__any_sync(WHOLE_WARP, stop)) return false;
  }
  return true;
}

__device__ __forceinline__ void tma_load_2d(uint32_t dst, const CUtensorMap* map, int c0, int c1, uint32_t bar) {
  asm volatile(
      "cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];"
      ::"r"(dst), "l"(map), "r"(c0), "r"(c1), "r"(bar)
      : "memory");
}

// The map's descriptor is on its way before the first load asks for it (it lies among the kernel's parameters).
__device__ __forceinline__ void prefetch_map(const CUtensorMap* map) {
  asm volatile("prefetch.tensormap [%0];" ::"l"(map) : "memory");
}

// Order of the tiles of a persistent launch.  band = 1: n tile by n tile, then the next m tile.  band > 1: bands of that
// many m tiles, each walked n tile by n tile with the m tiles innermost, so that the tiles in flight share their operands: in
// the first order a launch of 112 n tiles holds one or two m tiles at a time, and the weights (117 MB an expert) come from
// DRAM again for every 128 rows.
__device__ __forceinline__ void tile_at(int t, int num_m_tiles, int num_n_tiles, int band, int& m_tile, int& n_tile) {
  if (band <= 1) {
    m_tile = t / num_n_tiles;
    n_tile = t - m_tile * num_n_tiles;
    return;
  }
  const int per_band = band * num_n_tiles;
  const int m0 = t / per_band * band;
  const int l = t - m0 * num_n_tiles;
  const int height = min(band, num_m_tiles - m0);
  n_tile = l / height;
  m_tile = m0 + (l - n_tile * height);
}
// Bands of 4096 rows where a row of tiles has more than 16: 32 m tiles and four or five n tiles in flight, whose rows of A
// (29 MB at k = 7168) stay in L2 while B passes once per band.  Times before -> with bands, repeated passes at the power
// limit: 8192 x 24576 x 4096 FP8 with its quantiser 1280 -> 1056 us, 1000 x 24576 x 7168 291 -> 247, expert layer of 4096
// tokens, 8 experts, 4096 x 14336, 2386 -> 2157, 16-bit groups 32768 x 7168 x 4096 1645 -> 1560.  Bands of 2048 rows are up
// to 3 % slower, of 8192 rows up to 10 % (16-bit: A no longer fits); with 16 n tiles or fewer the first order already holds
// five or more m tiles, and bands measured the same or 4 % slower (16384 x 4096 x 3072).
inline int tile_band(int tile_rows, int num_n_tiles) { return num_n_tiles > 16 ? 4096 / tile_rows : 1; }

// True in exactly one lane of a converged warp.
__device__ __forceinline__ bool elect_one() {
  uint32_t pred;
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "elect.sync _|p, 0xffffffff;\n\t"
      "selp.u32 %0, 1, 0, p;\n\t}"
      : "=r"(pred));
  return pred != 0;
}

__device__ __forceinline__ void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }

__device__ __forceinline__ void tc_commit(uint32_t bar) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar) : "memory");
}

__device__ __forceinline__ void tc_mma_f8(uint32_t d_tmem, uint64_t a_desc, uint64_t b_desc, uint32_t idesc,
                                          uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::f8f6f4 [%0], %1, %2, %3, p;\n\t}"
      ::"r"(d_tmem), "l"(a_desc), "l"(b_desc), "r"(idesc), "r"(accumulate)
      : "memory");
}

// 32 lanes x 32 consecutive columns, one fp32 per register.
__device__ __forceinline__ void tmem_ld32(uint32_t taddr, uint32_t (&v)[32]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x32.b32 "
      "{%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,"
      "%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31}, [%32];"
      : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]),
        "=r"(v[8]), "=r"(v[9]), "=r"(v[10]), "=r"(v[11]), "=r"(v[12]), "=r"(v[13]), "=r"(v[14]), "=r"(v[15]),
        "=r"(v[16]), "=r"(v[17]), "=r"(v[18]), "=r"(v[19]), "=r"(v[20]), "=r"(v[21]), "=r"(v[22]), "=r"(v[23]),
        "=r"(v[24]), "=r"(v[25]), "=r"(v[26]), "=r"(v[27]), "=r"(v[28]), "=r"(v[29]), "=r"(v[30]), "=r"(v[31])
      : "r"(taddr)
      : "memory");
}
// Waits for all of this thread's outstanding tcgen05.ld.  Both staging buffers are listed as
// read-write operands so the compiler cannot schedule arithmetic on them above the wait.
__device__ __forceinline__ void tmem_ld_wait(uint32_t (&a)[32], uint32_t (&b)[32]) {
  asm volatile("tcgen05.wait::ld.sync.aligned;"
               : "+r"(a[0]), "+r"(a[1]), "+r"(a[2]), "+r"(a[3]), "+r"(a[4]), "+r"(a[5]), "+r"(a[6]), "+r"(a[7]),
                 "+r"(a[8]), "+r"(a[9]), "+r"(a[10]), "+r"(a[11]), "+r"(a[12]), "+r"(a[13]), "+r"(a[14]), "+r"(a[15]),
                 "+r"(a[16]), "+r"(a[17]), "+r"(a[18]), "+r"(a[19]), "+r"(a[20]), "+r"(a[21]), "+r"(a[22]),
                 "+r"(a[23]), "+r"(a[24]), "+r"(a[25]), "+r"(a[26]), "+r"(a[27]), "+r"(a[28]), "+r"(a[29]),
                 "+r"(a[30]), "+r"(a[31]), "+r"(b[0]), "+r"(b[1]), "+r"(b[2]), "+r"(b[3]), "+r"(b[4]), "+r"(b[5]),
                 "+r"(b[6]), "+r"(b[7]), "+r"(b[8]), "+r"(b[9]), "+r"(b[10]), "+r"(b[11]), "+r"(b[12]), "+r"(b[13]),
                 "+r"(b[14]), "+r"(b[15]), "+r"(b[16]), "+r"(b[17]), "+r"(b[18]), "+r"(b[19]), "+r"(b[20]),
                 "+r"(b[21]), "+r"(b[22]), "+r"(b[23]), "+r"(b[24]), "+r"(b[25]), "+r"(b[26]), "+r"(b[27]),
                 "+r"(b[28]), "+r"(b[29]), "+r"(b[30]), "+r"(b[31])
               :
               : "memory");
}
__device__ __forceinline__ void tmem_ld_wait(uint32_t (&a)[32]) {
  asm volatile("tcgen05.wait::ld.sync.aligned;"
               : "+r"(a[0]), "+r"(a[1]), "+r"(a[2]), "+r"(a[3]), "+r"(a[4]), "+r"(a[5]), "+r"(a[6]), "+r"(a[7]),
                 "+r"(a[8]), "+r"(a[9]), "+r"(a[10]), "+r"(a[11]), "+r"(a[12]), "+r"(a[13]), "+r"(a[14]), "+r"(a[15]),
                 "+r"(a[16]), "+r"(a[17]), "+r"(a[18]), "+r"(a[19]), "+r"(a[20]), "+r"(a[21]), "+r"(a[22]),
                 "+r"(a[23]), "+r"(a[24]), "+r"(a[25]), "+r"(a[26]), "+r"(a[27]), "+r"(a[28]), "+r"(a[29]),
                 "+r"(a[30]), "+r"(a[31])
               :
               : "memory");
}
__device__ __forceinline__ void tmem_ld_wait_plain() { asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory"); }

// Two fp32 FMAs per instruction (sm_100): d.xy = a.xy * b.xy + d.xy on packed register pairs.
__device__ __forceinline__ void fma2(uint64_t& d, uint32_t a_lo, uint32_t a_hi, uint64_t b) {
  uint64_t a;
  asm("mov.b64 %0, {%1, %2};" : "=l"(a) : "r"(a_lo), "r"(a_hi));
  asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(d) : "l"(a), "l"(b));
}
__device__ __forceinline__ uint64_t pack2(float lo, float hi) {
  uint64_t r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi));
  return r;
}
__device__ __forceinline__ void unpack2(uint64_t v, float& lo, float& hi) {
  asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(v));
}

// One row of the staging tile -> global memory, asynchronously (both addresses 16-byte aligned,
// size a multiple of 16).
__device__ __forceinline__ void bulk_store(void* gdst, uint32_t ssrc, uint32_t bytes) {
  asm volatile("cp.async.bulk.global.shared::cta.bulk_group [%0], [%1], %2;"
               ::"l"(__cvta_generic_to_global(gdst)), "r"(ssrc), "r"(bytes)
               : "memory");
}
__device__ __forceinline__ void bulk_commit() { asm volatile("cp.async.bulk.commit_group;" ::: "memory"); }
// all earlier bulk stores of this thread have read their shared-memory source
__device__ __forceinline__ void bulk_wait_read() { asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory"); }
// all earlier bulk stores of this thread are complete
__device__ __forceinline__ void bulk_wait_all() { asm volatile("cp.async.bulk.wait_group 0;" ::: "memory"); }

// ---- pairs of CTAs (clusters of 2, tcgen05 cta_group::2) ------------------------------------
__device__ __forceinline__ uint32_t cluster_ctarank() {
  uint32_t r;
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
  return r;
}
// address of the same shared-memory location in CTA `rank` of the cluster
__device__ __forceinline__ uint32_t mapa(uint32_t addr, uint32_t rank) {
  uint32_t r;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(addr), "r"(rank));
  return r;
}
__device__ __forceinline__ void mbar_arrive_cluster(uint32_t cluster_addr) {
  asm volatile("mbarrier.arrive.release.cluster.shared::cluster.b64 _, [%0];" ::"r"(cluster_addr) : "memory");
}
// The same for handing an accumulator back: relaxed, it orders no access to shared or global memory and must not publish any.
// Only TMEM reads have to come before it; tcgen05.wait::ld has seen their values arrive, and the tcgen05 fences on both sides
// order them against the MMAs that follow.  A release at cluster scope first waits for all the warp's earlier memory
// operations; one per K block made the FP8 kernel's pairs half as fast (4096 x 7168 x 2048: 870 against 1464 TFLOP/s).  The
// 16-bit kernel's pairs, with one per tile, do not notice (16384 x 4096 x 3072 in 16 groups: 361 us both ways).
__device__ __forceinline__ void mbar_arrive_cluster_relaxed(uint32_t cluster_addr) {
  asm volatile("mbarrier.arrive.relaxed.cluster.shared::cluster.b64 _, [%0];" ::"r"(cluster_addr) : "memory");
}
__device__ __forceinline__ void cluster_sync() {
  asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
  asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
}
// TMA load into this CTA's shared memory, completion counted on the barrier at `cluster_bar` (in the pair
// leader's shared memory)
__device__ __forceinline__ void tma_load_2d_pair(uint32_t dst, const CUtensorMap* map, int c0, int c1,
                                                 uint32_t cluster_bar) {
  asm volatile(
      "cp.async.bulk.tensor.2d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];"
      ::"r"(dst), "l"(map), "r"(c0), "r"(c1), "r"(cluster_bar)
      : "memory");
}
// arrives on the barrier at this offset in both CTAs of the pair once all earlier MMAs have retired
__device__ __forceinline__ void tc_commit_pair(uint32_t bar) {
  asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;"
               ::"r"(bar), "h"((uint16_t)3)
               : "memory");
}

__device__ __forceinline__ void tc_mma_f8_pair(uint32_t d_tmem, uint64_t a_desc, uint64_t b_desc, uint32_t idesc,
                                               uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::2.kind::f8f6f4 [%0], %1, %2, %3, {%5, %5, %5, %5, %5, %5, %5, %5}, p;\n\t}"
      ::"r"(d_tmem), "l"(a_desc), "l"(b_desc), "r"(idesc), "r"(accumulate), "r"(0u)
      : "memory");
}

template <int N> __device__ __forceinline__ void reg_dec() {
  asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(N));
}
template <int N> __device__ __forceinline__ void reg_inc() {
  asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(N));
}

// K-major operand, 128-byte swizzle: rows of 128 B, 8-row groups 1024 B apart.
__device__ __forceinline__ uint64_t make_smem_desc(uint32_t smem_addr) {
  uint64_t d = 0;
  d |= (uint64_t)((smem_addr >> 4) & 0x3fffu);  // start address
  d |= (uint64_t)1 << 16;                        // leading byte offset (unused with swizzle)
  d |= (uint64_t)(1024 >> 4) << 32;              // stride byte offset between 8-row groups
  d |= (uint64_t)1 << 46;                        // descriptor version (Blackwell)
  d |= (uint64_t)2 << 61;                        // SWIZZLE_128B
  return d;
}

// ---- host side -----------------------------------------------------------------
typedef CUresult (*EncodeTiledFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                                  const cuuint64_t*, const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave,
                                  CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

EncodeTiledFn get_encode_fn() {
  static EncodeTiledFn fn = nullptr;
  if (fn == nullptr) {
    void* p = nullptr;
    cudaDriverEntryPointQueryResult qres;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &qres) == cudaSuccess &&
        qres == cudaDriverEntryPointSuccess)
      fn = reinterpret_cast<EncodeTiledFn>(p);
  }
  return fn;
}

// 2-D map over a row-major [rows, k] byte matrix, box = box_rows rows x 128 bytes, 128 B swizzle.
int make_map_box(CUtensorMap* map, const void* base, uint64_t rows, uint64_t k, uint32_t box_rows) {
  EncodeTiledFn enc = get_encode_fn();
  if (enc == nullptr) return fail(DLB_ERR_CUDA, "cuTensorMapEncodeTiled is not available from the driver");
  const cuuint64_t gdim[2] = {k, rows};
  const cuuint64_t gstride[1] = {k};
  const cuuint32_t box[2] = {UMMA_BK_BYTES, box_rows};
  const cuuint32_t estr[2] = {1, 1};
  CUresult r = enc(map, CU_TENSOR_MAP_DATA_TYPE_UINT8, 2, const_cast<void*>(base), gdim, gstride, box, estr,
                   CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                   CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (r != CUDA_SUCCESS) return fail(DLB_ERR_CUDA, "cuTensorMapEncodeTiled failed with CUresult %d", (int)r);
  return DLB_OK;
}

// The operand tiles of the K-major kernels: 128 rows x 128 bytes.
int make_map(CUtensorMap* map, const void* base, uint64_t rows, uint64_t k) {
  return make_map_box(map, base, rows, k, 128);
}

int check_device() {
  static int ok[64] = {};
  int dev = 0;
  cudaGetDevice(&dev);
  if (dev < 64 && ok[dev] == 1) return DLB_OK;
  cudaDeviceProp prop;
  int rc = check_cuda(cudaGetDeviceProperties(&prop, dev), "cudaGetDeviceProperties");
  if (rc != DLB_OK) return rc;
  if (prop.major != 10) return fail(DLB_ERR_UNSUPPORTED, "device %d is sm_%d%d; this library is built for sm_100a only",
                                    dev, prop.major, prop.minor);
  if (dev < 64) ok[dev] = 1;
  return DLB_OK;
}

constexpr unsigned long long DEFAULT_TIMEOUT_CYCLES = 4000000000ull;  // about 2 s per barrier wait

}  // namespace
}  // namespace dlb
