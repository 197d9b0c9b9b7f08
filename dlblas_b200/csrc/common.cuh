// Shared helpers of the dlblas_b200 CUDA extension (sm_100a only).
#pragma once
#include <cuda_bf16.h>
#include <cuda_fp16.h>
#include <cuda_fp8.h>
#include <cuda_runtime.h>
#include <stdint.h>
#include <stdio.h>

#include <utility>

#include "../../include/dlblas_b200.h"

namespace dlb {

// Records the message returned by dlb_last_error_string() (thread local) and
// hands back the code so call sites can `return fail(...)`.
int fail(int code, const char* fmt, ...);

inline int check_cuda(cudaError_t e, const char* what) {
  if (e == cudaSuccess) return DLB_OK;
  return fail(DLB_ERR_CUDA, "%s: %s", what, cudaGetErrorString(e));
}

int sm_count();  // multiprocessors of the current device (cached per device)
void count_launch();  // bumps the per-thread kernel launch counter read by dlb_launch_count()
// limit of one barrier wait in SM clock cycles: the value given to dlb_set_wait_policy(), else `fallback`
unsigned long long wait_limit_cycles(unsigned long long fallback);
bool withhold_loads();  // dlb_set_wait_policy(): the GEMMs' load role issues nothing (makes the waits run out)

#define DLB_CHECK_LAUNCH(name)                                  \
  do {                                                          \
    cudaError_t e__ = cudaGetLastError();                       \
    if (e__ != cudaSuccess) return dlb::check_cuda(e__, name);  \
  } while (0)

#define DLB_REQUIRE(cond, code, ...)                 \
  do {                                               \
    if (!(cond)) return dlb::fail(code, __VA_ARGS__); \
  } while (0)

// ---- launches that overlap ------------------------------------------------- //
// Kernels of one operator follow one another on a stream, and most of them are short: from the end of one to the first
// instructions of the next 1.5 to 2 us pass.  after_predecessor() launches a kernel while its predecessor in the stream is
// still running (programmatic stream serialization); its blocks take up SMs as they become free, and
// wait_for_predecessor(), the first thing that every thread does (after a set-up that touches no global memory), returns when
// the predecessor has completed and its writes are visible.  Only then does a kernel let its own successor be launched, so
// one that starts early knows that everything up to its predecessor's predecessor is complete.  After kernels that know
// nothing of this (torch's, the peer-to-peer ones) the launch waits for their end as always.
// Passes among others, before -> after: expert layer of 64 tokens (six kernels) 36.9 -> 22.8 us, quantiser and GEMM of 100
// rows 16.4 -> 11.9, routing and aligned layout of 20000 tokens 45.1 -> 40.0, 16-bit expert layer of 500 tokens 203 -> 194,
// decode step of 128 tokens and 256 experts 478 -> 465, permutation both ways 525 -> 515.
// A kernel that runs for long and fills the SMs (the GEMMs) calls start_successor() when a block has nothing left but its
// end: with the successor waiting in line from the start, they were 1 to 2 % slower and the short ones no faster.
#ifdef __CUDACC__
__device__ __forceinline__ void start_successor() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
// The answer is always true.  The loads behind it hang on the branch, so that the compiler cannot move those it may take
// for constant (ld.global.nc) in front of the wait.
__device__ __forceinline__ bool wait_for_predecessor(bool then_start_successor = true) {
  uint32_t done;
  asm volatile("griddepcontrol.wait;\n\tmov.u32 %0, 1;" : "=r"(done)::"memory");
  if (then_start_successor) start_successor();
  return done != 0;
}
template <typename... P> struct LaunchAfterPredecessor {
  void (*kernel)(P...);
  dim3 grid, block;
  size_t smem;
  cudaStream_t stream;
  int cluster;
  template <typename... A> cudaError_t operator()(A&&... args) const {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = grid;
    cfg.blockDim = block;
    cfg.dynamicSmemBytes = smem;
    cfg.stream = stream;
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    attr[1].id = cudaLaunchAttributeClusterDimension;
    attr[1].val.clusterDim.x = cluster;
    attr[1].val.clusterDim.y = 1;
    attr[1].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = cluster > 1 ? 2 : 1;
    return cudaLaunchKernelEx(&cfg, kernel, std::forward<A>(args)...);
  }
};
// after_predecessor(kernel, grid, block, shared memory, stream)(arguments); errors as after a <<<>>> launch
template <typename... P>
LaunchAfterPredecessor<P...> after_predecessor(void (*kernel)(P...), dim3 grid, dim3 block, size_t smem,
                                               cudaStream_t stream, int cluster = 1) {
  return {kernel, grid, block, smem, stream, cluster};
}
#endif

__host__ __device__ inline int64_t ceil_div(int64_t a, int64_t b) { return (a + b - 1) / b; }

// Division of n < 2^31 by a divisor that is fixed for a launch, as one multiplication and a shift (Granlund and
// Montgomery, Division by invariant integers using multiplication, 1994): m = ceil(2^(32 + s) / d), s = ceil(log2 d).
// A kernel that walks a matrix by a flat index pays one such division per vector; the compiler's 64-bit division is a
// call of some seventy instructions and was a third of the quantiser's time.
struct FastDiv {
  uint32_t d, m, s;
  FastDiv() = default;
  __host__ explicit FastDiv(uint32_t div) : d(div), s(0) {
    while ((1ull << s) < d) ++s;
    m = (uint32_t)((((1ull << s) - d) << 32) / d + 1);
  }
  __device__ __forceinline__ uint32_t quot(uint32_t n) const { return (__umulhi(n, m) + n) >> s; }
};

// Masked layouts ([experts, rows_per_expert, ...] with only the first masked_m[e] rows of expert e in use) hold a few
// hundred valid rows among tens of thousands in a decode step.  These two helpers let a kernel walk the valid rows only:
// every block builds the running sums of min(masked_m[e], cap) in shared memory (prefix[experts] = their total; warp 0
// scans, all threads of the block must call), then item i of [0, total) is row i - prefix[e] of expert e.
constexpr int MASKED_MAX_EXPERTS = 1024;
#ifdef __CUDACC__
__device__ inline void masked_prefix(const int* __restrict__ masked_m, int experts, int cap, int* prefix) {
  if (threadIdx.x < 32) {
    const int lane = threadIdx.x;
    int carry = 0;
    for (int e0 = 0; e0 < experts; e0 += 32) {
      const int e = e0 + lane;
      const int v = e < experts ? min(max(__ldg(masked_m + e), 0), cap) : 0;
      int incl = v;
#pragma unroll
      for (int d = 1; d < 32; d <<= 1) {
        const int up = __shfl_up_sync(0xffffffffu, incl, d);
        if (lane >= d) incl += up;
      }
      if (e < experts) prefix[e] = carry + incl - v;
      carry += __shfl_sync(0xffffffffu, incl, 31);
    }
    if (lane == 0) prefix[experts] = carry;
  }
  __syncthreads();
}
// the expert that holds item `item` (< prefix[experts]): the last e with prefix[e] <= item
__device__ inline int masked_find(const int* prefix, int experts, int item) {
  int lo = 0, hi = experts;   // invariant: prefix[lo] <= item < prefix[hi]
  while (hi - lo > 1) {
    const int mid = (lo + hi) >> 1;
    if (prefix[mid] <= item) lo = mid; else hi = mid;
  }
  return lo;
}
#endif

// ---- warp helpers -------------------------------------------------------- //
__device__ __forceinline__ float warp_max(float v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, o));
  return v;
}
__device__ __forceinline__ float warp_sum(float v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

// ---- element conversion ---------------------------------------------------- //
template <typename T> __device__ __forceinline__ float to_f32(T v);
template <> __device__ __forceinline__ float to_f32<float>(float v) { return v; }
template <> __device__ __forceinline__ float to_f32<__nv_bfloat16>(__nv_bfloat16 v) { return __bfloat162float(v); }
template <> __device__ __forceinline__ float to_f32<__half>(__half v) { return __half2float(v); }

template <typename T> __device__ __forceinline__ T from_f32(float v);
template <> __device__ __forceinline__ float from_f32<float>(float v) { return v; }
template <> __device__ __forceinline__ __nv_bfloat16 from_f32<__nv_bfloat16>(float v) { return __float2bfloat16_rn(v); }
template <> __device__ __forceinline__ __half from_f32<__half>(float v) { return __float2half_rn(v); }

// The reference clamps before it casts (`tl.clamp(out, fp8_min, fp8_max)`, dlblas/kernels/moe.py:413,
// dlblas/kernels/fp8.py:48): min(max(x, -448), 448) with the non-propagating min / max of the GPU, so a NaN
// (0 / 0 of an all-zero group whose scale is 0) becomes -448 and never reaches the payload.  fmaxf / fminf
// return the non-NaN operand, which reproduces that.
__device__ __forceinline__ float clamp_e4m3(float x) { return fminf(fmaxf(x, -448.f), 448.f); }

// Two fp32 -> packed e4m3x2 (lo in bits 0-7): clamp to +-448, then round to nearest even.
__device__ __forceinline__ uint16_t f32x2_to_e4m3x2(float lo, float hi) {
  uint16_t r;
  asm("cvt.rn.satfinite.e4m3x2.f32 %0, %1, %2;" : "=h"(r) : "f"(clamp_e4m3(hi)), "f"(clamp_e4m3(lo)));
  return r;
}

// silu for the fused silu*up + quantise paths: fast exponential and a 2-ulp divide.  The result
// is multiplied by `up` and rounded to a 16-bit type straight away, so the extra fp32 error only
// shows where the product sits within 2 ulp of a 16-bit rounding boundary.
__device__ __forceinline__ float silu_fast(float g) { return __fdividef(g, 1.f + __expf(-g)); }

// Eight values times the reciprocal of their group's scale -> eight e4m3 bytes.  `inv` is the
// correctly rounded 1 / scale; v * inv is within one fp32 ulp of v / scale.
__device__ __forceinline__ uint2 quant8_rcp(const float (&v)[8], float inv) {
  uint2 r;
  r.x = (uint32_t)f32x2_to_e4m3x2(v[0] * inv, v[1] * inv) | ((uint32_t)f32x2_to_e4m3x2(v[2] * inv, v[3] * inv) << 16);
  r.y = (uint32_t)f32x2_to_e4m3x2(v[4] * inv, v[5] * inv) | ((uint32_t)f32x2_to_e4m3x2(v[6] * inv, v[7] * inv) << 16);
  return r;
}

// ---- packed fp32 pairs (sm_100: two fp32 operations per instruction) --------------- //
__device__ __forceinline__ uint64_t pack_f32x2(float lo, float hi) {
  uint64_t r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi));
  return r;
}
__device__ __forceinline__ uint64_t mul_f32x2(uint64_t a, uint64_t b) {
  uint64_t r;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
__device__ __forceinline__ uint64_t fma_f32x2(uint64_t a, uint64_t b, uint64_t c) {
  uint64_t r;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
  return r;
}
// max that hands a NaN on
__device__ __forceinline__ float max_nan(float a, float b) {
  float r;
  asm("max.NaN.f32 %0, %1, %2;" : "=f"(r) : "f"(a), "f"(b));
  return r;
}

// v / scale -> e4m3, N values (a multiple of 4), bit for bit what a correctly rounded division gives.
// The quotient starts from v * y, y the correctly rounded reciprocal of the scale (one per thread), and is corrected
// twice by its exact remainder; the second correction makes it the correctly rounded quotient (Markstein, Computation
// of elementary functions on the IBM RISC System/6000, 1990).  2.5 instructions per value on packed pairs in place of a
// divide of about ten.  `regular` says that the group holds no NaN and that its scale is far from the ends of the fp32
// range (so no remainder is subnormal); other groups divide.
template <int N>
__device__ __forceinline__ void div_to_e4m3(const float (&v)[N], float scale, bool regular, uint32_t (&out)[N / 4]) {
  if (regular) {
    const float inv = __frcp_rn(scale);
    const uint64_t ny = pack_f32x2(-inv, -inv), s = pack_f32x2(scale, scale);
#pragma unroll
    for (int i = 0; i < N; i += 4) {
      uint32_t half[2];
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        // with -v and -1 / scale: the remainder of a zero is then +0, and the correction -0 keeps the quotient's sign
        const uint64_t na = pack_f32x2(-v[i + 2 * h], -v[i + 2 * h + 1]);
        uint64_t q = mul_f32x2(na, ny);
        q = fma_f32x2(fma_f32x2(q, s, na), ny, q);
        q = fma_f32x2(fma_f32x2(q, s, na), ny, q);
        uint16_t r;
        asm("{\n\t.reg .f32 lo, hi;\n\tmov.b64 {lo, hi}, %1;\n\tcvt.rn.satfinite.e4m3x2.f32 %0, hi, lo;\n\t}"
            : "=h"(r)
            : "l"(q));
        half[h] = r;
      }
      out[i / 4] = half[0] | (half[1] << 16);
    }
  } else {
#pragma unroll
    for (int i = 0; i < N; i += 4)
      out[i / 4] = (uint32_t)f32x2_to_e4m3x2(v[i] / scale, v[i + 1] / scale) |
                   ((uint32_t)f32x2_to_e4m3x2(v[i + 2] / scale, v[i + 3] / scale) << 16);
  }
}
__device__ __forceinline__ bool regular_scale(float scale) { return scale >= 5.4210109e-20f && scale <= 1.8446744e19f; }

__device__ __forceinline__ uint64_t globaltimer_ns() {
  uint64_t t;
  asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
  return t;
}

}  // namespace dlb
