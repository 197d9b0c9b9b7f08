// HBM-bound kernels of the MoE expert path: 1xG FP8 quantisation (optionally fused with
// the token-by-expert permutation), row permutation, silu*up (+ quantisation), and the
// weighted / unweighted combine.  Every thread moves 16-byte vectors; consecutive threads
// touch consecutive vectors of a row, so global accesses are fully coalesced.
#include <algorithm>
#include <type_traits>

#include "common.cuh"
#include "sort.cuh"

namespace dlb {
namespace {

constexpr int THREADS = 256;

template <typename T> struct Vec8 {
  // eight consecutive elements of type T
  static __device__ __forceinline__ void load(const T* p, float (&v)[8]);
  static __device__ __forceinline__ void store(T* p, const float (&v)[8]);
};
template <> struct Vec8<float> {
  static __device__ __forceinline__ void load(const float* p, float (&v)[8]) {
    const float4 a = __ldg(reinterpret_cast<const float4*>(p));
    const float4 b = __ldg(reinterpret_cast<const float4*>(p) + 1);
    v[0] = a.x; v[1] = a.y; v[2] = a.z; v[3] = a.w; v[4] = b.x; v[5] = b.y; v[6] = b.z; v[7] = b.w;
  }
  static __device__ __forceinline__ void store(float* p, const float (&v)[8]) {
    reinterpret_cast<float4*>(p)[0] = make_float4(v[0], v[1], v[2], v[3]);
    reinterpret_cast<float4*>(p)[1] = make_float4(v[4], v[5], v[6], v[7]);
  }
};
template <> struct Vec8<__nv_bfloat16> {
  static __device__ __forceinline__ void load(const __nv_bfloat16* p, float (&v)[8]) {
    const uint4 r = __ldg(reinterpret_cast<const uint4*>(p));
    const __nv_bfloat162* h = reinterpret_cast<const __nv_bfloat162*>(&r);
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const float2 f = __bfloat1622float2(h[i]);
      v[2 * i] = f.x;
      v[2 * i + 1] = f.y;
    }
  }
  static __device__ __forceinline__ void store(__nv_bfloat16* p, const float (&v)[8]) {
    uint4 r;
    __nv_bfloat162* h = reinterpret_cast<__nv_bfloat162*>(&r);
#pragma unroll
    for (int i = 0; i < 4; ++i) h[i] = __floats2bfloat162_rn(v[2 * i], v[2 * i + 1]);
    *reinterpret_cast<uint4*>(p) = r;
  }
};
template <> struct Vec8<__half> {
  static __device__ __forceinline__ void load(const __half* p, float (&v)[8]) {
    const uint4 r = __ldg(reinterpret_cast<const uint4*>(p));
    const __half2* h = reinterpret_cast<const __half2*>(&r);
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const float2 f = __half22float2(h[i]);
      v[2 * i] = f.x;
      v[2 * i + 1] = f.y;
    }
  }
  static __device__ __forceinline__ void store(__half* p, const float (&v)[8]) {
    uint4 r;
    __half2* h = reinterpret_cast<__half2*>(&r);
#pragma unroll
    for (int i = 0; i < 4; ++i) h[i] = __floats2half2_rn(v[2 * i], v[2 * i + 1]);
    *reinterpret_cast<uint4*>(p) = r;
  }
};

// Eight consecutive elements as they lie in memory: a thread can hold several rows' vectors in flight and convert them
// when it needs them.
template <typename T> struct Raw8 {
  static constexpr int WORDS = sizeof(T) / 2;   // 16-byte words
  uint4 w[WORDS];
  __device__ __forceinline__ void load(const T* p) {
#pragma unroll
    for (int i = 0; i < WORDS; ++i) w[i] = __ldg(reinterpret_cast<const uint4*>(p) + i);
  }
  // Zeros when !live.  Volatile: the compiler otherwise sinks a predicated load to the predicated use, and the loads of
  // several rows wait for one another.
  __device__ __forceinline__ void load_if(bool live, const T* p) {
#pragma unroll
    for (int i = 0; i < WORDS; ++i)
      asm volatile(
          "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %5, 0;\n\tmov.b32 %0, 0;\n\tmov.b32 %1, 0;\n\tmov.b32 %2, 0;\n\t"
          "mov.b32 %3, 0;\n\t@p ld.global.nc.L1::no_allocate.v4.b32 {%0, %1, %2, %3}, [%4];\n\t}"
          : "=&r"(w[i].x), "=&r"(w[i].y), "=&r"(w[i].z), "=&r"(w[i].w)
          : "l"(reinterpret_cast<const uint4*>(p) + i), "r"((int)live));
  }
  __device__ __forceinline__ void get(float (&v)[8]) const {
    const T* e = reinterpret_cast<const T*>(w);
#pragma unroll
    for (int i = 0; i < 8; ++i) v[i] = to_f32<T>(e[i]);
  }
};

// absmax over the `lanes` (power of two, <= 32) consecutive lanes that share a group
__device__ __forceinline__ float group_max(float v, int lanes) {
  for (int o = lanes >> 1; o > 0; o >>= 1) v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, o));
  return v;
}

__device__ __forceinline__ float quant_scale(float amax, int mode, float eps) {
  // DLB_QUANT_RECIP_MUL: dlblas/kernels/moe.py:396,410 ; DLB_QUANT_DIV_EPS: dlblas/kernels/fp8.py:46-47
  return mode == DLB_QUANT_RECIP_MUL ? amax * (1.0f / 448.0f) : fmaxf(amax, eps) / 448.0f;
}

// 16 bytes to an address that is 16-byte aligned, or only 8-byte aligned (the C ABI allows that for q)
__device__ __forceinline__ void store16(uint8_t* p, uint4 v) {
  if ((reinterpret_cast<uintptr_t>(p) & 15) == 0) {
    *reinterpret_cast<uint4*>(p) = v;
  } else {
    reinterpret_cast<uint2*>(p)[0] = make_uint2(v.x, v.y);
    reinterpret_cast<uint2*>(p)[1] = make_uint2(v.z, v.w);
  }
}

// One thread per 16 elements (one 16-byte store per destination row); a quantisation group of G elements spans G/16 lanes.
// Bound by memory once the division is out of the way (div_to_e4m3) and the flat index needs no 64-bit division.
template <typename T>
__global__ void __launch_bounds__(THREADS) quant_fp8_kernel(const T* __restrict__ x, uint32_t total, FastDiv vec_per_row,
                                                            long long ldx, int group_lanes, int mode, float eps,
                                                            uint8_t* __restrict__ q, float* __restrict__ scales,
                                                            long long s_rs, long long s_gs,
                                                            const int* __restrict__ dst_pos, int fanout) {
  if (!wait_for_predecessor()) return;
  const long long k = (long long)vec_per_row.d * 16;
  for (uint32_t u0 = blockIdx.x * THREADS; u0 < total; u0 += gridDim.x * THREADS) {
    const uint32_t u = u0 + threadIdx.x;
    const bool active = u < total;
    const uint32_t row = active ? vec_per_row.quot(u) : 0u;
    const uint32_t cv = active ? u - row * vec_per_row.d : 0u;
    float v[16];
    if (active) {
      Raw8<T> lo, hi;
      const T* src = x + (long long)row * ldx + cv * 16;
      lo.load(src);
      hi.load(src + 8);
      lo.get(*reinterpret_cast<float(*)[8]>(v));
      hi.get(*reinterpret_cast<float(*)[8]>(v + 8));
    } else {
#pragma unroll
      for (int i = 0; i < 16; ++i) v[i] = 0.f;
    }
    float amax = 0.f;
#pragma unroll
    for (int i = 0; i < 16; ++i) amax = max_nan(amax, fabsf(v[i]));
    for (int o = group_lanes >> 1; o > 0; o >>= 1) amax = max_nan(amax, __shfl_xor_sync(0xffffffffu, amax, o));
    const bool has_nan = amax != amax;
    if (__any_sync(0xffffffffu, has_nan)) {   // the scale comes from the values that are numbers
      float m = 0.f;
#pragma unroll
      for (int i = 0; i < 16; ++i) m = fmaxf(m, fabsf(v[i]));
      m = group_max(m, group_lanes);
      if (has_nan) amax = m;
    }
    const float scale = quant_scale(amax, mode, eps);
    if (!active) continue;
    uint32_t packed[4];
    div_to_e4m3<16>(v, scale, !has_nan && regular_scale(scale), packed);
    const uint4 out = make_uint4(packed[0], packed[1], packed[2], packed[3]);
    const bool first = (cv & (group_lanes - 1)) == 0;
    const uint32_t gidx = cv / group_lanes;
    if (dst_pos == nullptr) {
      store16(q + (long long)row * k + cv * 16, out);
      if (first) scales[(long long)row * s_rs + gidx * s_gs] = scale;
    } else {
      const int* dp = dst_pos + (long long)row * fanout;
      for (int j0 = 0; j0 < fanout; j0 += 8) {
        int d[8];
#pragma unroll
        for (int j = 0; j < 8; ++j) d[j] = j0 + j < fanout ? __ldg(dp + j0 + j) : -1;
#pragma unroll
        for (int j = 0; j < 8; ++j) {
          if (d[j] < 0) continue;
          store16(q + (long long)d[j] * k + cv * 16, out);
          if (first) scales[(long long)d[j] * s_rs + gidx * s_gs] = scale;
        }
      }
    }
  }
}

// Row copies: one thread per 16 bytes of a row, plus the row's scales.
__global__ void __launch_bounds__(THREADS) permute_rows_kernel(const uint4* __restrict__ q, FastDiv vec_per_row,
                                                               const float* __restrict__ scales, uint32_t groups,
                                                               uint32_t total, const int* __restrict__ dst_pos, int fanout,
                                                               uint4* __restrict__ out_q, float* __restrict__ out_s) {
  if (!wait_for_predecessor()) return;
  for (uint32_t u = blockIdx.x * THREADS + threadIdx.x; u < total; u += gridDim.x * THREADS) {
    const uint32_t row = vec_per_row.quot(u);
    const uint32_t c = u - row * vec_per_row.d;
    const bool with_scale = scales != nullptr && c < groups;
    uint4 v = make_uint4(0, 0, 0, 0);
    float s = 0.f;
    bool loaded = false;               // rows without any destination are not read at all
    const int* dp = dst_pos + (long long)row * fanout;
    for (int j0 = 0; j0 < fanout; j0 += 8) {
      int d[8];
#pragma unroll
      for (int j = 0; j < 8; ++j) d[j] = j0 + j < fanout ? __ldg(dp + j0 + j) : -1;
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        if (d[j] < 0) continue;
        if (!loaded) {
          v = __ldg(q + u);
          if (with_scale) s = __ldg(scales + (long long)row * groups + c);
          loaded = true;
        }
        out_q[(long long)d[j] * vec_per_row.d + c] = v;
        if (with_scale) out_s[(long long)d[j] * groups + c] = s;
      }
    }
  }
}

template <typename T>
__global__ void __launch_bounds__(THREADS) silu_and_mul_kernel(const T* __restrict__ in, uint32_t total,
                                                               FastDiv vec_per_row, long long ld_in,
                                                               T* __restrict__ out, long long ld_out) {
  if (!wait_for_predecessor()) return;
  const long long n = (long long)vec_per_row.d * 8;
  for (uint32_t u = blockIdx.x * THREADS + threadIdx.x; u < total; u += gridDim.x * THREADS) {
    const uint32_t r = vec_per_row.quot(u);
    const long long row = r, c = (long long)(u - r * vec_per_row.d) * 8;
    float g[8], up[8], o[8];
    Raw8<T> rg, ru;
    rg.load(in + row * ld_in + c);
    ru.load(in + row * ld_in + n + c);
    rg.get(g);
    ru.get(up);
#pragma unroll
    for (int i = 0; i < 8; ++i) o[i] = (g[i] / (1.f + __expf(-g[i]))) * up[i];
    Vec8<T>::store(out + row * ld_out + c, o);
  }
}

// silu(gate) * up, rounded like the reference, then the 1x128 quantisation of the result.  With masked_m (masked
// layout, `experts` experts of rows_per_expert rows) only the valid rows are visited: a decode step holds a few
// hundred of them in a layout of tens of thousands.
template <typename T>
__global__ void __launch_bounds__(THREADS) silu_mul_quant_kernel(const T* __restrict__ in, uint32_t row0, uint32_t rows,
                                                                 FastDiv vec_per_row, int mode, float eps, int round_silu,
                                                                 const int* __restrict__ masked_m, int experts,
                                                                 long long rows_per_expert, uint8_t* __restrict__ q,
                                                                 float* __restrict__ scales) {
  if (!wait_for_predecessor()) return;
  __shared__ int prefix[MASKED_MAX_EXPERTS + 1];
  const long long n = (long long)vec_per_row.d * 8;
  const long long groups = n / 128;
  uint32_t my_rows = rows;
  if (masked_m != nullptr) {
    masked_prefix(masked_m, experts, (int)rows_per_expert, prefix);
    my_rows = (uint32_t)min(max(prefix[experts] - (int)row0, 0), (int)rows);
  }
  const uint32_t total = my_rows * vec_per_row.d;
  for (uint32_t u0 = blockIdx.x * THREADS; u0 < total; u0 += gridDim.x * THREADS) {
    const uint32_t u = u0 + threadIdx.x;
    const bool active = u < total;
    const uint32_t r = active ? vec_per_row.quot(u) : 0u;
    long long row = (long long)row0 + r;
    const long long c = active ? (long long)(u - r * vec_per_row.d) * 8 : 0;
    if (masked_m != nullptr && active) {
      const int e = masked_find(prefix, experts, (int)row);
      row = (long long)e * rows_per_expert + (row - prefix[e]);
    }
    float h[8];
#pragma unroll
    for (int i = 0; i < 8; ++i) h[i] = 0.f;
    if (active) {
      float g[8], up[8];
      Vec8<T>::load(in + row * 2 * n + c, g);
      Vec8<T>::load(in + row * 2 * n + n + c, up);
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        float s = silu_fast(g[i]);
        if (round_silu) s = to_f32<T>(from_f32<T>(s));
        h[i] = to_f32<T>(from_f32<T>(s * up[i]));
      }
    }
    float amax = 0.f;
#pragma unroll
    for (int i = 0; i < 8; ++i) amax = fmaxf(amax, fabsf(h[i]));
    amax = group_max(amax, 16);
    const float scale = quant_scale(amax, mode, eps);
    if (!active) continue;
    *reinterpret_cast<uint2*>(q + row * n + c) = quant8_rcp(h, 1.0f / scale);
    if (((c / 8) & 15) == 0) scales[row * groups + c / 128] = scale;
  }
}

// The combine kernels: one warp per (token, 256 columns).  A lane has the vectors of up to GATHER_ROWS rows in flight before
// it adds the first one (their addresses do not depend on one another), which is what a sum over a handful of scattered rows
// needs to run at the memory rate; splitting a token's columns over warps keeps the chip busy with few tokens.
template <typename T> constexpr int GATHER_ROWS = sizeof(T) == 4 ? 4 : 8;
// rows in flight for a given top_k: registers that no row needs cost occupancy
template <typename T, typename F> void with_rows_in_flight(int top_k, F&& f) {
  if (top_k <= 2) f(std::integral_constant<int, 2>());
  else if (top_k <= 4 || GATHER_ROWS<T> == 4) f(std::integral_constant<int, 4>());
  else f(std::integral_constant<int, GATHER_ROWS<T>>());
}

template <typename T, int R, typename IdT>
__global__ void __launch_bounds__(THREADS) sum_topk_kernel(const T* __restrict__ y, uint32_t units, FastDiv chunks,
                                                           int top_k, long long h, const IdT* __restrict__ ids,
                                                           long long id_lo, long long id_hi, int skip_unrouted,
                                                           T* __restrict__ out) {
  if (!wait_for_predecessor()) return;
  const int lane = threadIdx.x & 31;
  for (uint32_t w = blockIdx.x * (THREADS / 32) + (threadIdx.x >> 5); w < units; w += gridDim.x * (THREADS / 32)) {
    const uint32_t t = chunks.quot(w);
    const long long c = (long long)(w - t * chunks.d) * 256 + lane * 8;
    unsigned live = 0xffffffffu;                       // bit j: slot j contributes
    if (ids != nullptr) {
      bool in_range = false;
      if (lane < top_k) {                              // top_k <= 32 (checked by the caller)
        const long long id = (long long)ids[(long long)t * top_k + lane];
        in_range = id >= id_lo && id < id_hi;
      }
      live = __ballot_sync(0xffffffffu, in_range);
    }
    if (top_k < 32) live &= (1u << top_k) - 1u;
    if (live == 0u && skip_unrouted) continue;         // rows nobody routed to are left alone
    if (c >= h) continue;
    const T* src = y + (long long)t * top_k * h + c;
    float acc[8];
#pragma unroll
    for (int i = 0; i < 8; ++i) acc[i] = 0.f;
    for (int j0 = 0; j0 < top_k; j0 += R) {
      Raw8<T> raw[R];
#pragma unroll
      for (int j = 0; j < R; ++j) raw[j].load_if((live >> (j0 + j)) & 1u, src + (j0 + j) * h);
#pragma unroll
      for (int j = 0; j < R; ++j) {
        if (!((live >> (j0 + j)) & 1u)) continue;
        float v[8];
        raw[j].get(v);
#pragma unroll
        for (int i = 0; i < 8; ++i) acc[i] += v[i];
      }
    }
    Vec8<T>::store(out + (long long)t * h + c, acc);
  }
}

template <typename T, int R, typename IdxT>
__global__ void __launch_bounds__(THREADS) ep_gather_kernel(const T* __restrict__ in, long long h,
                                                            const IdxT* __restrict__ ids, const IdxT* __restrict__ index,
                                                            const float* __restrict__ weights, uint32_t units,
                                                            FastDiv chunks, int top_k, T* __restrict__ out) {
  if (!wait_for_predecessor()) return;
  const int lane = threadIdx.x & 31;
  for (uint32_t w = blockIdx.x * (THREADS / 32) + (threadIdx.x >> 5); w < units; w += gridDim.x * (THREADS / 32)) {
    const uint32_t t = chunks.quot(w);
    const long long c = (long long)(w - t * chunks.d) * 256 + lane * 8;
    if (c >= h) continue;
    float acc[8];
#pragma unroll
    for (int i = 0; i < 8; ++i) acc[i] = 0.f;
    const long long s0 = (long long)t * top_k;
    for (int j0 = 0; j0 < top_k; j0 += R) {
      bool live[R];
      Raw8<T> raw[R];
      long long row[R];
#pragma unroll
      for (int j = 0; j < R; ++j) {
        live[j] = j0 + j < top_k && (long long)ids[s0 + j0 + j] >= 0;
        row[j] = live[j] ? (long long)index[s0 + j0 + j] : 0;
      }
#pragma unroll
      for (int j = 0; j < R; ++j) raw[j].load_if(live[j], in + row[j] * h + c);
#pragma unroll
      for (int j = 0; j < R; ++j) {
        if (!live[j]) continue;
        const float wt = __ldg(weights + s0 + j0 + j);
        float v[8];
        raw[j].get(v);
#pragma unroll
        for (int i = 0; i < 8; ++i) acc[i] += v[i] * wt;
      }
    }
    Vec8<T>::store(out + (long long)t * h + c, acc);
  }
}

// ep_scatter bookkeeping: exclusive cumsum of the (aligned) per-expert counts and the
// expert id of every row of the contiguous layout.
__global__ void __launch_bounds__(1024) scatter_layout_kernel(const int* __restrict__ counts, int num_experts,
                                                              int* __restrict__ start_loc, int* __restrict__ m_indices,
                                                              long long m_indices_len) {
  if (!wait_for_predecessor()) return;
  extern __shared__ int s_start[];  // [num_experts + 1]
  if (threadIdx.x == 0) {
    int run = 0;
    for (int e = 0; e < num_experts; ++e) {
      s_start[e] = run;
      run += counts[e];
    }
    s_start[num_experts] = run;
  }
  __syncthreads();
  for (int e = threadIdx.x; e < num_experts; e += blockDim.x) start_loc[e] = s_start[e];
  for (int e = 0; e < num_experts; ++e) {
    const int b = s_start[e], t = s_start[e + 1];
    for (long long r = b + threadIdx.x; r < t && r < m_indices_len; r += blockDim.x) m_indices[r] = e;
  }
}

template <typename IdxT>
__global__ void __launch_bounds__(THREADS) scatter_index_kernel(const IdxT* __restrict__ ids, const int* __restrict__ rank,
                                                                const int* __restrict__ start_loc, long long slots,
                                                                IdxT* __restrict__ output_index, int* __restrict__ dst_pos) {
  if (!wait_for_predecessor()) return;
  for (long long f = (long long)blockIdx.x * THREADS + threadIdx.x; f < slots; f += (long long)gridDim.x * THREADS) {
    const long long e = (long long)ids[f];
    int d = -1;
    if (e >= 0) {
      d = start_loc[e] + rank[f];
      output_index[f] = (IdxT)d;   // slots with id < 0 keep their previous content, as in the reference
    }
    dst_pos[f] = d;
  }
}

template <typename IdxT>
__global__ void __launch_bounds__(THREADS) dest_ranks_kernel(const IdxT* __restrict__ ids, long long tokens, int top_k,
                                                             int num_local, int world, int* __restrict__ dest) {
  if (!wait_for_predecessor()) return;
  const long long total = tokens * world;
  for (long long u = (long long)blockIdx.x * THREADS + threadIdx.x; u < total; u += (long long)gridDim.x * THREADS) {
    const long long t = u / world;
    const int r = (int)(u - t * world);
    bool hit = false;
    for (int j = 0; j < top_k; ++j) {
      const long long id = (long long)ids[t * top_k + j];
      hit = hit || (id >= 0 && id / num_local == r);
    }
    dest[u] = hit ? r : world;
  }
}

int grid_for(long long total_threads) {
  long long blocks = ceil_div(total_threads, THREADS);
  const long long cap = (long long)sm_count() * 16;
  if (blocks > cap) blocks = cap;
  if (blocks < 1) blocks = 1;
  return (int)blocks;
}

// Products and sums "rounded to the tensor's type": for the 16-bit types one packed instruction per pair.  Same bits as
// the fp32 operation followed by a rounding: a product of two such numbers is exact in fp32, and a sum's second rounding is
// harmless with 24 >= 2 * 11 + 2 bits in between.
template <typename T> struct Rounded;
template <> struct Rounded<float> {
  using Pair = float2;
  static __device__ __forceinline__ Pair both(float x) { return make_float2(x, x); }
  static __device__ __forceinline__ Pair mul(Pair a, Pair b) { return make_float2(__fmul_rn(a.x, b.x), __fmul_rn(a.y, b.y)); }
  static __device__ __forceinline__ Pair add(Pair a, Pair b) { return make_float2(__fadd_rn(a.x, b.x), __fadd_rn(a.y, b.y)); }
  static __device__ __forceinline__ float2 wide(Pair a) { return a; }
};
template <> struct Rounded<__nv_bfloat16> {
  using Pair = __nv_bfloat162;
  static __device__ __forceinline__ Pair both(float x) { return __bfloat162bfloat162(__float2bfloat16_rn(x)); }
  static __device__ __forceinline__ Pair mul(Pair a, Pair b) { return __hmul2_rn(a, b); }
  static __device__ __forceinline__ Pair add(Pair a, Pair b) { return __hadd2_rn(a, b); }
  static __device__ __forceinline__ float2 wide(Pair a) { return __bfloat1622float2(a); }
};
template <> struct Rounded<__half> {
  using Pair = __half2;
  static __device__ __forceinline__ Pair both(float x) { return __half2half2(__float2half_rn(x)); }
  static __device__ __forceinline__ Pair mul(Pair a, Pair b) { return __hmul2_rn(a, b); }
  static __device__ __forceinline__ Pair add(Pair a, Pair b) { return __hadd2_rn(a, b); }
  static __device__ __forceinline__ float2 wide(Pair a) { return __half22float2(a); }
};

// ---- training-side un-permute (dlblas/kernels/permute/moe_triton_kernels.py) -----------------
// out[t] = sum over k of prob[t, k] * in[row_id_map[k * T + t]] (entries -1 skipped), accumulated in
// the tensor's own type with a rounding after every product and every add, as gather_kernel
// (:229-271) does.  Without probs it is the plain sum of permute's backward (:140-167).
template <typename T, int R>
__global__ void __launch_bounds__(THREADS) unpermute_kernel(const T* __restrict__ in, const int* __restrict__ row_id_map,
                                                            const float* __restrict__ probs, uint32_t tokens,
                                                            uint32_t units, FastDiv chunks, int top_k, long long h,
                                                            T* __restrict__ out) {
  if (!wait_for_predecessor()) return;
  const int lane = threadIdx.x & 31;
  for (uint32_t w = blockIdx.x * (THREADS / 32) + (threadIdx.x >> 5); w < units; w += gridDim.x * (THREADS / 32)) {
    const uint32_t t = chunks.quot(w);
    const long long c = (long long)(w - t * chunks.d) * 256 + lane * 8;
    if (c >= h) continue;
    using P = Rounded<T>;
    alignas(16) typename P::Pair acc[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) acc[i] = P::both(0.f);
    bool copy = true;                        // slot 0 starts the sum; zeros do when it is unrouted, as in the reference
    for (int j0 = 0; j0 < top_k; j0 += R) {
      int row[R];
      Raw8<T> raw[R];
#pragma unroll
      for (int j = 0; j < R; ++j) row[j] = j0 + j < top_k ? __ldg(row_id_map + (long long)(j0 + j) * tokens + t) : -1;
#pragma unroll
      for (int j = 0; j < R; ++j) raw[j].load_if(row[j] >= 0, in + (long long)row[j] * h + c);
#pragma unroll
      for (int j = 0; j < R; ++j) {
        if (row[j] >= 0) {
          typename P::Pair v[4];
#pragma unroll
          for (int i = 0; i < 4; ++i) v[i] = reinterpret_cast<const typename P::Pair*>(raw[j].w)[i];
          if (probs != nullptr) {
            const typename P::Pair p = P::both(__ldg(probs + (long long)t * top_k + j0 + j));
#pragma unroll
            for (int i = 0; i < 4; ++i) v[i] = P::mul(v[i], p);
          }
#pragma unroll
          for (int i = 0; i < 4; ++i) acc[i] = copy ? v[i] : P::add(acc[i], v[i]);
        }
        copy = false;
      }
    }
    uint4* dst = reinterpret_cast<uint4*>(out + (long long)t * h + c);
#pragma unroll
    for (int i = 0; i < Raw8<T>::WORDS; ++i) dst[i] = reinterpret_cast<const uint4*>(acc)[i];
  }
}

// Rows that some slot refers to (a row without one gets a zero gradient).
__global__ void __launch_bounds__(THREADS) mark_rows_kernel(const int* __restrict__ row_id_map, uint32_t slots,
                                                            uint8_t* __restrict__ marks) {
  if (!wait_for_predecessor()) return;
  for (uint32_t i = blockIdx.x * THREADS + threadIdx.x; i < slots; i += gridDim.x * THREADS) {
    const int row = __ldg(row_id_map + i);
    if (row >= 0) marks[row] = 1;
  }
}

// Backward of the weighted un-permute (scatter_bwd_kernel_optimized, :427-478): one block per token;
// act_grad[row] = grad_out[t] * prob[t, k] (product in the tensors' type, stored as OutT),
// prob_grad[t, k] = sum over columns of the type-rounded products grad_out[t] * fwd_in[row], in fp32.
// grad_out is read once per token and up to eight rows' vectors are in flight per thread.  Storing the gradient in the
// tensors' own type (what autograd hands on) instead of fp32 followed by a conversion, and zeroing only the rows that no
// slot refers to (`marks`, by the blocks behind the tokens') instead of all of them, took the backward of 8192 tokens x
// top-8 x 4096 bf16 columns from 0.83 ms (three kernels, 4.7 GB moved) to the one pass over its 1.1 GB.
template <typename T, typename OutT>
__global__ void __launch_bounds__(THREADS) unpermute_bwd_kernel(const T* __restrict__ grad_out,
                                                                const T* __restrict__ fwd_in,
                                                                const int* __restrict__ row_id_map,
                                                                const float* __restrict__ probs, uint32_t tokens,
                                                                int top_k, long long h, const uint8_t* __restrict__ marks,
                                                                uint32_t rows, OutT* __restrict__ act_grad,
                                                                float* __restrict__ prob_grad) {
  if (!wait_for_predecessor()) return;
  constexpr int R = GATHER_ROWS<T>;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, warps = blockDim.x >> 5;
  if (blockIdx.x >= tokens) {
    const uint32_t zero_blocks = gridDim.x - tokens;
    for (uint32_t r0 = ((blockIdx.x - tokens) * warps + warp) * 32; r0 < rows; r0 += zero_blocks * warps * 32) {
      unsigned bare = __ballot_sync(0xffffffffu, r0 + lane < rows && marks[r0 + lane] == 0);
      while (bare != 0) {
        const long long row = r0 + __ffs(bare) - 1;
        bare &= bare - 1;
        const float zero[8] = {};
        for (long long c = lane * 8; c < h; c += 256) Vec8<OutT>::store(act_grad + row * h + c, zero);
      }
    }
    return;
  }
  const uint32_t t = blockIdx.x;
  __shared__ float sums[THREADS / 32][R];
  for (int j0 = 0; j0 < top_k; j0 += R) {
    using P = Rounded<T>;
    int row[R];
    typename P::Pair p[R];
    float dot[R];
#pragma unroll
    for (int j = 0; j < R; ++j) {
      row[j] = j0 + j < top_k ? __ldg(row_id_map + (long long)(j0 + j) * tokens + t) : -1;
      p[j] = P::both(j0 + j < top_k ? __ldg(probs + (long long)t * top_k + j0 + j) : 0.f);
      dot[j] = 0.f;
    }
    for (long long c = (long long)threadIdx.x * 8; c < h; c += (long long)blockDim.x * 8) {
      Raw8<T> raw_go, raw[R];
      raw_go.load(grad_out + (long long)t * h + c);
#pragma unroll
      for (int j = 0; j < R; ++j) raw[j].load_if(row[j] >= 0, fwd_in + (long long)row[j] * h + c);
      const typename P::Pair* go = reinterpret_cast<const typename P::Pair*>(raw_go.w);
#pragma unroll
      for (int j = 0; j < R; ++j) {
        if (row[j] < 0) continue;
        const typename P::Pair* fw = reinterpret_cast<const typename P::Pair*>(raw[j].w);
        OutT* dst = act_grad + (long long)row[j] * h + c;
        alignas(16) typename P::Pair ag[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          ag[i] = P::mul(go[i], p[j]);
          const float2 d = P::wide(P::mul(go[i], fw[i]));
          dot[j] += d.x;
          dot[j] += d.y;
        }
        if constexpr (sizeof(OutT) == sizeof(T)) {
#pragma unroll
          for (int i = 0; i < Raw8<T>::WORDS; ++i)
            reinterpret_cast<uint4*>(dst)[i] = reinterpret_cast<const uint4*>(ag)[i];
        } else {
          float wide[8];
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            const float2 d = P::wide(ag[i]);
            wide[2 * i] = d.x;
            wide[2 * i + 1] = d.y;
          }
          Vec8<float>::store(dst, wide);
        }
      }
    }
#pragma unroll
    for (int j = 0; j < R; ++j) {
      dot[j] = warp_sum(dot[j]);
      if (lane == 0) sums[warp][j] = dot[j];
    }
    __syncthreads();
    if (threadIdx.x < R && j0 + threadIdx.x < top_k) {
      float s = 0.f;
      for (int i = 0; i < warps; ++i) s += sums[i][threadIdx.x];
      prob_grad[(long long)t * top_k + j0 + threadIdx.x] = s;
    }
    __syncthreads();
  }
}

// Flat indices of these kernels are 32-bit; launches over more units run in slabs of whole rows.
long long slab_rows(long long units_per_row) { return std::max(1ll, ((1ll << 31) - 1) / units_per_row); }

}  // namespace
}  // namespace dlb

using namespace dlb;

extern "C" int dlb_quant_fp8(const void* x, int x_dtype, int64_t m, int64_t k, int64_t ldx, int group_size, int mode,
                             float eps, void* q, float* scales, int64_t scale_row_stride, int64_t scale_group_stride,
                             const int32_t* dst_pos, int fanout, void* stream) {
  DLB_REQUIRE(m >= 0 && k > 0, DLB_ERR_INVALID, "quant_fp8: bad sizes m=%lld k=%lld", (long long)m, (long long)k);
  DLB_REQUIRE(group_size == 32 || group_size == 64 || group_size == 128 || group_size == 256, DLB_ERR_INVALID,
              "quant_fp8: group_size %d not supported (32, 64, 128, 256)", group_size);
  DLB_REQUIRE(k % group_size == 0, DLB_ERR_INVALID, "quant_fp8: k=%lld is not a multiple of group_size=%d",
              (long long)k, group_size);
  DLB_REQUIRE(mode == DLB_QUANT_RECIP_MUL || mode == DLB_QUANT_DIV_EPS, DLB_ERR_INVALID, "quant_fp8: bad mode %d", mode);
  DLB_REQUIRE(dst_pos == nullptr || fanout > 0, DLB_ERR_INVALID, "quant_fp8: fanout must be positive with dst_pos");
  if (m == 0) return DLB_OK;
  DLB_REQUIRE(x && q && scales, DLB_ERR_INVALID, "quant_fp8: null pointer");
  const int esz = x_dtype == DLB_F32 ? 4 : 2;
  DLB_REQUIRE((uintptr_t)x % 16 == 0 && (ldx * esz) % 16 == 0 && (uintptr_t)q % 8 == 0, DLB_ERR_INVALID,
              "quant_fp8: x rows must be 16-byte aligned and q 8-byte aligned");
  DLB_REQUIRE(x_dtype == DLB_BF16 || x_dtype == DLB_F16 || x_dtype == DLB_F32, DLB_ERR_INVALID,
              "quant_fp8: unsupported input dtype %d", x_dtype);
  cudaStream_t st = (cudaStream_t)stream;
  const FastDiv vpr((uint32_t)(k / 16));
  const long long slab = slab_rows(k / 16);
  for (long long r0 = 0; r0 < m; r0 += slab) {
    const long long rows = std::min<long long>(slab, m - r0);
    const uint32_t total = (uint32_t)(rows * (k / 16));
    const int grid = grid_for(total);
    uint8_t* qq = reinterpret_cast<uint8_t*>(q) + (dst_pos == nullptr ? r0 * k : 0);
    float* ss = scales + (dst_pos == nullptr ? r0 * scale_row_stride : 0);
    const int* dp = dst_pos == nullptr ? nullptr : dst_pos + r0 * fanout;
    auto launch = [&](auto* xp) {
      using T = std::remove_const_t<std::remove_pointer_t<decltype(xp)>>;
      after_predecessor(quant_fp8_kernel<T>, grid, THREADS, 0, st)(xp + r0 * ldx, total, vpr, ldx, group_size / 16, mode,
                                                                   eps, qq, ss, scale_row_stride, scale_group_stride, dp,
                                                                   fanout);
    };
    if (x_dtype == DLB_BF16) launch(reinterpret_cast<const __nv_bfloat16*>(x));
    else if (x_dtype == DLB_F16) launch(reinterpret_cast<const __half*>(x));
    else launch(reinterpret_cast<const float*>(x));
    count_launch();
    DLB_CHECK_LAUNCH("quant_fp8_kernel");
  }
  return DLB_OK;
}

extern "C" int dlb_permute_rows(const void* q, int64_t row_bytes, const float* scales, int64_t groups, int64_t m,
                                const int32_t* dst_pos, int fanout, void* out_q, float* out_scales, void* stream) {
  DLB_REQUIRE(m >= 0 && row_bytes > 0 && row_bytes % 16 == 0, DLB_ERR_INVALID,
              "permute_rows: row_bytes=%lld must be a positive multiple of 16", (long long)row_bytes);
  DLB_REQUIRE(groups >= 0 && groups <= row_bytes / 16, DLB_ERR_INVALID, "permute_rows: too many scale groups per row");
  DLB_REQUIRE(fanout > 0, DLB_ERR_INVALID, "permute_rows: fanout must be positive");
  if (m == 0) return DLB_OK;
  DLB_REQUIRE(q && dst_pos && out_q && (scales == nullptr || out_scales != nullptr), DLB_ERR_INVALID,
              "permute_rows: null pointer");
  DLB_REQUIRE((uintptr_t)q % 16 == 0 && (uintptr_t)out_q % 16 == 0, DLB_ERR_INVALID,
              "permute_rows: q and out_q must be 16-byte aligned");
  const long long vpr = row_bytes / 16;
  const long long slab = slab_rows(vpr);
  for (long long r0 = 0; r0 < m; r0 += slab) {
    const uint32_t total = (uint32_t)(std::min<long long>(slab, m - r0) * vpr);
    after_predecessor(permute_rows_kernel, grid_for(total), THREADS, 0, (cudaStream_t)stream)(
        reinterpret_cast<const uint4*>(q) + r0 * vpr, FastDiv((uint32_t)vpr),
        scales == nullptr ? nullptr : scales + r0 * groups, (uint32_t)groups, total, dst_pos + r0 * fanout, fanout,
        reinterpret_cast<uint4*>(out_q), out_scales);
    count_launch();
    DLB_CHECK_LAUNCH("permute_rows_kernel");
  }
  return DLB_OK;
}

extern "C" int dlb_silu_and_mul(const void* gate_up, int dtype, int64_t rows, int64_t n, int64_t ld_in, void* out,
                                int64_t ld_out, void* stream) {
  DLB_REQUIRE(rows >= 0 && n > 0 && n % 8 == 0, DLB_ERR_INVALID, "silu_and_mul: n=%lld must be a positive multiple of 8",
              (long long)n);
  if (rows == 0) return DLB_OK;
  DLB_REQUIRE(gate_up && out, DLB_ERR_INVALID, "silu_and_mul: null pointer");
  const int esz = dtype == DLB_F32 ? 4 : 2;
  DLB_REQUIRE((uintptr_t)gate_up % 16 == 0 && (uintptr_t)out % 16 == 0 && (ld_in * esz) % 16 == 0 &&
                  (ld_out * esz) % 16 == 0 && (n * esz) % 16 == 0,
              DLB_ERR_INVALID, "silu_and_mul: rows must be 16-byte aligned");
  DLB_REQUIRE(dtype == DLB_BF16 || dtype == DLB_F16 || dtype == DLB_F32, DLB_ERR_INVALID,
              "silu_and_mul: unsupported dtype %d", dtype);
  cudaStream_t st = (cudaStream_t)stream;
  const long long slab = slab_rows(n / 8);
  for (long long r0 = 0; r0 < rows; r0 += slab) {
    const uint32_t total = (uint32_t)(std::min<long long>(slab, rows - r0) * (n / 8));
    auto launch = [&](auto* in, auto* o) {
      using T = std::remove_pointer_t<decltype(o)>;
      after_predecessor(silu_and_mul_kernel<T>, grid_for(total), THREADS, 0, st)(
          in + r0 * ld_in, total, FastDiv((uint32_t)(n / 8)), ld_in, o + r0 * ld_out, ld_out);
    };
    if (dtype == DLB_BF16) launch(reinterpret_cast<const __nv_bfloat16*>(gate_up), reinterpret_cast<__nv_bfloat16*>(out));
    else if (dtype == DLB_F16) launch(reinterpret_cast<const __half*>(gate_up), reinterpret_cast<__half*>(out));
    else launch(reinterpret_cast<const float*>(gate_up), reinterpret_cast<float*>(out));
    count_launch();
    DLB_CHECK_LAUNCH("silu_and_mul_kernel");
  }
  return DLB_OK;
}

extern "C" int dlb_silu_mul_quant(const void* gate_up, int dtype, int64_t rows, int64_t n, int quant_mode, float eps,
                                  int round_silu, const int32_t* masked_m, int64_t rows_per_expert, void* q,
                                  float* scales, void* stream) {
  DLB_REQUIRE(rows >= 0 && n > 0 && n % 128 == 0, DLB_ERR_INVALID,
              "silu_mul_quant: n=%lld must be a positive multiple of 128", (long long)n);
  DLB_REQUIRE(quant_mode == DLB_QUANT_RECIP_MUL || quant_mode == DLB_QUANT_DIV_EPS, DLB_ERR_INVALID,
              "silu_mul_quant: bad mode %d", quant_mode);
  DLB_REQUIRE(masked_m == nullptr || rows_per_expert > 0, DLB_ERR_INVALID, "silu_mul_quant: rows_per_expert needed");
  if (rows == 0) return DLB_OK;
  DLB_REQUIRE(gate_up && q && scales, DLB_ERR_INVALID, "silu_mul_quant: null pointer");
  DLB_REQUIRE((uintptr_t)gate_up % 16 == 0 && (uintptr_t)q % 8 == 0, DLB_ERR_INVALID, "silu_mul_quant: misaligned");
  int experts = 0;
  if (masked_m != nullptr) {
    DLB_REQUIRE(rows % rows_per_expert == 0 && rows / rows_per_expert <= MASKED_MAX_EXPERTS, DLB_ERR_INVALID,
                "silu_mul_quant: rows=%lld must be a whole number (at most %d) of experts of %lld rows", (long long)rows,
                MASKED_MAX_EXPERTS, (long long)rows_per_expert);
    experts = (int)(rows / rows_per_expert);
  }
  DLB_REQUIRE(dtype == DLB_BF16 || dtype == DLB_F16, DLB_ERR_INVALID,
              "silu_mul_quant: unsupported dtype %d (bf16 / fp16)", dtype);
  cudaStream_t st = (cudaStream_t)stream;
  uint8_t* qq = reinterpret_cast<uint8_t*>(q);
  const long long slab = slab_rows(n / 8);
  for (long long r0 = 0; r0 < rows; r0 += slab) {
    const long long here = std::min<long long>(slab, rows - r0);
    int grid = grid_for(here * (n / 8));
    if (masked_m != nullptr) grid = std::min(grid, 4 * sm_count());   // the valid rows are few; every block pays for the sums
    auto launch = [&](auto* in) {
      using T = std::remove_const_t<std::remove_pointer_t<decltype(in)>>;
      after_predecessor(silu_mul_quant_kernel<T>, grid, THREADS, 0, st)(
          in, (uint32_t)r0, (uint32_t)here, FastDiv((uint32_t)(n / 8)), quant_mode, eps, round_silu, masked_m, experts,
          rows_per_expert, qq, scales);
    };
    if (dtype == DLB_BF16) launch(reinterpret_cast<const __nv_bfloat16*>(gate_up));
    else launch(reinterpret_cast<const __half*>(gate_up));
    count_launch();
    DLB_CHECK_LAUNCH("silu_mul_quant_kernel");
  }
  return DLB_OK;
}

// Units of the combine kernels: one warp per (token, 256 columns).
namespace {
int gather_grid(uint32_t units) {
  return (int)std::min<long long>(ceil_div(units, (long long)(THREADS / 32)), (long long)sm_count() * 16);
}
}  // namespace

namespace {
template <typename T>
int launch_sum_topk(const void* y, int64_t tokens, int top_k, int64_t h, const void* ids, int ids_dtype, int64_t lo,
                    int64_t hi, int skip, void* out, cudaStream_t st) {
  const FastDiv chunks((uint32_t)ceil_div(h, (int64_t)256));
  const long long slab = slab_rows(chunks.d);
  for (long long t0 = 0; t0 < tokens; t0 += slab) {
    const uint32_t units = (uint32_t)(std::min<long long>(slab, tokens - t0) * chunks.d);
    auto launch = [&](auto* idp) {
      with_rows_in_flight<T>(top_k, [&](auto r) {
        using IdT = std::remove_const_t<std::remove_pointer_t<decltype(idp)>>;
        after_predecessor(sum_topk_kernel<T, r.value, IdT>, gather_grid(units), THREADS, 0, st)(
            reinterpret_cast<const T*>(y) + t0 * top_k * h, units, chunks, top_k, h,
            idp == nullptr ? idp : idp + t0 * top_k, lo, hi, skip, reinterpret_cast<T*>(out) + t0 * h);
      });
    };
    if (ids != nullptr && ids_dtype == DLB_I32) launch(reinterpret_cast<const int*>(ids));
    else launch(reinterpret_cast<const long long*>(ids));
    count_launch();
    DLB_CHECK_LAUNCH("sum_topk_kernel");
  }
  return DLB_OK;
}
}  // namespace

extern "C" int dlb_moe_sum_topk(const void* y, int dtype, int64_t tokens, int top_k, int64_t h, const void* ids,
                                int ids_dtype, int64_t id_lo, int64_t id_hi, int skip_unrouted_rows, void* out,
                                void* stream) {
  DLB_REQUIRE(tokens >= 0 && top_k > 0 && top_k <= 32 && h > 0 && h % 8 == 0, DLB_ERR_INVALID,
              "sum_topk: h=%lld must be a positive multiple of 8 and top_k=%d at most 32", (long long)h, top_k);
  DLB_REQUIRE(ids == nullptr || ids_dtype == DLB_I32 || ids_dtype == DLB_I64, DLB_ERR_INVALID,
              "sum_topk: ids must be int32/int64");
  if (tokens == 0) return DLB_OK;
  DLB_REQUIRE(y && out, DLB_ERR_INVALID, "sum_topk: null pointer");
  DLB_REQUIRE((uintptr_t)y % 16 == 0 && (uintptr_t)out % 16 == 0, DLB_ERR_INVALID, "sum_topk: misaligned");
  cudaStream_t st = (cudaStream_t)stream;
  const int skip = (ids != nullptr && skip_unrouted_rows) ? 1 : 0;
  if (dtype == DLB_BF16)
    return launch_sum_topk<__nv_bfloat16>(y, tokens, top_k, h, ids, ids_dtype, id_lo, id_hi, skip, out, st);
  if (dtype == DLB_F16) return launch_sum_topk<__half>(y, tokens, top_k, h, ids, ids_dtype, id_lo, id_hi, skip, out, st);
  if (dtype == DLB_F32) return launch_sum_topk<float>(y, tokens, top_k, h, ids, ids_dtype, id_lo, id_hi, skip, out, st);
  return fail(DLB_ERR_INVALID, "sum_topk: unsupported dtype %d", dtype);
}

namespace {
template <typename T>
int launch_gather(const void* in, int64_t h, const void* ids, const void* index, int idx_dtype, const float* weights,
                  int64_t tokens, int top_k, void* out, cudaStream_t st) {
  const FastDiv chunks((uint32_t)ceil_div(h, (int64_t)256));
  const long long slab = slab_rows(chunks.d);
  for (long long t0 = 0; t0 < tokens; t0 += slab) {
    const uint32_t units = (uint32_t)(std::min<long long>(slab, tokens - t0) * chunks.d);
    const long long s0 = t0 * top_k;
    auto launch = [&](auto* idp, auto* ixp) {
      with_rows_in_flight<T>(top_k, [&](auto r) {
        using IdxT = std::remove_const_t<std::remove_pointer_t<decltype(idp)>>;
        after_predecessor(ep_gather_kernel<T, r.value, IdxT>, gather_grid(units), THREADS, 0, st)(
            reinterpret_cast<const T*>(in), h, idp + s0, ixp + s0, weights + s0, units, chunks, top_k,
            reinterpret_cast<T*>(out) + t0 * h);
      });
    };
    if (idx_dtype == DLB_I32) launch(reinterpret_cast<const int*>(ids), reinterpret_cast<const int*>(index));
    else launch(reinterpret_cast<const long long*>(ids), reinterpret_cast<const long long*>(index));
    count_launch();
    DLB_CHECK_LAUNCH("ep_gather_kernel");
  }
  return DLB_OK;
}
}  // namespace

extern "C" int dlb_ep_gather(const void* in, int dtype, int64_t h, const void* ids, const void* index, int idx_dtype,
                             const float* weights, int64_t tokens, int top_k, void* out, void* stream) {
  DLB_REQUIRE(tokens >= 0 && top_k > 0 && h > 0 && h % 8 == 0, DLB_ERR_INVALID,
              "ep_gather: h=%lld must be a positive multiple of 8", (long long)h);
  DLB_REQUIRE(idx_dtype == DLB_I32 || idx_dtype == DLB_I64, DLB_ERR_INVALID, "ep_gather: ids must be int32/int64");
  if (tokens == 0) return DLB_OK;
  DLB_REQUIRE(in && ids && index && weights && out, DLB_ERR_INVALID, "ep_gather: null pointer");
  DLB_REQUIRE((uintptr_t)in % 16 == 0 && (uintptr_t)out % 16 == 0, DLB_ERR_INVALID, "ep_gather: misaligned");
  cudaStream_t st = (cudaStream_t)stream;
  if (dtype == DLB_BF16) return launch_gather<__nv_bfloat16>(in, h, ids, index, idx_dtype, weights, tokens, top_k, out, st);
  if (dtype == DLB_F16) return launch_gather<__half>(in, h, ids, index, idx_dtype, weights, tokens, top_k, out, st);
  if (dtype == DLB_F32) return launch_gather<float>(in, h, ids, index, idx_dtype, weights, tokens, top_k, out, st);
  return fail(DLB_ERR_INVALID, "ep_gather: unsupported dtype %d", dtype);
}

namespace {
size_t align256(size_t v) { return (v + 255) / 256 * 256; }
}

extern "C" size_t dlb_ep_scatter_workspace_size(int64_t tokens, int top_k, int num_experts) {
  if (tokens <= 0 || top_k <= 0 || num_experts <= 0) return 0;
  const long long slots = tokens * top_k;
  return align256((size_t)slots * 4) * 2 + sort_workspace_size(slots, num_experts);
}

extern "C" int dlb_ep_scatter(const void* x, int64_t row_bytes, const float* x_scale, int64_t groups, const void* ids,
                              int idx_dtype, int64_t tokens, int top_k, const int32_t* counts, int num_experts,
                              int32_t* expert_start_loc, void* out_x, float* out_scale, int32_t* m_indices,
                              int64_t m_indices_len, void* output_index, void* workspace, size_t workspace_bytes,
                              void* stream) {
  DLB_REQUIRE(tokens >= 0 && top_k > 0 && num_experts > 0 && num_experts <= 8192, DLB_ERR_INVALID,
              "ep_scatter: bad sizes");
  DLB_REQUIRE(idx_dtype == DLB_I32 || idx_dtype == DLB_I64, DLB_ERR_INVALID, "ep_scatter: ids must be int32/int64");
  DLB_REQUIRE(row_bytes > 0 && row_bytes % 16 == 0, DLB_ERR_INVALID, "ep_scatter: row_bytes must be a multiple of 16");
  DLB_REQUIRE(counts && expert_start_loc && m_indices, DLB_ERR_INVALID, "ep_scatter: null pointer");
  cudaStream_t st = (cudaStream_t)stream;
  after_predecessor(scatter_layout_kernel, 1, 1024, (size_t)(num_experts + 1) * 4, st)(counts, num_experts,
                                                                                       expert_start_loc, m_indices,
                                                                                       m_indices_len);
  count_launch();
  DLB_CHECK_LAUNCH("scatter_layout_kernel");
  if (tokens == 0) return DLB_OK;
  DLB_REQUIRE(x && ids && out_x && output_index, DLB_ERR_INVALID, "ep_scatter: null pointer");
  const long long slots = tokens * top_k;
  const size_t need = dlb_ep_scatter_workspace_size(tokens, top_k, num_experts);
  DLB_REQUIRE(workspace != nullptr && workspace_bytes >= need, DLB_ERR_WORKSPACE,
              "ep_scatter: workspace of %zu bytes needed, %zu given", need, workspace_bytes);
  char* ws = reinterpret_cast<char*>(workspace);
  int* rank = reinterpret_cast<int*>(ws);
  int* dst_pos = reinterpret_cast<int*>(ws + align256((size_t)slots * 4));
  void* sort_ws = ws + 2 * align256((size_t)slots * 4);
  int rc = sort_by_expert(ids, idx_dtype, slots, num_experts, nullptr, nullptr, nullptr, nullptr, rank, nullptr, sort_ws,
                          workspace_bytes - 2 * align256((size_t)slots * 4), st);
  if (rc != DLB_OK) return rc;
  if (idx_dtype == DLB_I32)
    after_predecessor(scatter_index_kernel<int>, grid_for(slots), THREADS, 0, st)(reinterpret_cast<const int*>(ids), rank,
                                                                  expert_start_loc, slots,
                                                                  reinterpret_cast<int*>(output_index), dst_pos);
  else
    after_predecessor(scatter_index_kernel<long long>, grid_for(slots), THREADS, 0, st)(
        reinterpret_cast<const long long*>(ids), rank, expert_start_loc, slots,
        reinterpret_cast<long long*>(output_index), dst_pos);
  count_launch();
  DLB_CHECK_LAUNCH("scatter_index_kernel");
  return dlb_permute_rows(x, row_bytes, x_scale, groups, tokens, dst_pos, top_k, out_x, out_scale, stream);
}

extern "C" int dlb_ep_dest_ranks(const void* ids, int ids_dtype, int64_t tokens, int top_k, int num_local_experts,
                                 int world, int32_t* dest, void* stream) {
  DLB_REQUIRE(tokens >= 0 && top_k > 0 && num_local_experts > 0 && world > 0, DLB_ERR_INVALID, "ep_dest_ranks: bad sizes");
  DLB_REQUIRE(ids_dtype == DLB_I32 || ids_dtype == DLB_I64, DLB_ERR_INVALID, "ep_dest_ranks: ids must be int32/int64");
  if (tokens == 0) return DLB_OK;
  DLB_REQUIRE(ids && dest, DLB_ERR_INVALID, "ep_dest_ranks: null pointer");
  const int grid = grid_for(tokens * world);
  cudaStream_t st = (cudaStream_t)stream;
  if (ids_dtype == DLB_I32)
    after_predecessor(dest_ranks_kernel<int>, grid, THREADS, 0, st)(
        reinterpret_cast<const int*>(ids), tokens, top_k, num_local_experts, world, dest);
  else
    after_predecessor(dest_ranks_kernel<long long>, grid, THREADS, 0, st)(
        reinterpret_cast<const long long*>(ids), tokens, top_k, num_local_experts, world, dest);
  count_launch();
  DLB_CHECK_LAUNCH("dest_ranks_kernel");
  return DLB_OK;
}

extern "C" int dlb_unpermute(const void* in, int dtype, const int32_t* row_id_map, const float* probs, int64_t tokens,
                             int top_k, int64_t h, void* out, void* stream) {
  DLB_REQUIRE(tokens >= 0 && top_k > 0 && h > 0 && h % 8 == 0, DLB_ERR_INVALID,
              "unpermute: bad sizes tokens=%lld top_k=%d h=%lld (h must be a multiple of 8)", (long long)tokens, top_k,
              (long long)h);
  if (tokens == 0) return DLB_OK;
  DLB_REQUIRE(in && row_id_map && out, DLB_ERR_INVALID, "unpermute: null pointer");
  DLB_REQUIRE((uintptr_t)in % 16 == 0 && (uintptr_t)out % 16 == 0, DLB_ERR_INVALID, "unpermute: misaligned tensors");
  const FastDiv chunks((uint32_t)ceil_div(h, (int64_t)256));
  DLB_REQUIRE(tokens * (long long)chunks.d < (1ll << 31), DLB_ERR_INVALID, "unpermute: tokens=%lld x h=%lld is too large",
              (long long)tokens, (long long)h);
  const uint32_t units = (uint32_t)(tokens * chunks.d);
  cudaStream_t st = (cudaStream_t)stream;
  auto launch = [&](auto* ip, auto* op) {
    using T = std::remove_pointer_t<decltype(op)>;
    with_rows_in_flight<T>(top_k, [&](auto r) {
      after_predecessor(unpermute_kernel<T, r.value>, gather_grid(units), THREADS, 0, st)(
          ip, row_id_map, probs, (uint32_t)tokens, units, chunks, top_k, h, op);
    });
  };
  if (dtype == DLB_BF16) launch(reinterpret_cast<const __nv_bfloat16*>(in), reinterpret_cast<__nv_bfloat16*>(out));
  else if (dtype == DLB_F16) launch(reinterpret_cast<const __half*>(in), reinterpret_cast<__half*>(out));
  else if (dtype == DLB_F32) launch(reinterpret_cast<const float*>(in), reinterpret_cast<float*>(out));
  else return fail(DLB_ERR_INVALID, "unpermute: unsupported dtype %d", dtype);
  count_launch();
  DLB_CHECK_LAUNCH("unpermute_kernel");
  return DLB_OK;
}

// act_dtype: DLB_F32, or the tensors' own type.  marks: [rows] bytes of workspace; rows that no slot refers to become zero.
// nullptr: they are left alone.
static int unpermute_bwd(const void* grad_out, const void* fwd_in, int dtype, const int32_t* row_id_map, const float* probs,
                         int64_t tokens, int top_k, int64_t h, int64_t rows, void* act_grad, int act_dtype,
                         float* prob_grad, uint8_t* marks, void* stream) {
  DLB_REQUIRE(tokens >= 0 && tokens < (1ll << 31) - 4096 && top_k > 0 && h > 0 && h % 8 == 0, DLB_ERR_INVALID,
              "unpermute_bwd: bad sizes tokens=%lld top_k=%d h=%lld", (long long)tokens, top_k, (long long)h);
  DLB_REQUIRE(rows >= 0 && rows < (1ll << 31) && tokens * top_k < (1ll << 31), DLB_ERR_INVALID,
              "unpermute_bwd: too many rows");
  DLB_REQUIRE(dtype == DLB_BF16 || dtype == DLB_F16 || dtype == DLB_F32, DLB_ERR_INVALID,
              "unpermute_bwd: unsupported dtype %d", dtype);
  DLB_REQUIRE(act_dtype == DLB_F32 || act_dtype == dtype, DLB_ERR_INVALID,
              "unpermute_bwd: the gradient is fp32 or of the tensors' type");
  cudaStream_t st = (cudaStream_t)stream;
  if (tokens == 0) return DLB_OK;
  DLB_REQUIRE(grad_out && fwd_in && row_id_map && probs && act_grad && prob_grad, DLB_ERR_INVALID,
              "unpermute_bwd: null pointer");
  DLB_REQUIRE((uintptr_t)grad_out % 16 == 0 && (uintptr_t)fwd_in % 16 == 0 && (uintptr_t)act_grad % 16 == 0,
              DLB_ERR_INVALID, "unpermute_bwd: misaligned tensors");
  if (marks != nullptr && rows > 0) {
    int rc = check_cuda(cudaMemsetAsync(marks, 0, (size_t)rows, st), "cudaMemsetAsync(unpermute_bwd)");
    if (rc != DLB_OK) return rc;
    after_predecessor(mark_rows_kernel, grid_for(tokens * top_k), THREADS, 0, st)(
        row_id_map, (uint32_t)(tokens * top_k), marks);
    count_launch();
    DLB_CHECK_LAUNCH("mark_rows_kernel");
  }
  // as many threads as a row has vectors, up to 256
  const int threads = h <= 512 ? 64 : h <= 1024 ? 128 : THREADS;
  const int zero_blocks = marks == nullptr ? 0 : (int)std::min<long long>(ceil_div(rows, 8ll * 32), sm_count());
  auto launch = [&](auto* go, auto* ag) {
    using T = std::remove_const_t<std::remove_pointer_t<decltype(go)>>;
    using O = std::remove_pointer_t<decltype(ag)>;
    after_predecessor(unpermute_bwd_kernel<T, O>, (int)tokens + zero_blocks, threads, 0, st)(
        go, reinterpret_cast<const T*>(fwd_in), row_id_map, probs, (uint32_t)tokens, top_k, h, marks, (uint32_t)rows, ag,
        prob_grad);
  };
  auto typed = [&](auto* go) {
    using T = std::remove_const_t<std::remove_pointer_t<decltype(go)>>;
    if (act_dtype == DLB_F32) launch(go, reinterpret_cast<float*>(act_grad));
    else launch(go, reinterpret_cast<T*>(act_grad));
  };
  if (dtype == DLB_BF16) typed(reinterpret_cast<const __nv_bfloat16*>(grad_out));
  else if (dtype == DLB_F16) typed(reinterpret_cast<const __half*>(grad_out));
  else launch(reinterpret_cast<const float*>(grad_out), reinterpret_cast<float*>(act_grad));
  count_launch();
  DLB_CHECK_LAUNCH("unpermute_bwd_kernel");
  return DLB_OK;
}

extern "C" int dlb_unpermute_bwd(const void* grad_out, const void* fwd_in, int dtype, const int32_t* row_id_map,
                                 const float* probs, int64_t tokens, int top_k, int64_t h, float* act_grad,
                                 float* prob_grad, void* stream) {
  return unpermute_bwd(grad_out, fwd_in, dtype, row_id_map, probs, tokens, top_k, h, 0, act_grad, DLB_F32, prob_grad,
                       nullptr, stream);
}

extern "C" int dlb_unpermute_bwd_rows(const void* grad_out, const void* fwd_in, int dtype, const int32_t* row_id_map,
                                      const float* probs, int64_t tokens, int top_k, int64_t h, int64_t rows,
                                      void* act_grad, int act_dtype, float* prob_grad, void* row_marks, void* stream) {
  DLB_REQUIRE(row_marks != nullptr || rows == 0, DLB_ERR_WORKSPACE, "unpermute_bwd_rows: %lld bytes of row marks needed",
              (long long)rows);
  if (tokens == 0 && rows > 0)
    return check_cuda(cudaMemsetAsync(act_grad, 0, (size_t)(rows * h * (act_dtype == DLB_F32 ? 4 : 2)), (cudaStream_t)stream),
                      "cudaMemsetAsync(unpermute_bwd_rows)");
  return unpermute_bwd(grad_out, fwd_in, dtype, row_id_map, probs, tokens, top_k, h, rows, act_grad, act_dtype, prob_grad,
                       reinterpret_cast<uint8_t*>(row_marks), stream);
}
