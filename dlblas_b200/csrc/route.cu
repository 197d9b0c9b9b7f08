// Routing kernels: one warp per token row, scores in registers, arg-max over the warp with a deterministic
// tie-break (lowest expert index wins).  What bounds them is the chain of arg-max rounds, not memory: a round is two integer
// warp reductions (redux) on an order-preserving key and on the index, where a butterfly of shuffles took ten of them and
// ten compare-and-selects.
#include "common.cuh"
#include "sort.cuh"

namespace dlb {
namespace {

constexpr int WARPS = 8;
constexpr int MAX_VPT = 32;  // up to 1024 experts

struct ArgMax {
  float v;
  int i;
};
// larger value wins; equal values: smaller index wins
__device__ __forceinline__ ArgMax better(ArgMax a, ArgMax b) {
  return (b.v > a.v || (b.v == a.v && b.i < a.i)) ? b : a;
}
// fp32 as an unsigned integer of the same order; -0 counts as +0, and a NaN comes last (it is never chosen)
__device__ __forceinline__ uint32_t order_key(float v) {
  const uint32_t b = __float_as_uint(v + 0.f);
  return v != v ? 0u : b ^ ((uint32_t)((int32_t)b >> 31) | 0x80000000u);
}
__device__ __forceinline__ float key_value(uint32_t k) {
  return k == 0u ? -__builtin_huge_valf() : __uint_as_float((k & 0x80000000u) ? k ^ 0x80000000u : ~k);
}
__device__ __forceinline__ ArgMax warp_argmax(ArgMax a) {
  const uint32_t key = order_key(a.v);
  const uint32_t best = __reduce_max_sync(0xffffffffu, key);
  const unsigned at = __reduce_min_sync(0xffffffffu, key == best ? (unsigned)a.i : 0x7fffffffu);
  return ArgMax{key_value(best), (int)at};
}

constexpr float NEG_INF = -__builtin_huge_valf();

// Element e of a row lives in lane e % 32, register e / 32 (coalesced loads).
template <typename T, int VPT>
__device__ __forceinline__ void load_row(const T* row, int experts, int lane, float (&x)[VPT]) {
#pragma unroll
  for (int s = 0; s < VPT; ++s) {
    const int e = s * 32 + lane;
    x[s] = e < experts ? to_f32<T>(row[e]) : NEG_INF;
  }
}

template <int VPT>
__device__ __forceinline__ ArgMax row_argmax(const float (&x)[VPT], int lane) {
  ArgMax a = {NEG_INF, 0x7fffffff};
#pragma unroll
  for (int s = 0; s < VPT; ++s) a = better(a, ArgMax{x[s], s * 32 + lane});
  return warp_argmax(a);
}

template <int VPT>
__device__ __forceinline__ void knock_out(float (&x)[VPT], int idx, int lane) {
#pragma unroll
  for (int s = 0; s < VPT; ++s)
    if (s * 32 + lane == idx) x[s] = NEG_INF;
}

// topk(softmax(logits)) : selection on the logits themselves (softmax is monotone), weights
// = exp(x - max) / sum.
template <typename T, int VPT, typename IdT>
__global__ void __launch_bounds__(WARPS * 32) softmax_topk_kernel(const T* __restrict__ logits, long long tokens,
                                                                  int experts, int top_k, int renorm,
                                                                  float* __restrict__ weights, IdT* __restrict__ ids) {
  if (!wait_for_predecessor()) return;
  const int lane = threadIdx.x & 31;
  const long long t = (long long)blockIdx.x * WARPS + (threadIdx.x >> 5);
  if (t >= tokens) return;
  float x[VPT];
  load_row<T, VPT>(logits + t * experts, experts, lane, x);
  float mx = NEG_INF;
#pragma unroll
  for (int s = 0; s < VPT; ++s) mx = fmaxf(mx, x[s]);
  mx = warp_max(mx);
  float sum = 0.f;
#pragma unroll
  for (int s = 0; s < VPT; ++s) sum += (s * 32 + lane < experts) ? expf(x[s] - mx) : 0.f;
  sum = warp_sum(sum);
  float my_w = 0.f;
  int my_id = 0;
  float wsum = 0.f;
  for (int j = 0; j < top_k; ++j) {   // top_k <= 32: lane j keeps slot j
    const ArgMax a = row_argmax<VPT>(x, lane);
    const float w = expf(a.v - mx) / sum;
    wsum += w;
    if (lane == j) {
      my_w = w;
      my_id = a.i;
    }
    knock_out<VPT>(x, a.i, lane);
  }
  if (lane < top_k) {
    weights[t * top_k + lane] = renorm ? my_w / wsum : my_w;
    ids[t * top_k + lane] = (IdT)my_id;
  }
}

// Logistic function whose result does not depend on any library's exponential: evaluated in fp64 with
// individually rounded IEEE operations only (no fused multiply-add, no transcendental call) and rounded
// once to fp32, so that a restatement with the same sequence of operations on any IEEE machine gives the
// same bits.  exp(z), z = -x: n = rint(z * log2(e)), r = z - n * ln2 (two-part constant),
// degree-13 Taylor polynomial in r (|r| <= 0.35: truncation below 1e-17), scaled by 2^n in two exact steps.
// The score differs from a correctly rounded fp32 sigmoid in well under one input in a million, and from
// torch's fp32 sigmoid by at most one unit in the last place.
__device__ __forceinline__ double pow2_exact(int n) { return __longlong_as_double((long long)(n + 1023) << 52); }

__device__ __noinline__ float sigmoid_exact(float x) {
  double z = -(double)x;
  z = fmin(fmax(z, -750.0), 750.0);
  const double n = rint(__dmul_rn(z, 1.4426950408889634));
  double r = __dsub_rn(z, __dmul_rn(n, 0.6931471803691238));
  r = __dsub_rn(r, __dmul_rn(n, 1.9082149292705877e-10));
  double p = 1.6059043836821613e-10;
  p = __dadd_rn(__dmul_rn(p, r), 2.08767569878681e-09);
  p = __dadd_rn(__dmul_rn(p, r), 2.505210838544172e-08);
  p = __dadd_rn(__dmul_rn(p, r), 2.755731922398589e-07);
  p = __dadd_rn(__dmul_rn(p, r), 2.7557319223985893e-06);
  p = __dadd_rn(__dmul_rn(p, r), 2.48015873015873e-05);
  p = __dadd_rn(__dmul_rn(p, r), 0.0001984126984126984);
  p = __dadd_rn(__dmul_rn(p, r), 0.001388888888888889);
  p = __dadd_rn(__dmul_rn(p, r), 0.008333333333333333);
  p = __dadd_rn(__dmul_rn(p, r), 0.041666666666666664);
  p = __dadd_rn(__dmul_rn(p, r), 0.16666666666666666);
  p = __dadd_rn(__dmul_rn(p, r), 0.5);
  p = __dadd_rn(__dmul_rn(p, r), 1.0);
  p = __dadd_rn(__dmul_rn(p, r), 1.0);
  const int ni = (int)n;              // |n| <= 1083
  const int n1 = ni / 2, n2 = ni - n1;  // both powers of two are normal numbers
  const double e = __dmul_rn(__dmul_rn(p, pow2_exact(n1)), pow2_exact(n2));
  return __double2float_rn(__ddiv_rn(1.0, __dadd_rn(1.0, e)));
}

// The same bits for a third of the fp64 operations: the polynomial stops at degree 10 and uses fused operations, the
// quotient is the hardware's reciprocal estimate y corrected by three terms of the geometric series
// 1 / d = y (1 + e + e^2 + ...), e = 1 - d y, and both conversions are integer arithmetic.  The value is then
// within 2^-41 of the logistic function (truncation 3.2e-13; the series leaves e^3, which asks for an estimate better than
// 2^-14), sigmoid_exact within 2^-46; where the fp32 rounding boundary
// is more than 2^-40 away both round alike.  False otherwise (one value in 10^4 at most), and for |x| >= 80, where exp
// leaves the range of normal floats, and NaN.
__device__ __forceinline__ bool sigmoid_quick(float x, float& s) {
  const uint32_t u = __float_as_uint(x);
  // -x; zeros and subnormals become +-2^-127 or so, which gives the same 0.5
  const double z = __hiloint2double((int)((((u & 0x7fffffffu) >> 3) + 0x38000000u) | (~u & 0x80000000u)), (int)(u << 29));
  const double t = __fma_rn(z, 1.4426950408889634, 6755399441055744.0);   // 1.5 * 2^52: n in the low word
  const int n = __double2loint(t);
  const double nd = __dsub_rn(t, 6755399441055744.0);
  double r = __fma_rn(nd, -0.6931471803691238, z);
  r = __fma_rn(nd, -1.9082149292705877e-10, r);
  double p = 2.755731922398589e-07;
  p = __fma_rn(p, r, 2.7557319223985893e-06);
  p = __fma_rn(p, r, 2.48015873015873e-05);
  p = __fma_rn(p, r, 0.0001984126984126984);
  p = __fma_rn(p, r, 0.001388888888888889);
  p = __fma_rn(p, r, 0.008333333333333333);
  p = __fma_rn(p, r, 0.041666666666666664);
  p = __fma_rn(p, r, 0.16666666666666666);
  p = __fma_rn(p, r, 0.5);
  p = __fma_rn(p, r, 1.0);
  p = __fma_rn(p, r, 1.0);
  const double d = __dadd_rn(1.0, __hiloint2double(__double2hiint(p) + (n << 20), __double2loint(p)));
  double y;
  asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(d));
  double e = __fma_rn(-d, y, 1.0);
  e = __fma_rn(e, e, e);
  y = __fma_rn(y, e, y);
  const uint32_t hi = (uint32_t)__double2hiint(y), lo = (uint32_t)__double2loint(y);
  const uint32_t tail = lo & 0x1fffffffu;                                  // the bits below the float's last place
  s = __uint_as_float((((hi - 0x38000000u) << 3) | (lo >> 29)) + (tail >> 28));
  return fabsf(x) < 80.f && tail - (0x10000000u - 0x2000u) >= 0x4000u;     // 2^13 units of 2^-53 around the tie
}

// A lane's scores.  fp64 runs at half the rate of fp32, and 256 of the full evaluations per token were a third of the routing
// kernel: 20000 x 256 fp32 logits with the aligned layout 53 -> 45 us.
template <int VPT> __device__ __forceinline__ void sigmoid_row(const float (&x)[VPT], float (&s)[VPT]) {
  uint32_t unsure = 0;
#pragma unroll
  for (int i = 0; i < VPT; ++i) unsure |= (sigmoid_quick(x[i], s[i]) ? 0u : 1u) << i;
  if (unsure != 0) {
#pragma unroll
    for (int i = 0; i < VPT; ++i)
      if ((unsure >> i) & 1u) s[i] = sigmoid_exact(x[i]);
  }
}

// DeepSeek-V3 style grouped routing (dlblas/kernels/moe.py:477-521).
template <typename T, int VPT>
__global__ void __launch_bounds__(WARPS * 32) grouped_topk_kernel(const T* __restrict__ logits,
                                                                  const float* __restrict__ bias, long long tokens,
                                                                  int experts, int num_groups, int topk_group, int top_k,
                                                                  int renorm, float* __restrict__ weights,
                                                                  int* __restrict__ ids) {
  if (!wait_for_predecessor()) return;
  const int lane = threadIdx.x & 31;
  const long long t = (long long)blockIdx.x * WARPS + (threadIdx.x >> 5);
  if (t >= tokens) return;
  const int per_group = experts / num_groups;
  float sc[VPT];   // unbiased sigmoid scores
  float ch[VPT];   // biased scores used for the choice
  {
    float x[VPT];
    load_row<T, VPT>(logits + t * experts, experts, lane, x);
#pragma unroll
    for (int s = 0; s < VPT; ++s)
      if (s * 32 + lane >= experts) x[s] = 0.f;   // the filling's minus infinity would take the slow way
    sigmoid_row<VPT>(x, sc);
#pragma unroll
    for (int s = 0; s < VPT; ++s) {
      const int e = s * 32 + lane;
      if (e < experts) {
        ch[s] = sc[s] + __ldg(bias + e);
      } else {
        sc[s] = 0.f;
        ch[s] = NEG_INF;
      }
    }
  }
  // group score = sum of the two largest biased scores of the group; lane g keeps group g's score
  float gscore = NEG_INF;
  for (int g = 0; g < num_groups; ++g) {
    const int lo = g * per_group, hi = lo + per_group;
    ArgMax a = {NEG_INF, 0x7fffffff};
#pragma unroll
    for (int s = 0; s < VPT; ++s) {
      const int e = s * 32 + lane;
      if (e >= lo && e < hi) a = better(a, ArgMax{ch[s], e});
    }
    a = warp_argmax(a);
    ArgMax b = {NEG_INF, 0x7fffffff};
#pragma unroll
    for (int s = 0; s < VPT; ++s) {
      const int e = s * 32 + lane;
      if (e >= lo && e < hi && e != a.i) b = better(b, ArgMax{ch[s], e});
    }
    b = warp_argmax(b);
    if (lane == g) gscore = a.v + b.v;
  }
  // keep the topk_group best groups (bit mask, same in every lane)
  unsigned keep = 0;
  for (int j = 0; j < topk_group; ++j) {
    ArgMax a = {gscore, lane};
    if (lane >= num_groups) a = ArgMax{NEG_INF, 0x7fffffff};
    a = warp_argmax(a);
    keep |= 1u << a.i;
    if (lane == a.i) gscore = NEG_INF;
  }
#pragma unroll
  for (int s = 0; s < VPT; ++s) {
    const int e = s * 32 + lane;
    if (e < experts && !((keep >> (e / per_group)) & 1u)) ch[s] = NEG_INF;
  }
  float wsum = 0.f;
  float my_w = 0.f;
  int my_id = 0;
  for (int j = 0; j < top_k; ++j) {
    const ArgMax a = row_argmax<VPT>(ch, lane);
    // owner lane broadcasts the unbiased score of the chosen expert
    float w = 0.f;
#pragma unroll
    for (int s = 0; s < VPT; ++s)
      if (s * 32 + lane == a.i) w = sc[s];
    w = __shfl_sync(0xffffffffu, w, a.i & 31);
    wsum += w;
    if (lane == j) {
      my_w = w;
      my_id = a.i;
    }
    knock_out<VPT>(ch, a.i, lane);
  }
  if (lane < top_k) {
    weights[t * top_k + lane] = renorm ? my_w / wsum : my_w;
    ids[t * top_k + lane] = my_id;
  }
}

// The same for 32 * VPT experts in groups of whole lanes: lane l holds experts [l * VPT, (l + 1) * VPT), so that a group is a
// power of two of neighbouring lanes (`group_lanes`).  All groups' two largest scores then come out of one butterfly over
// group_lanes lanes (the kernel above takes two arg-max rounds per group: 16 of its 28 rounds with 8 groups), a lane's
// position is its experts' position, so the lowest index among equal scores is the lowest lane of a ballot, and a round only
// touches the winner's registers.
template <typename T, int VPT, bool VEC>
__global__ void __launch_bounds__(WARPS * 32) grouped_topk_lanes_kernel(const T* __restrict__ logits,
                                                                        const float* __restrict__ bias, long long tokens,
                                                                        int num_groups, int group_lanes, int topk_group,
                                                                        int top_k, int renorm, float* __restrict__ weights,
                                                                        int* __restrict__ ids) {
  if (!wait_for_predecessor()) return;
  const int lane = threadIdx.x & 31;
  const long long t = (long long)blockIdx.x * WARPS + (threadIdx.x >> 5);
  if (t >= tokens) return;
  float sc[VPT], ch[VPT];
  {
    const T* row = logits + t * (32 * VPT) + lane * VPT;
    constexpr int BYTES = VPT * sizeof(T);
    alignas(16) T x[VPT];
    if constexpr (VEC && BYTES % 16 == 0) {
#pragma unroll
      for (int i = 0; i < BYTES / 16; ++i) reinterpret_cast<uint4*>(x)[i] = __ldg(reinterpret_cast<const uint4*>(row) + i);
    } else if constexpr (VEC && BYTES % 8 == 0) {
#pragma unroll
      for (int i = 0; i < BYTES / 8; ++i) reinterpret_cast<uint2*>(x)[i] = __ldg(reinterpret_cast<const uint2*>(row) + i);
    } else {
#pragma unroll
      for (int i = 0; i < VPT; ++i) x[i] = row[i];
    }
    float xf[VPT];
#pragma unroll
    for (int i = 0; i < VPT; ++i) xf[i] = to_f32<T>(x[i]);
    sigmoid_row<VPT>(xf, sc);
#pragma unroll
    for (int i = 0; i < VPT; ++i) ch[i] = fmaxf(sc[i] + __ldg(bias + lane * VPT + i), NEG_INF);   // a NaN is never chosen
  }
  // the two largest scores of the lane, then of its group
  float v1 = ch[0], v2 = NEG_INF;
#pragma unroll
  for (int i = 1; i < VPT; ++i) {
    v2 = fmaxf(v2, fminf(v1, ch[i]));
    v1 = fmaxf(v1, ch[i]);
  }
  for (int o = 1; o < group_lanes; o <<= 1) {
    const float w1 = __shfl_xor_sync(0xffffffffu, v1, o), w2 = __shfl_xor_sync(0xffffffffu, v2, o);
    v2 = fmaxf(fminf(v1, w1), fmaxf(v2, w2));
    v1 = fmaxf(v1, w1);
  }
  const float gscore = v1 + v2;
  const int my_group = lane / group_lanes;
  int better_groups = 0;
  for (int g = 0; g < num_groups; ++g) {
    const float s = __shfl_sync(0xffffffffu, gscore, g * group_lanes);
    better_groups += (s > gscore || (s == gscore && g < my_group)) ? 1 : 0;
  }
  // Groups of minus infinity (a bias that switches experts off) lose to all others.  Where there are not enough others, the
  // rounds of the kernel above take the first group of the row again and again, and the first expert once no score is left.
  const bool scored = gscore > NEG_INF;
  const bool too_few = __popc(__ballot_sync(0xffffffffu, scored)) < topk_group * group_lanes;
  const bool kept = (scored && better_groups < topk_group) || (too_few && my_group == 0);
  // best remaining expert of the lane
  float best = NEG_INF, best_score = sc[0];
  int best_at = 0;
  auto scan = [&] {
    best = NEG_INF;
    best_at = 0;
    best_score = sc[0];
#pragma unroll
    for (int i = 0; i < VPT; ++i)
      if (ch[i] > best) {
        best = ch[i];
        best_at = i;
        best_score = sc[i];
      }
  };
  if (kept) scan();
  uint32_t key = order_key(best);
  float wsum = 0.f, my_w = 0.f;
  int my_id = 0;
  for (int j = 0; j < top_k; ++j) {
    const uint32_t top = __reduce_max_sync(0xffffffffu, key);
    const int owner = __ffs(__ballot_sync(0xffffffffu, key == top)) - 1;
    const float w = __shfl_sync(0xffffffffu, best_score, owner);
    const int at = __shfl_sync(0xffffffffu, best_at, owner);
    wsum += w;
    if (lane == j) {
      my_w = w;
      my_id = owner * VPT + at;
    }
    if (lane == owner && kept) {
#pragma unroll
      for (int i = 0; i < VPT; ++i)
        if (i == best_at) ch[i] = NEG_INF;
      scan();
      key = order_key(best);
    }
  }
  if (lane < top_k) {
    weights[t * top_k + lane] = renorm ? my_w / wsum : my_w;
    ids[t * top_k + lane] = my_id;
  }
}

// ---- capacity-limited gating (dlblas.topk_gating) -----------------------------------
// part 1: gates = exp(x) / sum(exp(x)) (no max subtraction, topk_gating_fwd_part1.py:38-41),
// k rounds of arg-max on the gates; ids and chosen gates are written k-major.  The block also adds up its tokens' gates and
// first choices per expert (psum, pcnt [blocks][experts]): the column sums over all tokens then only have the blocks to add.
// (A kernel of its own for them, one warp row per 32 experts, was two blocks walking 4096 tokens: 70 of the forward's 105 us.)
// Fixed summation order, no atomics on the sums.
constexpr int GATING_TOKENS = 4;   // tokens per warp, one after the other
template <typename T, int VPT>
__global__ void __launch_bounds__(WARPS * 32) gating_part1_kernel(const T* __restrict__ logits, long long tokens,
                                                                  int experts, int top_k, float* __restrict__ gates,
                                                                  int* __restrict__ ids_km, float* __restrict__ gate_km,
                                                                  float* __restrict__ psum, int* __restrict__ pcnt,
                                                                  int* __restrict__ ticket) {
  if (!wait_for_predecessor()) return;
  extern __shared__ float sm[];
  float* s_sum = sm;                                            // [WARPS][experts]
  int* s_cnt = reinterpret_cast<int*>(sm + WARPS * experts);    // [experts]
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  for (int e = threadIdx.x; e < experts; e += blockDim.x) s_cnt[e] = 0;
  if (blockIdx.x == 0 && threadIdx.x == 0) *ticket = 0;
  __syncthreads();
  float col[VPT];
#pragma unroll
  for (int s = 0; s < VPT; ++s) col[s] = 0.f;
  const long long first = ((long long)blockIdx.x * WARPS + warp) * GATING_TOKENS;
  for (long long t = first; t < min(first + GATING_TOKENS, tokens); ++t) {
    float x[VPT];
    load_row<T, VPT>(logits + t * experts, experts, lane, x);
    float sum = 0.f;
#pragma unroll
    for (int s = 0; s < VPT; ++s) {
      x[s] = (s * 32 + lane < experts) ? expf(x[s]) : NEG_INF;
      sum += (s * 32 + lane < experts) ? x[s] : 0.f;
    }
    sum = warp_sum(sum);
#pragma unroll
    for (int s = 0; s < VPT; ++s) {
      const int e = s * 32 + lane;
      if (e < experts) {
        x[s] = x[s] / sum;
        gates[t * experts + e] = x[s];
        col[s] += x[s];
      }
    }
    for (int j = 0; j < top_k; ++j) {
      const ArgMax a = row_argmax<VPT>(x, lane);
      if (lane == 0) {
        ids_km[(long long)j * tokens + t] = a.i;
        gate_km[(long long)j * tokens + t] = a.v;
        if (j == 0 && a.i < experts) atomicAdd(s_cnt + a.i, 1);
      }
      knock_out<VPT>(x, a.i, lane);
    }
  }
#pragma unroll
  for (int s = 0; s < VPT; ++s)
    if (s * 32 + lane < experts) s_sum[warp * experts + s * 32 + lane] = col[s];
  __syncthreads();
  for (int e = threadIdx.x; e < experts; e += blockDim.x) {
    float sum = 0.f;
    for (int w = 0; w < WARPS; ++w) sum += s_sum[w * experts + e];
    psum[(long long)blockIdx.x * experts + e] = sum;
    pcnt[(long long)blockIdx.x * experts + e] = s_cnt[e];
  }
}

// part 2, in the blocks behind the tokens' of part 3, one warp per expert: me = mean of gates, ce = share of tokens whose
// first choice it is (topk_gating_fwd_part2.py:31-36), and, for an expert with fewer than `capacity` tokens, the remaining
// slots of expert_select_token_idx: the tokens that did not choose it, in ascending order (what a stable descending sort of
// the reference's int mask gives).  The last of these blocks (it waits for nobody) adds up the auxiliary loss.
template <typename T>
__device__ void gating_expert_part(const int* __restrict__ ids_km, const int* __restrict__ counts,
                                   const float* __restrict__ psum, const int* __restrict__ pcnt, int part_blocks,
                                   long long tokens, int experts, int top_k, long long capacity, int block, int blocks,
                                   float* __restrict__ res, float* __restrict__ ce_out, int* __restrict__ ticket,
                                   T* __restrict__ l_aux, long long* __restrict__ select) {
  __shared__ bool last;
  const int lane = threadIdx.x & 31;
  const int e = block * (int)(blockDim.x >> 5) + (threadIdx.x >> 5);
  if (e < experts) {
    float sum = 0.f;
    int cnt = 0;
#pragma unroll 4
    for (int b = lane; b < part_blocks; b += 32) {
      sum += psum[(long long)b * experts + e];
      cnt += pcnt[(long long)b * experts + e];
    }
    sum = warp_sum(sum);
    cnt = __reduce_add_sync(0xffffffffu, cnt);
    if (lane == 0) {
      const float me = sum / (float)tokens;
      const float ce = (float)cnt / (float)tokens;
      res[e] = me * ce * (float)experts * (float)experts;
      ce_out[e] = ce;                                     // kept for the backward pass
    }
    long long filled = counts[e];
    for (long long t0 = 0; t0 < tokens && filled < capacity; t0 += 32) {
      const long long t = t0 + lane;
      bool free_tok = t < tokens;
#pragma unroll 8
      for (int j = 0; j < top_k; ++j) free_tok = free_tok & (t < tokens && ids_km[(long long)j * tokens + t] != e);
      const unsigned m = __ballot_sync(0xffffffffu, free_tok);
      const long long pos = filled + __popc(m & ((1u << lane) - 1u));
      if (free_tok && pos < capacity) select[(long long)e * capacity + pos] = t;
      filled += __popc(m);
    }
  }
  __threadfence();
  __syncthreads();
  if (threadIdx.x == 0) last = atomicAdd(ticket, 1) == blocks - 1;
  __syncthreads();
  if (last && threadIdx.x < 32) {
    __threadfence();
    float s = 0.f;
    for (int i = lane; i < experts; i += 32) s += __ldcg(res + i);
    s = warp_sum(s);
    if (lane == 0) *l_aux = from_f32<T>(s / (float)experts);
  }
}

// part 3: drop entries beyond the capacity, renormalise the kept gates, emit the indices
// (topk_gating_fwd_part3.py:9-61) and the kept part of expert_select_token_idx.  An entry without an expert is dropped
// as well: a row whose gates are all NaN (a NaN logit, or every exp of it 0) has none, the sort gives it rank -1.
__device__ __forceinline__ bool gating_kept(int rank, long long capacity) { return rank >= 0 && rank < capacity; }
constexpr int GATING_SLOTS = 8;   // slots of a token whose loads are in flight together
template <typename T>
__global__ void __launch_bounds__(64) gating_part3_kernel(const int* __restrict__ ids_km,
                                                          const float* __restrict__ gate_km,
                                                          const int* __restrict__ rank, const int* __restrict__ counts,
                                                          const float* __restrict__ psum, const int* __restrict__ pcnt,
                                                          int part_blocks, long long tokens, int experts, int top_k,
                                                          long long capacity, int token_blocks, float* __restrict__ res,
                                                          float* __restrict__ ce_out, int* __restrict__ ticket,
                                                          T* __restrict__ l_aux, int* __restrict__ ec_idx,
                                                          T* __restrict__ out_w, long long* __restrict__ select) {
  if (!wait_for_predecessor()) return;
  if ((int)blockIdx.x >= token_blocks) {
    gating_expert_part<T>(ids_km, counts, psum, pcnt, part_blocks, tokens, experts, top_k, capacity,
                          blockIdx.x - token_blocks, gridDim.x - token_blocks, res, ce_out, ticket, l_aux, select);
    return;
  }
  const long long t = (long long)blockIdx.x * 64 + threadIdx.x;
  if (t >= tokens) return;
  float denom = 0.f;
  int loc[GATING_SLOTS];
  float gate[GATING_SLOTS];
  auto fetch = [&](int j0) {
#pragma unroll
    for (int j = 0; j < GATING_SLOTS; ++j) {
      const long long f = (long long)(j0 + j) * tokens + t;
      loc[j] = j0 + j < top_k ? __ldg(rank + f) : 0x7fffffff;
      gate[j] = j0 + j < top_k ? __ldg(gate_km + f) : 0.f;
    }
  };
  for (int j0 = 0; j0 < top_k; j0 += GATING_SLOTS) {
    fetch(j0);
#pragma unroll
    for (int j = 0; j < GATING_SLOTS; ++j)
      if (gating_kept(loc[j], capacity)) denom += gate[j];
  }
  const float eps = sizeof(T) == 2 ? 9.765625e-4f : 1.1920929e-7f;   // torch.finfo(dtype).eps
  denom = denom < eps ? eps : denom;
  for (int j0 = 0; j0 < top_k; j0 += GATING_SLOTS) {
    if (top_k > GATING_SLOTS) fetch(j0);
    int id[GATING_SLOTS];
#pragma unroll
    for (int j = 0; j < GATING_SLOTS; ++j) id[j] = j0 + j < top_k ? __ldg(ids_km + (long long)(j0 + j) * tokens + t) : 0;
#pragma unroll
    for (int j = 0; j < GATING_SLOTS; ++j) {
      if (j0 + j >= top_k) break;
      const long long f = (long long)(j0 + j) * tokens + t;
      const bool kept = gating_kept(loc[j], capacity);
      out_w[f] = from_f32<T>(kept ? gate[j] / denom : 0.f);
      ec_idx[f] = kept ? (int)((long long)id[j] * capacity + loc[j]) : 0;
      if (kept) select[(long long)id[j] * capacity + loc[j]] = t;
    }
  }
}

template <template <int> class Launcher, typename... Args>
int dispatch_vpt(int experts, Args... args) {
  if (experts <= 32) return Launcher<1>::run(args...);
  if (experts <= 64) return Launcher<2>::run(args...);
  if (experts <= 128) return Launcher<4>::run(args...);
  if (experts <= 256) return Launcher<8>::run(args...);
  if (experts <= 512) return Launcher<16>::run(args...);
  return Launcher<32>::run(args...);
}

struct SoftmaxArgs {
  const void* logits;
  int dtype;
  long long tokens;
  int experts, top_k, renorm;
  float* weights;
  void* ids;
  int ids_dtype;
  cudaStream_t st;
};
template <int VPT> struct SoftmaxLauncher {
  template <typename T> static void go(const SoftmaxArgs& a) {
    const int grid = (int)ceil_div(a.tokens, WARPS);
    if (a.ids_dtype == DLB_I32)
      after_predecessor(softmax_topk_kernel<T, VPT, int>, grid, WARPS * 32, 0, a.st)(
          reinterpret_cast<const T*>(a.logits), a.tokens, a.experts, a.top_k, a.renorm, a.weights,
          reinterpret_cast<int*>(a.ids));
    else
      after_predecessor(softmax_topk_kernel<T, VPT, long long>, grid, WARPS * 32, 0, a.st)(
          reinterpret_cast<const T*>(a.logits), a.tokens, a.experts, a.top_k, a.renorm, a.weights,
          reinterpret_cast<long long*>(a.ids));
  }
  static int run(SoftmaxArgs a) {
    if (a.dtype == DLB_F32) go<float>(a);
    else if (a.dtype == DLB_BF16) go<__nv_bfloat16>(a);
    else go<__half>(a);
    count_launch();
    DLB_CHECK_LAUNCH("softmax_topk_kernel");
    return DLB_OK;
  }
};

struct GroupedArgs {
  const void* logits;
  int dtype;
  const float* bias;
  long long tokens;
  int experts, num_groups, topk_group, top_k, renorm;
  float* weights;
  int* ids;
  cudaStream_t st;
};
template <int VPT> struct GroupedLauncher {
  template <typename T> static void go(const GroupedArgs& a) {
    const int per_group = a.experts / a.num_groups;
    const int lanes = per_group / VPT;
    if (a.experts == 32 * VPT && per_group % VPT == 0 && (lanes & (lanes - 1)) == 0) {
      const int grid = (int)ceil_div(a.tokens, WARPS);
      if ((uintptr_t)a.logits % 16 == 0)   // every row then is, too
        after_predecessor(grouped_topk_lanes_kernel<T, VPT, true>, grid, WARPS * 32, 0, a.st)(
            reinterpret_cast<const T*>(a.logits), a.bias, a.tokens, a.num_groups, lanes, a.topk_group, a.top_k, a.renorm,
            a.weights, a.ids);
      else
        after_predecessor(grouped_topk_lanes_kernel<T, VPT, false>, grid, WARPS * 32, 0, a.st)(
            reinterpret_cast<const T*>(a.logits), a.bias, a.tokens, a.num_groups, lanes, a.topk_group, a.top_k, a.renorm,
            a.weights, a.ids);
      return;
    }
    after_predecessor(grouped_topk_kernel<T, VPT>, (int)ceil_div(a.tokens, WARPS), WARPS * 32, 0, a.st)(
        reinterpret_cast<const T*>(a.logits), a.bias, a.tokens, a.experts, a.num_groups, a.topk_group, a.top_k, a.renorm,
        a.weights, a.ids);
  }
  static int run(GroupedArgs a) {
    if (a.dtype == DLB_F32) go<float>(a);
    else if (a.dtype == DLB_BF16) go<__nv_bfloat16>(a);
    else go<__half>(a);
    count_launch();
    DLB_CHECK_LAUNCH("grouped_topk_kernel");
    return DLB_OK;
  }
};

struct GatingArgs {
  const void* logits;
  int dtype;
  long long tokens;
  int experts, top_k;
  float* gates;
  int* ids_km;
  float* gate_km;
  float* psum;
  int* pcnt;
  int* ticket;
  cudaStream_t st;
};
int gating_blocks(long long tokens) { return (int)ceil_div(tokens, (int64_t)(WARPS * GATING_TOKENS)); }
template <int VPT> struct GatingLauncher {
  static int run(GatingArgs a) {
    const int grid = gating_blocks(a.tokens);
    const size_t smem = (size_t)(WARPS + 1) * a.experts * 4;    // at most 36 KB
    if (a.dtype == DLB_F32)
      after_predecessor(gating_part1_kernel<float, VPT>, grid, WARPS * 32, smem, a.st)(
          reinterpret_cast<const float*>(a.logits), a.tokens, a.experts, a.top_k, a.gates, a.ids_km, a.gate_km, a.psum,
          a.pcnt, a.ticket);
    else
      after_predecessor(gating_part1_kernel<__half, VPT>, grid, WARPS * 32, smem, a.st)(
          reinterpret_cast<const __half*>(a.logits), a.tokens, a.experts, a.top_k, a.gates, a.ids_km, a.gate_km, a.psum,
          a.pcnt, a.ticket);
    count_launch();
    DLB_CHECK_LAUNCH("gating_part1_kernel");
    return DLB_OK;
  }
};

// Backward of the gating: d(l_aux)/d(logits) and, on request, d(token_exp_weights)/d(logits).
//   add[e]  = ce[e] * grad_l_aux * E / T                                  (dlblas/kernels/topk_gating_bwd.py:31-33)
//           + sum over kept slots j with ids[j] == e of
//             ( gw[j] / D + [D not clamped] * sum_i(-gw[i] * g[i] / D^2) )   (w[j] = g[j] / D, D = sum of kept gates)
//   grad[e] = gates[e] * (add[e] - sum_i gates[i] * add[i])                (softmax backward, :40-44)
// One warp per token; reads what the forward left in its workspace.  Lane j looks after slot j of the token (32 slots at a
// time): the slots' terms are formed once, in registers, and handed to the lanes that hold the experts' gates.
template <typename T, int VPT>
__global__ void __launch_bounds__(WARPS * 32) gating_bwd_kernel(const float* __restrict__ gates,
                                                                const float* __restrict__ ce,
                                                                const int* __restrict__ ids_km,
                                                                const float* __restrict__ gate_km,
                                                                const int* __restrict__ rank, long long tokens,
                                                                int experts, int top_k, long long capacity,
                                                                const T* __restrict__ grad_l_aux,
                                                                const T* __restrict__ grad_w, T* __restrict__ grad_logits) {
  if (!wait_for_predecessor()) return;
  const int lane = threadIdx.x & 31;
  const long long t = (long long)blockIdx.x * WARPS + (threadIdx.x >> 5);
  if (t >= tokens) return;
  float g[VPT], add[VPT];
  const float gl = to_f32<T>(*grad_l_aux) * (float)experts / (float)tokens;
#pragma unroll
  for (int s = 0; s < VPT; ++s) {
    const int e = s * 32 + lane;
    g[s] = e < experts ? __ldg(gates + t * experts + e) : 0.f;
    add[s] = e < experts ? __ldg(ce + e) * gl : 0.f;
  }
  if (grad_w != nullptr) {
    const float eps = sizeof(T) == 2 ? 9.765625e-4f : 1.1920929e-7f;   // torch.finfo(dtype).eps
    float denom = 0.f, weighted = 0.f;
    int id = -1;
    float gate = 0.f, gw = 0.f;
    bool kept = false;
    auto fetch = [&](int j0) {
      const long long f = (long long)(j0 + lane) * tokens + t;
      kept = j0 + lane < top_k && gating_kept(__ldg(rank + f), capacity);
      id = kept ? __ldg(ids_km + f) : -1;
      gate = kept ? __ldg(gate_km + f) : 0.f;
      gw = kept ? to_f32<T>(grad_w[f]) : 0.f;
    };
    for (int j0 = 0; j0 < top_k; j0 += 32) {
      fetch(j0);
      denom += warp_sum(gate);
      weighted += warp_sum(gw * gate);
    }
    const bool clamped = denom < eps;
    if (clamped) denom = eps;
    const float coupling = clamped ? 0.f : -weighted / (denom * denom);
    for (int j0 = 0; j0 < top_k; j0 += 32) {
      if (top_k > 32) fetch(j0);
      const float term = gw / denom + coupling;
      for (int j = 0; j < min(32, top_k - j0); ++j) {
        const int e = __shfl_sync(0xffffffffu, id, j);
        const float v = __shfl_sync(0xffffffffu, term, j);
        if (e >= 0 && (e & 31) == lane) {
#pragma unroll
          for (int s = 0; s < VPT; ++s)
            if (s == (e >> 5)) add[s] += v;
        }
      }
    }
  }
  float dot = 0.f;
#pragma unroll
  for (int s = 0; s < VPT; ++s) dot += g[s] * add[s];
  dot = warp_sum(dot);
#pragma unroll
  for (int s = 0; s < VPT; ++s)
    if (s * 32 + lane < experts) grad_logits[t * experts + s * 32 + lane] = from_f32<T>(g[s] * (add[s] - dot));
}

size_t align256(size_t v) { return (v + 255) / 256 * 256; }

struct GatingBwdArgs {
  const float *gates, *ce;
  const int* ids_km;
  const float* gate_km;
  const int* rank;
  int dtype;
  long long tokens;
  int experts, top_k;
  long long capacity;
  const void *grad_l_aux, *grad_w;
  void* grad_logits;
  cudaStream_t st;
};
template <int VPT> struct GatingBwdLauncher {
  template <typename T> static void go(const GatingBwdArgs& a) {
    after_predecessor(gating_bwd_kernel<T, VPT>, (int)ceil_div(a.tokens, WARPS), WARPS * 32, 0, a.st)(
        a.gates, a.ce, a.ids_km, a.gate_km, a.rank, a.tokens, a.experts, a.top_k, a.capacity,
        reinterpret_cast<const T*>(a.grad_l_aux), reinterpret_cast<const T*>(a.grad_w), reinterpret_cast<T*>(a.grad_logits));
  }
  static int run(GatingBwdArgs a) {
    if (a.dtype == DLB_F32) go<float>(a);
    else go<__half>(a);
    count_launch();
    DLB_CHECK_LAUNCH("gating_bwd_kernel");
    return DLB_OK;
  }
};

struct GatingWs {
  size_t gates, ids_km, gate_km, rank, res, ce, counts, psum, pcnt, ticket, sort, bytes;
};
GatingWs gating_ws(long long tokens, int experts, int top_k) {
  GatingWs w;
  size_t off = 0;
  w.gates = off; off += align256((size_t)tokens * experts * 4);
  w.ids_km = off; off += align256((size_t)tokens * top_k * 4);
  w.gate_km = off; off += align256((size_t)tokens * top_k * 4);
  w.rank = off; off += align256((size_t)tokens * top_k * 4);
  w.res = off; off += align256((size_t)experts * 4);
  w.ce = off; off += align256((size_t)experts * 4);
  w.counts = off; off += align256((size_t)experts * 4);
  w.psum = off; off += align256((size_t)gating_blocks(tokens) * experts * 4);
  w.pcnt = off; off += align256((size_t)gating_blocks(tokens) * experts * 4);
  w.ticket = off; off += 256;
  w.sort = off; off += sort_workspace_size(tokens * top_k, experts);
  w.bytes = off;
  return w;
}

// Logical -> physical expert ids for replicated experts: slot (t, k) of a token picks replica
// hash32((t << 16) ^ (k << 8) ^ seed) & 0x7fffffff mod logcnt[e] of its logical expert e
// (dlblas/kernels/moe.py:524-556; all arithmetic in 32 bits, as in the golden model of
// tests/kernels/test_eplb.py:60-90).  Negative ids and experts without a replica give -1.
constexpr int EPLB_THREADS = 256;
template <typename IdT>
__global__ void __launch_bounds__(EPLB_THREADS) eplb_map_hash_kernel(const IdT* __restrict__ topk_idx,
                                                                const int* __restrict__ log2phy,
                                                                const int* __restrict__ logcnt, long long slots,
                                                                int top_k, int num_logical, int max_replica,
                                                                uint32_t seed, int* __restrict__ out) {
  if (!wait_for_predecessor()) return;
  for (long long i = (long long)blockIdx.x * EPLB_THREADS + threadIdx.x; i < slots; i += (long long)gridDim.x * EPLB_THREADS) {
    const long long e = (long long)topk_idx[i];
    int phy = -1;
    if (e >= 0 && e < num_logical) {
      const int cnt = __ldg(logcnt + e);
      if (cnt > 0) {
        const uint32_t t = (uint32_t)(i / top_k);
        const uint32_t k = (uint32_t)(i - (long long)t * top_k);
        uint32_t x = (t << 16) ^ (k << 8) ^ seed;
        x = ((x >> 16) ^ x) * 0x45d9f3bu;
        x = ((x >> 16) ^ x) * 0x45d9f3bu;
        x = (x >> 16) ^ x;
        const uint32_t replica = (x & 0x7fffffffu) % (uint32_t)cnt;
        phy = __ldg(log2phy + e * max_replica + replica);
      }
    }
    out[i] = phy;
  }
}

}  // namespace
}  // namespace dlb

using namespace dlb;

extern "C" int dlb_eplb_map_hash(const void* topk_idx, int ids_dtype, const int32_t* log2phy, const int32_t* logcnt,
                                 int64_t tokens, int top_k, int num_logical, int max_replica, uint32_t seed,
                                 int32_t* physical_idx, void* stream) {
  DLB_REQUIRE(tokens >= 0 && top_k > 0 && num_logical > 0 && max_replica > 0, DLB_ERR_INVALID,
              "eplb_map_hash: bad sizes tokens=%lld top_k=%d experts=%d replicas=%d", (long long)tokens, top_k,
              num_logical, max_replica);
  if (tokens == 0) return DLB_OK;
  DLB_REQUIRE(topk_idx && log2phy && logcnt && physical_idx, DLB_ERR_INVALID, "eplb_map_hash: null pointer");
  const long long slots = tokens * top_k;
  const int grid = (int)std::min<long long>(ceil_div(slots, (long long)EPLB_THREADS), (long long)sm_count() * 16);
  cudaStream_t st = (cudaStream_t)stream;
  if (ids_dtype == DLB_I32) {
    after_predecessor(eplb_map_hash_kernel<int>, grid, EPLB_THREADS, 0, st)(
        reinterpret_cast<const int*>(topk_idx), log2phy, logcnt, slots, top_k, num_logical, max_replica, seed,
        physical_idx);
  } else if (ids_dtype == DLB_I64) {
    after_predecessor(eplb_map_hash_kernel<long long>, grid, EPLB_THREADS, 0, st)(
        reinterpret_cast<const long long*>(topk_idx), log2phy, logcnt, slots, top_k, num_logical, max_replica, seed,
        physical_idx);
  } else {
    return fail(DLB_ERR_INVALID, "eplb_map_hash: ids must be int32 or int64 (got %d)", ids_dtype);
  }
  count_launch();
  DLB_CHECK_LAUNCH("eplb_map_hash_kernel");
  return DLB_OK;
}

extern "C" int dlb_route_softmax_topk(const void* logits, int dtype, int64_t tokens, int experts, int top_k,
                                      int renormalize, float* weights, void* ids, int ids_dtype, void* stream) {
  DLB_REQUIRE(tokens >= 0 && experts > 0 && experts <= 32 * MAX_VPT, DLB_ERR_INVALID,
              "route_softmax_topk: experts=%d must be in [1, 1024]", experts);
  DLB_REQUIRE(top_k > 0 && top_k <= experts && top_k <= 32, DLB_ERR_INVALID,
              "route_softmax_topk: top_k=%d must be in [1, min(experts, 32)]", top_k);
  DLB_REQUIRE(dtype == DLB_F32 || dtype == DLB_BF16 || dtype == DLB_F16, DLB_ERR_INVALID,
              "route_softmax_topk: unsupported logits dtype %d", dtype);
  DLB_REQUIRE(ids_dtype == DLB_I32 || ids_dtype == DLB_I64, DLB_ERR_INVALID, "route_softmax_topk: ids must be int32/int64");
  if (tokens == 0) return DLB_OK;
  DLB_REQUIRE(logits && weights && ids, DLB_ERR_INVALID, "route_softmax_topk: null pointer");
  SoftmaxArgs a = {logits, dtype, tokens, experts, top_k, renormalize, weights, ids, ids_dtype, (cudaStream_t)stream};
  return dispatch_vpt<SoftmaxLauncher>(experts, a);
}

extern "C" int dlb_route_grouped_topk(const void* logits, int dtype, const float* bias, int64_t tokens, int experts,
                                      int num_groups, int topk_group, int top_k, int renormalize, float* weights,
                                      int32_t* ids, void* stream) {
  DLB_REQUIRE(tokens >= 0 && experts > 0 && experts <= 32 * MAX_VPT, DLB_ERR_INVALID,
              "route_grouped_topk: experts=%d must be in [1, 1024]", experts);
  DLB_REQUIRE(num_groups > 0 && num_groups <= 32 && experts % num_groups == 0 && experts / num_groups >= 2,
              DLB_ERR_INVALID, "route_grouped_topk: num_groups=%d must divide experts, be <= 32, with >= 2 experts each",
              num_groups);
  DLB_REQUIRE(topk_group > 0 && topk_group <= num_groups, DLB_ERR_INVALID, "route_grouped_topk: bad topk_group %d",
              topk_group);
  DLB_REQUIRE(top_k > 0 && top_k <= 32 && top_k <= topk_group * (experts / num_groups), DLB_ERR_INVALID,
              "route_grouped_topk: top_k=%d out of range", top_k);
  DLB_REQUIRE(dtype == DLB_F32 || dtype == DLB_BF16 || dtype == DLB_F16, DLB_ERR_INVALID,
              "route_grouped_topk: unsupported logits dtype %d", dtype);
  if (tokens == 0) return DLB_OK;
  DLB_REQUIRE(logits && bias && weights && ids, DLB_ERR_INVALID, "route_grouped_topk: null pointer");
  GroupedArgs a = {logits, dtype, bias, tokens, experts, num_groups, topk_group, top_k, renormalize, weights, ids,
                   (cudaStream_t)stream};
  // 32 lanes of 5 experts, for the kernel of whole lanes: the one count that the package's shapes have beside the powers of two.
  // Other multiples of 32 (96, 192, 384) would fit it as well; each is one more instantiation for every type, and they take the
  // general kernel.  20000 rows of 160, top-6 of 3 of 8 groups: general kernel 60.3 us, whole lanes 18.2; 64 rows 7.4, 3.3.
  if (experts == 160) return GroupedLauncher<5>::run(a);
  return dispatch_vpt<GroupedLauncher>(experts, a);
}

extern "C" size_t dlb_topk_gating_workspace_size(int64_t tokens, int experts, int top_k) {
  if (tokens <= 0 || experts <= 0 || top_k <= 0) return 0;
  return gating_ws(tokens, experts, top_k).bytes;
}

extern "C" int dlb_topk_gating(const void* logits, int dtype, int64_t tokens, int experts, int top_k, int64_t capacity,
                               void* l_aux, int32_t* ec_idx, void* gate_weights, int64_t* select, void* workspace,
                               size_t workspace_bytes, void* stream) {
  DLB_REQUIRE(tokens > 0 && experts > 0 && experts <= 32 * MAX_VPT, DLB_ERR_INVALID,
              "topk_gating: experts=%d must be in [1, 1024] and tokens positive", experts);
  DLB_REQUIRE(top_k > 0 && top_k <= experts, DLB_ERR_INVALID, "topk_gating: top_k=%d out of range", top_k);
  DLB_REQUIRE(capacity > 0 && capacity <= tokens, DLB_ERR_INVALID,
              "topk_gating: capacity=%lld must be in [1, tokens=%lld]", (long long)capacity, (long long)tokens);
  DLB_REQUIRE(dtype == DLB_F32 || dtype == DLB_F16, DLB_ERR_INVALID, "topk_gating: logits must be fp32 or fp16");
  DLB_REQUIRE(logits && l_aux && ec_idx && gate_weights && select, DLB_ERR_INVALID, "topk_gating: null pointer");
  const GatingWs w = gating_ws(tokens, experts, top_k);
  DLB_REQUIRE(workspace != nullptr && workspace_bytes >= w.bytes, DLB_ERR_WORKSPACE,
              "topk_gating: workspace of %zu bytes needed, %zu given", w.bytes, workspace_bytes);
  char* ws = reinterpret_cast<char*>(workspace);
  float* gates = reinterpret_cast<float*>(ws + w.gates);
  int* ids_km = reinterpret_cast<int*>(ws + w.ids_km);
  float* gate_km = reinterpret_cast<float*>(ws + w.gate_km);
  int* rank = reinterpret_cast<int*>(ws + w.rank);
  float* res = reinterpret_cast<float*>(ws + w.res);
  int* counts = reinterpret_cast<int*>(ws + w.counts);
  cudaStream_t st = (cudaStream_t)stream;
  float* psum = reinterpret_cast<float*>(ws + w.psum);
  int* pcnt = reinterpret_cast<int*>(ws + w.pcnt);
  int* ticket = reinterpret_cast<int*>(ws + w.ticket);
  GatingArgs a = {logits, dtype, tokens, experts, top_k, gates, ids_km, gate_km, psum, pcnt, ticket, st};
  int rc = dispatch_vpt<GatingLauncher>(experts, a);
  if (rc != DLB_OK) return rc;
  // position of every (slot, token) entry inside its expert, in k-major / token-minor order:
  // the cumulative sum of the one-hot masks of the reference (topk_gating_fwd_part2.py:31)
  rc = sort_by_expert(ids_km, DLB_I32, tokens * top_k, experts, nullptr, nullptr, nullptr, nullptr, rank, counts,
                      ws + w.sort, workspace_bytes - w.sort, st);
  if (rc != DLB_OK) return rc;
  const int token_blocks = (int)ceil_div(tokens, 64), expert_blocks = (int)ceil_div(experts, 2);
  auto part3 = [&](auto* out_l_aux, auto* out_w) {
    using T = std::remove_pointer_t<decltype(out_w)>;
    after_predecessor(gating_part3_kernel<T>, token_blocks + expert_blocks, 64, 0, st)(
        ids_km, gate_km, rank, counts, psum, pcnt, gating_blocks(tokens), tokens, experts, top_k, capacity, token_blocks, res,
        reinterpret_cast<float*>(ws + w.ce), ticket, out_l_aux, ec_idx, out_w, reinterpret_cast<long long*>(select));
  };
  if (dtype == DLB_F32) part3(reinterpret_cast<float*>(l_aux), reinterpret_cast<float*>(gate_weights));
  else part3(reinterpret_cast<__half*>(l_aux), reinterpret_cast<__half*>(gate_weights));
  count_launch();
  DLB_CHECK_LAUNCH("gating_part3_kernel");
  return DLB_OK;
}

extern "C" int dlb_topk_gating_bwd(const void* workspace, size_t workspace_bytes, int dtype, int64_t tokens, int experts,
                                   int top_k, int64_t capacity, const void* grad_l_aux, const void* grad_weights,
                                   void* grad_logits, void* stream) {
  DLB_REQUIRE(tokens > 0 && experts > 0 && experts <= 32 * MAX_VPT && top_k > 0 && top_k <= experts, DLB_ERR_INVALID,
              "topk_gating_bwd: bad sizes tokens=%lld experts=%d top_k=%d", (long long)tokens, experts, top_k);
  DLB_REQUIRE(dtype == DLB_F32 || dtype == DLB_F16, DLB_ERR_INVALID, "topk_gating_bwd: dtype must be fp32 or fp16");
  DLB_REQUIRE(workspace && grad_l_aux && grad_logits, DLB_ERR_INVALID, "topk_gating_bwd: null pointer");
  const GatingWs w = gating_ws(tokens, experts, top_k);
  DLB_REQUIRE(workspace_bytes >= w.bytes, DLB_ERR_WORKSPACE,
              "topk_gating_bwd: the forward's workspace has %zu bytes, %zu given", w.bytes, workspace_bytes);
  const char* ws = reinterpret_cast<const char*>(workspace);
  const float* gates = reinterpret_cast<const float*>(ws + w.gates);
  const float* ce = reinterpret_cast<const float*>(ws + w.ce);
  const int* ids_km = reinterpret_cast<const int*>(ws + w.ids_km);
  const float* gate_km = reinterpret_cast<const float*>(ws + w.gate_km);
  const int* rank = reinterpret_cast<const int*>(ws + w.rank);
  GatingBwdArgs a = {gates, ce, ids_km, gate_km, rank, dtype, tokens, experts, top_k, capacity, grad_l_aux, grad_weights,
                     grad_logits, (cudaStream_t)stream};
  return dispatch_vpt<GatingBwdLauncher>(experts, a);
}
