// Fused router tail: logits -> (fp32 softmax) -> top-k -> (softmax over the k) -> (renormalise) -> scores, indices
// and the per-expert load histogram, one warp per token, one launch.
//
// Replaces the chain of torch launches behind topk_router (reference: src/moe_explore/router.py:17-35: softmax,
// torch.topk, softmax, division, cast).  The logits themselves (input @ router_weight) stay a library GEMM.
//
// router_topk_kernel is OPT-IN.  The reference's routing is defined by torch.topk, whose choice among equal logits and whose
// output order (sorted=False) are implementation details of torch; the default router of this package follows them, by the
// torch ops or by router_tail_kernel below, which makes its indices bit-identical to the reference's on the same device.
// router_topk_kernel declares its own rule instead:
//   * among equal values the LOWEST expert index is selected first;
//   * the k selected experts are returned in descending order of value (ties: ascending index);
//   * NaN logits are never selected.
// On inputs without ties among the selected values the SET of indices per token equals torch.topk's.
// Arithmetic is fp32 on the upcast logits; HBM-bound: T*E logits read once, 10*T*k bytes written.
#include "common.cuh"

#include <math_constants.h>

namespace moe {

constexpr int kRouterWarps = 8;
constexpr int kRouterMaxPerLane = 32;  // E <= 1024

template <typename T> __device__ __forceinline__ float load_logit(const T* p) { return Elem<T>::to_float(*p); }
template <> __device__ __forceinline__ float load_logit<float>(const float* p) { return *p; }
template <typename T> __device__ __forceinline__ void store_score(T* p, float v) { *p = Elem<T>::from_float(v); }
template <> __device__ __forceinline__ void store_score<float>(float* p, float v) { *p = v; }

template <typename T, int PER_LANE>
__global__ void __launch_bounds__(kRouterWarps * 32)
router_topk_kernel(const T* __restrict__ logits, T* __restrict__ scores, int64_t* __restrict__ indices,
                   int32_t* __restrict__ expert_counts, int64_t num_tokens, int E, int topk, int softmax_before,
                   int normalize) {
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int64_t t = static_cast<int64_t>(blockIdx.x) * kRouterWarps + warp;
  if (t >= num_tokens) return;
  // expert e = i * 32 + lane lives in v[i]
  float v[PER_LANE];
  const T* row = logits + t * E;
  float vmax = -CUDART_INF_F;
#pragma unroll
  for (int i = 0; i < PER_LANE; ++i) {
    const int e = i * 32 + lane;
    float x = e < E ? load_logit<T>(row + e) : -CUDART_INF_F;
    if (x != x) x = -CUDART_INF_F;  // NaN: never selected
    v[i] = x;
    vmax = fmaxf(vmax, x);
  }
  float denom = 1.0f;
  if (softmax_before) {
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) vmax = fmaxf(vmax, __shfl_xor_sync(0xFFFFFFFFu, vmax, off));
    float sum = 0.0f;
#pragma unroll
    for (int i = 0; i < PER_LANE; ++i) {
      const int e = i * 32 + lane;
      if (e < E && v[i] > -CUDART_INF_F) sum += expf(v[i] - vmax);
    }
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) sum += __shfl_xor_sync(0xFFFFFFFFu, sum, off);
    denom = sum;
  }
  // k rounds of warp arg-max; the winner's slot is cleared.  Lane s keeps the s-th winner (k <= 32).
  float my_val = 0.0f;
  int my_idx = 0;
  for (int s = 0; s < topk; ++s) {
    float best = -CUDART_INF_F;
    int best_e = 0x7FFFFFFF;
#pragma unroll
    for (int i = 0; i < PER_LANE; ++i) {
      const int e = i * 32 + lane;
      if (e < E && v[i] > best) {  // strict: the lowest index of equal values within a lane stays
        best = v[i];
        best_e = e;
      }
    }
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) {
      const float ob = __shfl_xor_sync(0xFFFFFFFFu, best, off);
      const int oe = __shfl_xor_sync(0xFFFFFFFFu, best_e, off);
      if (ob > best || (ob == best && oe < best_e)) {
        best = ob;
        best_e = oe;
      }
    }
    if (best_e == 0x7FFFFFFF) best_e = s < E ? s : 0;  // fewer than k finite logits: deterministic filler
    if ((best_e & 31) == lane) {
#pragma unroll
      for (int i = 0; i < PER_LANE; ++i)
        if (i == (best_e >> 5)) v[i] = -CUDART_INF_F;
    }
    if (lane == s) {
      my_val = best;
      my_idx = best_e;
    }
  }
  // scores of the selected experts
  float score = 0.0f;
  const bool mine = lane < topk;
  if (softmax_before) {
    score = mine && my_val > -CUDART_INF_F ? expf(my_val - vmax) / denom : 0.0f;
  } else {
    float m = mine ? my_val : -CUDART_INF_F;
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) m = fmaxf(m, __shfl_xor_sync(0xFFFFFFFFu, m, off));
    float ex = mine && my_val > -CUDART_INF_F ? expf(my_val - m) : 0.0f;
    float sum = ex;
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) sum += __shfl_xor_sync(0xFFFFFFFFu, sum, off);
    score = sum > 0.0f ? ex / sum : 0.0f;
  }
  if (normalize) {
    float sum = mine ? score : 0.0f;
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) sum += __shfl_xor_sync(0xFFFFFFFFu, sum, off);
    score = score / sum;
  }
  if (mine) {
    store_score<T>(scores + t * topk + lane, score);
    indices[t * topk + lane] = my_idx;
    if (expert_counts != nullptr) atomicAdd(expert_counts + my_idx, 1);
  }
}

template <typename T>
static int launch_router(const void* logits, void* scores, int64_t* indices, int32_t* counts, int64_t T_, int E, int topk,
                         int softmax_before, int normalize, cudaStream_t s) {
  const int blocks = static_cast<int>((T_ + kRouterWarps - 1) / kRouterWarps);
  const T* l = static_cast<const T*>(logits);
  T* sc = static_cast<T*>(scores);
#define MOE_ROUTER(PL)                                                                                                   \
  router_topk_kernel<T, PL><<<blocks, kRouterWarps * 32, 0, s>>>(l, sc, indices, counts, T_, E, topk, softmax_before, normalize)
  if (E <= 64) MOE_ROUTER(2);
  else if (E <= 128) MOE_ROUTER(4);
  else if (E <= 256) MOE_ROUTER(8);
  else if (E <= 512) MOE_ROUTER(16);
  else MOE_ROUTER(32);
#undef MOE_ROUTER
  MOE_CUDA(cudaGetLastError());
  return MOE_OK;
}

}  // namespace moe

using namespace moe;

extern "C" int moe_router_topk(const void* logits, void* scores, int64_t* indices, int32_t* expert_counts,
                               int64_t num_tokens, int num_experts, int topk, int softmax_before_topk, int normalize,
                               int dtype, void* stream) {
  MOE_CHECK_ARG(num_tokens >= 0 && num_experts > 0 && topk > 0, "moe_router_topk: bad sizes T=%lld E=%d k=%d",
                (long long)num_tokens, num_experts, topk);
  if (num_experts > 32 * kRouterMaxPerLane || topk > 32 || topk > num_experts) {
    set_error("moe_router_topk: supports E <= %d and k <= min(32, E); got E=%d k=%d", 32 * kRouterMaxPerLane, num_experts, topk);
    return MOE_ERR_UNSUPPORTED;
  }
  if (num_tokens == 0) return MOE_OK;
  MOE_CHECK_ARG(logits && scores && indices, "moe_router_topk: null pointer argument");
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  if (expert_counts != nullptr) MOE_CUDA(cudaMemsetAsync(expert_counts, 0, sizeof(int32_t) * num_experts, s));
  if (dtype == MOE_DTYPE_BF16)
    return launch_router<__nv_bfloat16>(logits, scores, indices, expert_counts, num_tokens, num_experts, topk,
                                        softmax_before_topk, normalize, s);
  if (dtype == MOE_DTYPE_F16)
    return launch_router<__half>(logits, scores, indices, expert_counts, num_tokens, num_experts, topk, softmax_before_topk,
                                 normalize, s);
  if (dtype == MOE_DTYPE_F32)
    return launch_router<float>(logits, scores, indices, expert_counts, num_tokens, num_experts, topk, softmax_before_topk,
                                normalize, s);
  set_error("moe_router_topk: unknown dtype %d", dtype);
  return MOE_ERR_INVALID;
}

namespace moe {

// The router tail with torch's choices: what softmax, torch.topk(sorted=False), softmax, division by the sum and the cast leave,
// in one launch instead of four to seven (one of which, the radix selection, takes 18-44 us for 3000 to 16384 tokens).  A warp
// per token.
//   * Selection: keys order as the bits do (-0 below +0, NaN above all); the k-th largest key by rounds of redux.sync over what is
//     below the last one; then, as torch writes them, the larger keys in ascending expert index, then keys equal to the k-th in
//     ascending index until k are there.
//   * Arithmetic: the fp32 operations of those launches in their order (a lane's elements 32 apart one by one, then a butterfly,
//     far lanes first), so scores are the same bits.
//   * Order of selection and of summation are torch's own and promised by nobody: as of torch 2.11, which the tests compare with.
// 16384 tokens x 60 experts, four launches of 48 us -> 7.8; 3001 x 128, six of 36 -> 5.0; one token, four of 9.6 -> 2.1.
__device__ __forceinline__ uint32_t order_key(float f) {
  const uint32_t u = __float_as_uint(f);
  return f != f ? 0xFFFFFFFFu : u ^ ((u >> 31) ? 0xFFFFFFFFu : 0x80000000u);
}

//   * With `bias` the selection is by probability + bias and the scores are the probabilities (the ERNIE router); its sum is
//     held at 1e-12 or above (normalize 2).
template <typename T, typename S, int PER_LANE>
__global__ void __launch_bounds__(kRouterWarps * 32)
router_tail_kernel(const T* __restrict__ logits, const float* __restrict__ bias, S* __restrict__ scores, int64_t* __restrict__ indices,
                   int64_t num_tokens, int E, int topk, int softmax_before, int normalize) {
  __shared__ float sh_val[kRouterWarps][32];
  __shared__ int sh_idx[kRouterWarps][32];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int64_t t = static_cast<int64_t>(blockIdx.x) * kRouterWarps + warp;
  if (t >= num_tokens) return;
  const T* row = logits + t * E;
  float v[PER_LANE];  // expert i * 32 + lane
#pragma unroll
  for (int i = 0; i < PER_LANE; ++i) {
    const int e = i * 32 + lane;
    v[i] = e < E ? load_logit<T>(row + e) : -CUDART_INF_F;
  }
  if (softmax_before) {
    float top = v[0];
#pragma unroll
    for (int i = 1; i < PER_LANE; ++i) top = top > v[i] ? top : v[i];
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) {
      const float o = __shfl_xor_sync(0xFFFFFFFFu, top, off);
      top = top < o ? o : top;
    }
    float sum = 0.0f;
#pragma unroll
    for (int i = 0; i < PER_LANE; ++i) {
      v[i] = expf(v[i] - top);
      sum += v[i];
    }
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) sum += __shfl_xor_sync(0xFFFFFFFFu, sum, off);
#pragma unroll
    for (int i = 0; i < PER_LANE; ++i) v[i] = v[i] / sum;
  }
  uint32_t key[PER_LANE];  // 0: no expert (every expert's key is larger)
#pragma unroll
  for (int i = 0; i < PER_LANE; ++i) {
    const int e = i * 32 + lane;
    key[i] = e < E ? order_key(bias != nullptr ? v[i] + bias[e] : v[i]) : 0u;
  }
  uint32_t kth = 0;
  for (int left = topk, first = 1; left > 0; first = 0) {
    uint32_t best = 0;
#pragma unroll
    for (int i = 0; i < PER_LANE; ++i)
      if (first || key[i] < kth) best = key[i] > best ? key[i] : best;
    kth = __reduce_max_sync(0xFFFFFFFFu, best);
#pragma unroll
    for (int i = 0; i < PER_LANE; ++i) left -= __popc(__ballot_sync(0xFFFFFFFFu, key[i] == kth));
  }
  int place = 0;
#pragma unroll
  for (int pass = 0; pass < 2; ++pass) {
#pragma unroll
    for (int i = 0; i < PER_LANE; ++i) {
      const bool take = pass == 0 ? key[i] > kth : key[i] == kth;
      const unsigned all = __ballot_sync(0xFFFFFFFFu, take);
      const int at = place + __popc(all & ((1u << lane) - 1));
      if (take && at < topk) {
        sh_val[warp][at] = v[i];
        sh_idx[warp][at] = i * 32 + lane;
      }
      place += __popc(all);
    }
  }
  __syncwarp();
  const bool mine = lane < topk;
  float s = mine ? sh_val[warp][lane] : -CUDART_INF_F;
  if (!softmax_before) {
    float top = s;
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) {
      const float o = __shfl_xor_sync(0xFFFFFFFFu, top, off);
      top = top < o ? o : top;
    }
    s = mine ? expf(s - top) : 0.0f;
    float sum = s;
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) sum += __shfl_xor_sync(0xFFFFFFFFu, sum, off);
    s = s / sum;
  }
  if (normalize) {
    float sum = mine ? s : 0.0f;
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) sum += __shfl_xor_sync(0xFFFFFFFFu, sum, off);
    if (normalize == 2) sum = sum < 1e-12f ? 1e-12f : sum;
    s = s / sum;
  }
  if (mine) {
    store_score<S>(scores + t * topk + lane, s);
    indices[t * topk + lane] = sh_idx[warp][lane];
  }
}

template <typename T, typename S>
static int launch_router_tail(const void* logits, const float* bias, void* scores, int64_t* indices, int64_t num_tokens, int E,
                              int topk, int softmax_before, int normalize, cudaStream_t s) {
  const int blocks = static_cast<int>((num_tokens + kRouterWarps - 1) / kRouterWarps);
  const T* l = static_cast<const T*>(logits);
  S* sc = static_cast<S*>(scores);
#define MOE_TAIL(PL) \
  router_tail_kernel<T, S, PL><<<blocks, kRouterWarps * 32, 0, s>>>(l, bias, sc, indices, num_tokens, E, topk, softmax_before, normalize)
  if (E <= 32) MOE_TAIL(1);
  else if (E <= 64) MOE_TAIL(2);
  else if (E <= 128) MOE_TAIL(4);
  else if (E <= 256) MOE_TAIL(8);
  else if (E <= 512) MOE_TAIL(16);
  else MOE_TAIL(32);
#undef MOE_TAIL
  MOE_CUDA(cudaGetLastError());
  return MOE_OK;
}

}  // namespace moe

extern "C" int moe_router_tail(const void* logits, const float* bias, void* scores, int64_t* indices, int64_t num_tokens,
                               int num_experts, int topk, int softmax_before_topk, int normalize, int dtype, int scores_dtype,
                               void* stream) {
  MOE_CHECK_ARG(num_tokens >= 0 && num_experts > 0 && topk > 0, "moe_router_tail: bad sizes T=%lld E=%d k=%d",
                (long long)num_tokens, num_experts, topk);
  if (num_experts > 32 * kRouterMaxPerLane || topk > 32 || topk > num_experts || num_tokens > (1ll << 33)) {
    set_error("moe_router_tail: supports E <= %d and k <= min(32, E); got E=%d k=%d", 32 * kRouterMaxPerLane, num_experts, topk);
    return MOE_ERR_UNSUPPORTED;
  }
  if (num_tokens == 0) return MOE_OK;
  MOE_CHECK_ARG(logits && scores && indices, "moe_router_tail: null pointer argument");
  cudaStream_t s = static_cast<cudaStream_t>(stream);
#define MOE_TAIL_TYPES(CODE, T, SCODE, S)                                                                              \
  if (dtype == CODE && scores_dtype == SCODE)                                                                          \
    return launch_router_tail<T, S>(logits, bias, scores, indices, num_tokens, num_experts, topk, softmax_before_topk, \
                                    normalize, s);
  MOE_TAIL_TYPES(MOE_DTYPE_BF16, __nv_bfloat16, MOE_DTYPE_BF16, __nv_bfloat16)
  MOE_TAIL_TYPES(MOE_DTYPE_F16, __half, MOE_DTYPE_F16, __half)
  MOE_TAIL_TYPES(MOE_DTYPE_F32, float, MOE_DTYPE_F32, float)
  MOE_TAIL_TYPES(MOE_DTYPE_F32, float, MOE_DTYPE_BF16, __nv_bfloat16)
  MOE_TAIL_TYPES(MOE_DTYPE_F32, float, MOE_DTYPE_F16, __half)
#undef MOE_TAIL_TYPES
  set_error("moe_router_tail: dtypes %d, %d", dtype, scores_dtype);
  return MOE_ERR_INVALID;
}

namespace moe {

// Backward of the router tail "softmax over the topk selected logits (, renormalised: the same gradient, the softmax sums to
// one)" in one launch: a warp per token recomputes the probabilities p from the logits and leaves
//   dl[t, s] = p_s (d_s - sum_j p_j d_j)   in fp32, and the dense row of it in the 16-bit type (what the router-weight
// gradient contracts with; its rows are padded with zeros to whole 16 bytes, so that the contraction is an aligned one: 60
// experts, 16384 tokens 53 -> 22 us); the CTAs after those transpose the router weight for the fold of the input gradient.
// It stands for seven element-wise launches (casts, product, softmax backward, fill, scatter: 25-30 us).
constexpr int kTransposeTile = 32;
template <typename T>
__global__ void __launch_bounds__(256)
router_backward_kernel(const T* logits, const int64_t* experts, const T* d_scores, const T* router_w, float* dl, T* dlogits,
                       T* router_t, int64_t num_tokens, int E, int topk, int cols, int token_blocks) {
  const int ld = (E + 7) & ~7;  // of dlogits
  grid_release();
  grid_wait();
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  if (static_cast<int>(blockIdx.x) < token_blocks) {
    for (int64_t t = static_cast<int64_t>(blockIdx.x) * 8 + warp; t < num_tokens; t += static_cast<int64_t>(token_blocks) * 8) {
      const T* row = logits + t * E;
      // slots in rounds of 32 lanes (one round up to 32 slots); the three passes re-read a few cached words
      float top = -INFINITY;
      for (int s = lane; s < topk; s += 32) top = fmaxf(top, Elem<T>::to_float(row[experts[t * topk + s]]));
#pragma unroll
      for (int off = 16; off > 0; off >>= 1) top = fmaxf(top, __shfl_xor_sync(0xFFFFFFFFu, top, off));
      float sum = 0.0f, dot = 0.0f;
      for (int s = lane; s < topk; s += 32) {
        const float w = expf(Elem<T>::to_float(row[experts[t * topk + s]]) - top);
        sum += w;
        dot = fmaf(w, Elem<T>::to_float(d_scores[t * topk + s]), dot);
      }
#pragma unroll
      for (int off = 16; off > 0; off >>= 1) {
        sum += __shfl_xor_sync(0xFFFFFFFFu, sum, off);
        dot += __shfl_xor_sync(0xFFFFFFFFu, dot, off);
      }
      dot /= sum;
      for (int e = lane; e < ld; e += 32) dlogits[t * ld + e] = Elem<T>::from_float(0.0f);
      __syncwarp();
      for (int s = lane; s < topk; s += 32) {
        const int64_t e = experts[t * topk + s];
        const float p = expf(Elem<T>::to_float(row[e]) - top) / sum;
        const float g = p * (Elem<T>::to_float(d_scores[t * topk + s]) - dot);
        dl[t * topk + s] = g;
        dlogits[t * ld + e] = Elem<T>::from_float(g);
      }
    }
    return;
  }
  // router_t[e, c] = router_w[c, e]
  __shared__ T tile[kTransposeTile][kTransposeTile + 2];
  const int tiles_e = (E + kTransposeTile - 1) / kTransposeTile;
  const int b = blockIdx.x - token_blocks;
  const int e0 = (b % tiles_e) * kTransposeTile, c0 = (b / tiles_e) * kTransposeTile;
  for (int i = warp; i < kTransposeTile; i += 8)
    if (c0 + i < cols && e0 + lane < E) tile[i][lane] = router_w[static_cast<int64_t>(c0 + i) * E + e0 + lane];
  __syncthreads();
  for (int i = warp; i < kTransposeTile; i += 8)
    if (e0 + i < E && c0 + lane < cols) router_t[static_cast<int64_t>(e0 + i) * cols + c0 + lane] = tile[lane][i];
}

int router_backward(const void* logits, const int64_t* experts, const void* d_scores, const void* router_w, float* dl,
                    void* dlogits, void* router_t, int64_t num_tokens, int num_experts, int topk, int cols, int dtype,
                    void* stream) {
  MOE_CHECK_ARG(logits && experts && d_scores && router_w && dl && dlogits && router_t, "router backward: null pointer argument");
  MOE_CHECK_ARG(num_tokens > 0 && num_experts > 0 && topk > 0 && cols > 0, "router backward: bad sizes");
  MOE_CHECK_ARG(dtype == MOE_DTYPE_BF16 || dtype == MOE_DTYPE_F16, "router backward: unknown dtype %d", dtype);
  const int64_t want = (num_tokens + 7) / 8, cap = static_cast<int64_t>(sm_count()) * 8;
  const int token_blocks = static_cast<int>(want < cap ? want : cap);
  const int tiles = ((num_experts + kTransposeTile - 1) / kTransposeTile) * ((cols + kTransposeTile - 1) / kTransposeTile);
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  const auto go = [&](auto kernel, auto type) {
    using T = decltype(type);
    return launch_kernel(kernel, token_blocks + tiles, 256, s, static_cast<const T*>(logits), experts,
                         static_cast<const T*>(d_scores), static_cast<const T*>(router_w), dl, static_cast<T*>(dlogits),
                         static_cast<T*>(router_t), num_tokens, num_experts, topk, cols, token_blocks);
  };
  MOE_CUDA(dtype == MOE_DTYPE_BF16 ? go(router_backward_kernel<__nv_bfloat16>, __nv_bfloat16{})
                                   : go(router_backward_kernel<__half>, __half{}));
  return MOE_OK;
}

}  // namespace moe
