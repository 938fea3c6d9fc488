// Shared host/device helpers for the sm_100a MoE expert-compute library.
//
// Everything here is internal: the only public surface is the C-ABI declared in
// include/moe_sm100.h.  Host helpers record a thread-local error string that
// moe_last_error() returns; device helpers wrap the PTX this library issues by hand
// (mbarrier, TMA tile loads, tcgen05 MMA / TMEM).
#pragma once

#include <cuda.h>
#include <cuda_runtime.h>
#include <cuda_bf16.h>
#include <cuda_fp16.h>
#include <stdint.h>
#include <stdio.h>
#include <stdarg.h>

#include "../../include/moe_sm100.h"

namespace moe {

// ----------------------------------------------------------------------------------
// host side: error reporting
// ----------------------------------------------------------------------------------
void set_error(const char* fmt, ...);
int cuda_fail(cudaError_t e, const char* what);

#define MOE_CHECK_ARG(cond, ...)                       \
  do {                                                 \
    if (!(cond)) {                                     \
      ::moe::set_error(__VA_ARGS__);                   \
      return MOE_ERR_INVALID;                          \
    }                                                  \
  } while (0)

#define MOE_CUDA(call)                                 \
  do {                                                 \
    cudaError_t e__ = (call);                          \
    if (e__ != cudaSuccess) return ::moe::cuda_fail(e__, #call); \
  } while (0)

int sm_count();  // SM count of the current device (cached per device)

// Chained launches.  Inside one library call that launches several kernels in a row on one stream, the kernels after the
// first are launched with programmatic stream serialization: their launch and prologue (barriers, TMEM, descriptors)
// overlap the tail of the kernel before, and grid_wait() holds them back until that kernel has completed and its writes are
// visible.  Every kernel that can be launched so calls grid_wait() before its first access to global memory (but
// for what RowCounts::settled names) and before it ends, so the order of the stream holds for all earlier kernels too.  Thread-local and set only for the duration of such a call.
bool& chained_launches();

class Chain {
 public:
  Chain() { chained_launches() = false; }
  ~Chain() { chained_launches() = false; }
};

#define MOE_STEP(call)                  \
  do {                                  \
    const int rc__ = (call);            \
    if (rc__ != MOE_OK) return rc__;    \
    ::moe::chained_launches() = true;   \
  } while (0)

// In a row map for gather_rows with skip_marked: leave the row of dst as it is.
constexpr int32_t kSkipRow = -2;

template <typename... Params, typename... Args>
inline cudaError_t launch_kernel(void (*kernel)(Params...), int grid, int block, cudaStream_t stream, Args... args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(static_cast<unsigned>(grid), 1, 1);
  cfg.blockDim = dim3(static_cast<unsigned>(block), 1, 1);
  cfg.stream = stream;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = chained_launches() ? 1 : 0;
  return cudaLaunchKernelEx(&cfg, kernel, static_cast<Params>(args)...);
}

// moe_routing_metadata; `workspace_always` false: a workspace is asked for only where the kernels use one (csrc/routing.cu).
int routing_metadata(const int64_t* expert_idx, int64_t num_rows, int num_experts, int32_t* group_indices, int64_t* perm,
                     int32_t* pad_offsets, int32_t* row_src, int32_t* dst_row, int32_t* mtile_expert, int32_t* tile_pairs,
                     int32_t* num_mtiles, int32_t* status, void* workspace, size_t workspace_bytes,
                     bool workspace_always, void* stream);

// The rows that exist in the padded layout (both null: all of them): see GemmArgs::group_indices.
struct RowCounts {
  const int32_t* pad_offsets = nullptr;
  const int32_t* group_indices = nullptr;
  // Operands and results that are not in the padded layout but hold their rows without padding, expert by expert: their row
  // counts (-1: padded).  With one expert that is a plain matrix; the copy engine fills loads past its end with zeros and
  // drops stores there.
  int64_t a_rows = -1;
  int64_t b_rows = -1;    // K-grouped
  int64_t out_rows = -1;  // M-grouped plain stores, one expert
  // A word that work items are claimed from (GemmArgs::work_counter), zero; null: they are dealt out.
  uint32_t* work_counter = nullptr;
  int64_t routed_rows = -1;  // M-grouped: about how many rows there are (what sizes row units and decides on claiming; required)
  // The kernel that wrote the maps and counts is complete, and so is whatever wrote the weights, before a contraction that is
  // chained to the kernel before it can begin: that kernel (or one since) lets its successor up only after its own grid_wait().
  // Complete is not yet visible to every load before the contraction's own grid_wait(): it reads the maps and counts past L1
  // (map_word in gemm_kernel.cuh), and the weights as copies, which do not go through L1.
  bool settled = false;
};
// Words that the first row kernel of a pass, or its layout kernel, sets to zero for the contractions after it.
constexpr int kWorkCounters = 4;

// The entry points of the same names, told which rows exist.
int mgrouped_gemm(const void* a, const void* w, void* out, void* pre_act, const int32_t* mtile_expert, const int32_t*
                  tile_pairs, const int32_t* num_mtiles, int64_t padded_rows, int K, int N, int num_experts, int
                  w_transposed, int act, int dtype, int chunk_index, int chunk_count, const moe_gemm_options* options,
                  int32_t* status, void* stream, const RowCounts& counts);
int mgrouped_gemm_gather(const void* src, int64_t src_rows, const int32_t* row_src, int div, const void* w, void* out,
                         void* pre_act, const int32_t* mtile_expert, const int32_t* tile_pairs, const int32_t* num_mtiles,
                         int64_t padded_rows, int K, int N, int num_experts, int act, int dtype, const moe_gemm_options*
                         options, int32_t* status, void* stream, const RowCounts& counts);
int mgrouped_gemm_combine(const void* a, const void* w, void* out, const int32_t* row_src, const void* scores, int topk,
                          const int32_t* mtile_expert, const int32_t* tile_pairs, const int32_t* num_mtiles, int64_t
                          padded_rows, int K, int N, int num_experts, int w_transposed, int dtype, const moe_gemm_options*
                          options, int32_t* status, void* stream, const RowCounts& counts);
int mgrouped_gemm_dglu(const void* g, const void* w, const void* pre_act, void* d_pre, const int32_t* mtile_expert, const
                       int32_t* tile_pairs, const int32_t* num_mtiles, int64_t padded_rows, int K, int N, int num_experts,
                       int act, int dtype, int chunk_index, int chunk_count, const moe_gemm_options* options, int32_t*
                       status, void* stream, const RowCounts& counts);
int kgrouped_gemm(const void* a, const void* b, void* dw, const int32_t* pad_offsets, int64_t padded_rows, int M, int N,
                  int num_experts, int dtype, const moe_gemm_options* options, int32_t* status, void* stream, const
                  RowCounts& counts);
int kgrouped_gemm_gather(const void* src, int64_t src_rows, const int32_t* row_src, int div, const void* b, void* dw,
                         const int32_t* pad_offsets, int64_t padded_rows, int M, int N, int num_experts, int dtype, const
                         moe_gemm_options* options, int32_t* status, void* stream, const RowCounts& counts);

// Grouped GEMM whose row p goes to out_rows[p] (negative: nowhere), gated activations included; compact_rows >= 0: `a` holds
// that many rows in expert order without padding.
int mgrouped_gemm_rows(const void* a, int64_t compact_rows, const void* w, void* out, const int32_t* out_rows,
                       const int32_t* mtile_expert, const int32_t* tile_pairs, const int32_t* num_mtiles, int64_t padded_rows,
                       int K, int N, int num_experts, int act, int dtype, int32_t* status, void* stream,
                       const RowCounts& counts);
// moe_gather_rows; `skip_marked`: row_src comes from the library and its kSkipRow entries are obeyed.
int gather_rows(const void* src, int64_t src_rows, const int32_t* row_src, const int32_t* num_mtiles, void* dst,
                int64_t padded_rows, int cols, int div, int dtype, void* stream, bool skip_marked);
int dispatch_rows(const void* src, const int32_t* dst_row, const int32_t* row_src, const int32_t* num_mtiles, void* dst,
                  int64_t num_tokens, int topk, int64_t padded_rows, int cols, int dtype, void* stream, bool live_blocks_only,
                  uint32_t* work_counters);
int dispatch_rows_only(const void* src, const int32_t* dst_row, void* dst, int64_t num_tokens, int topk, int cols, int dtype,
                       void* stream, uint32_t* work_counters, void* clear);
// moe_combine_topk with further summands, all nullable (FoldExtra in csrc/rows.cu).
int combine_topk(const void* ys, const void* scores, const int32_t* dst_row, void* out, int64_t num_tokens, int topk, int cols,
                 int dtype, const void* addend, const float* dlogits, const int64_t* experts, const void* router_t,
                 void* stream);
// Backward of "softmax over the selected logits" (csrc/router.cu).
int router_backward(const void* logits, const int64_t* experts, const void* d_scores, const void* router_w, float* dl,
                    void* dlogits, void* router_t, int64_t num_tokens, int num_experts, int topk, int cols, int dtype,
                    void* stream);
int combine_bwd_tokens(const void* dout, const void* scores, const void* ys, const int32_t* dst_row, const int32_t* row_src,
                       const int32_t* num_mtiles, void* gs, void* dscores, int64_t num_tokens, int topk, int cols, int dtype,
                       void* stream, bool live_blocks_only, uint32_t* work_counters);

// Status codes written by kernels into the caller's device status word.
enum DeviceStatus : int {
  DS_OK = 0,
  DS_TIMEOUT_PRODUCER = 1,  // TMA producer gave up waiting for a free shared-memory stage
  DS_TIMEOUT_MMA = 2,       // MMA issuer gave up waiting for operands or a free accumulator
  DS_TIMEOUT_EPILOGUE = 3,  // epilogue gave up waiting for an accumulator
  DS_WAVE_FALLBACK = 4,     // the wave barrier of the persistent workers ran out; the launch finished with the static
                            // stride instead (its results are valid)
  DS_BAD_LAYOUT = 5,        // the routing metadata handed to a kernel was built for another padded row count
  DS_BAD_EXPERT_ID = 100,   // routing metadata saw an expert id outside [0, num_experts); the row was dropped
};

// Limit (in SM clock cycles) of every device-side wait of the launches that follow; see moe_set_wait_limit_cycles.
long long wait_limit_cycles();

// ----------------------------------------------------------------------------------
// device side: element types
// ----------------------------------------------------------------------------------
template <typename T> struct Elem;
template <> struct Elem<__nv_bfloat16> {
  static constexpr uint32_t kUmmaFormat = 1;  // BF16 operand code of the tcgen05 instruction descriptor
  __device__ static __forceinline__ uint32_t pack2(float a, float b) {
    __nv_bfloat162 v = __floats2bfloat162_rn(a, b);
    return *reinterpret_cast<uint32_t*>(&v);
  }
  __device__ static __forceinline__ float2 unpack2(uint32_t u) {
    __nv_bfloat162 v = *reinterpret_cast<__nv_bfloat162*>(&u);
    return __bfloat1622float2(v);
  }
  __device__ static __forceinline__ float to_float(__nv_bfloat16 v) { return __bfloat162float(v); }
  __device__ static __forceinline__ __nv_bfloat16 from_float(float v) { return __float2bfloat16_rn(v); }
};
template <> struct Elem<__half> {
  static constexpr uint32_t kUmmaFormat = 0;  // F16 operand code
  __device__ static __forceinline__ uint32_t pack2(float a, float b) {
    __half2 v = __floats2half2_rn(a, b);
    return *reinterpret_cast<uint32_t*>(&v);
  }
  __device__ static __forceinline__ float2 unpack2(uint32_t u) {
    __half2 v = *reinterpret_cast<__half2*>(&u);
    return __half22float2(v);
  }
  __device__ static __forceinline__ float to_float(__half v) { return __half2float(v); }
  __device__ static __forceinline__ __half from_float(float v) { return __float2half_rn(v); }
};

// ----------------------------------------------------------------------------------
// device side: PTX wrappers
// ----------------------------------------------------------------------------------
__device__ __forceinline__ uint32_t smem_u32(const void* p) {
  return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}

// See chained_launches(): waits for the kernels this one was chained to / lets the next chained kernel start its prologue.
// A chained kernel begins before its predecessor has written the last of what it reads.  So in a kernel that can be launched
// chained nothing may be promised to be constant for the kernel's whole life: its pointer parameters carry no __restrict__ and it
// reads without __ldg (either lets the compiler use the non-coherent path, or move a load over the wait); what the
// predecessor wrote is then read by ordinary loads after grid_wait(), which makes it visible.  Functions that run after the wait
// may take __restrict__ pointers: their promise begins there.
__device__ __forceinline__ void grid_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void grid_release() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }

__device__ __forceinline__ void mbar_init(uint32_t bar, uint32_t count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bar), "r"(count) : "memory");
}
__device__ __forceinline__ void mbar_fence_init() {
  asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
}
__device__ __forceinline__ void mbar_arrive_expect_tx(uint32_t bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
}
__device__ __forceinline__ void mbar_arrive(uint32_t bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory");
}
__device__ __forceinline__ bool mbar_try_wait(uint32_t bar, uint32_t parity) {
  uint32_t ok;
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
      "selp.b32 %0, 1, 0, p;\n\t}"
      : "=r"(ok)
      : "r"(bar), "r"(parity)
      : "memory");
  return ok != 0;
}

// True in exactly one lane of a fully converged warp.
__device__ __forceinline__ bool elect_one() {
  uint32_t pred;
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "elect.sync _|p, 0xFFFFFFFF;\n\t"
      "selp.b32 %0, 1, 0, p;\n\t}"
      : "=r"(pred));
  return pred != 0;
}

// Non-blocking probe of a barrier phase (try_wait may suspend the thread for a while when the phase is not
// complete; this one returns at once).
__device__ __forceinline__ bool mbar_test_wait(uint32_t bar, uint32_t parity) {
  uint32_t ok;
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "mbarrier.test_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
      "selp.b32 %0, 1, 0, p;\n\t}"
      : "=r"(ok)
      : "r"(bar), "r"(parity)
      : "memory");
  return ok != 0;
}

// Every wait in this library is bounded: after `limit` clock cycles the waiter raises the abort flag of its
// CTA (and of the other CTA of its pair), records why in the caller's status word and returns false.  All
// other waiters see the flag and give up too, so the kernel always terminates by itself.
constexpr long long kDefaultWaitLimitCycles = 1ll << 32;  // ~2 s at B200 clocks

struct WaitCtx {
  volatile int* abort_flag;  // this CTA's flag (shared memory)
  uint32_t peer_abort;       // shared::cluster address of the flag of the other CTA of the pair; 0 without a pair
  int* status;               // caller's status word (may be null)
  long long limit;           // cycles
};

__device__ __forceinline__ void raise_abort(const WaitCtx& w, int code) {
  *w.abort_flag = 1;
  if (w.peer_abort != 0) asm volatile("st.shared::cluster.u32 [%0], %1;" ::"r"(w.peer_abort), "r"(1) : "memory");
  if (w.status != nullptr) atomicCAS(w.status, 0, code);
}

__device__ __forceinline__ bool mbar_wait(uint32_t bar, uint32_t parity, const WaitCtx& w, int code) {
  if (mbar_try_wait(bar, parity)) return true;
  const long long t0 = clock64();
  int spins = 0;
  while (true) {
    if (mbar_try_wait(bar, parity)) return true;
    if (((++spins) & 63) == 0) {
      if (*w.abort_flag) return false;
      if (clock64() - t0 > w.limit) {
        raise_abort(w, code);
        return false;
      }
    }
  }
}

// TMA tile loads (no cluster qualifiers anywhere: every CTA fetches its own tiles).
// L2 policy handed to the tile loads (normal priority: marking weight tiles evict-first made CTA pairs that share a
// weight tile miss it, measured +50 % DRAM reads).
__device__ __forceinline__ uint64_t l2_policy_evict_normal() {
  uint64_t p;
  asm volatile("createpolicy.fractional.L2::evict_normal.b64 %0, 1.0;" : "=l"(p));
  return p;
}
__device__ __forceinline__ void tma_load_2d(uint32_t dst, const CUtensorMap* map, int c0, int c1, uint32_t bar,
                                            uint64_t policy) {
  asm volatile(
      "cp.async.bulk.tensor.2d.shared::cta.global.tile.mbarrier::complete_tx::bytes.L2::cache_hint "
      "[%0], [%1, {%2, %3}], [%4], %5;"
      ::"r"(dst), "l"(map), "r"(c0), "r"(c1), "r"(bar), "l"(policy)
      : "memory");
}
__device__ __forceinline__ void tma_load_3d(uint32_t dst, const CUtensorMap* map, int c0, int c1, int c2,
                                            uint32_t bar, uint64_t policy) {
  asm volatile(
      "cp.async.bulk.tensor.3d.shared::cta.global.tile.mbarrier::complete_tx::bytes.L2::cache_hint "
      "[%0], [%1, {%2, %3, %4}], [%5], %6;"
      ::"r"(dst), "l"(map), "r"(c0), "r"(c1), "r"(c2), "r"(bar), "l"(policy)
      : "memory");
}
__device__ __forceinline__ void tma_load_4d(uint32_t dst, const CUtensorMap* map, int c0, int c1, int c2, int c3,
                                            uint32_t bar, uint64_t policy) {
  asm volatile(
      "cp.async.bulk.tensor.4d.shared::cta.global.tile.mbarrier::complete_tx::bytes.L2::cache_hint "
      "[%0], [%1, {%2, %3, %4, %5}], [%6], %7;"
      ::"r"(dst), "l"(map), "r"(c0), "r"(c1), "r"(c2), "r"(c3), "r"(bar), "l"(policy)
      : "memory");
}
__device__ __forceinline__ void tma_prefetch_desc(const CUtensorMap* map) {
  asm volatile("prefetch.tensormap [%0];" ::"l"(map) : "memory");
}

// Four rows of a 2-D tensor gathered by row index into four consecutive 128-byte shared-memory rows (tensor map
// with a {64, 1} box and the 128-byte swizzle).  Rows outside the tensor read as zeros.  c0 (elements) must be a
// multiple of 8.  Any number of lanes of a warp may issue one of these each.
__device__ __forceinline__ void tma_gather4(uint32_t dst, const CUtensorMap* map, int c0, const int4& rows, uint32_t bar,
                                            uint64_t policy) {
  asm volatile(
      "cp.async.bulk.tensor.2d.shared::cta.global.tile::gather4.mbarrier::complete_tx::bytes.cta_group::1.L2::cache_hint "
      "[%0], [%1, {%2, %3, %4, %5, %6}], [%7], %8;"
      ::"r"(dst), "l"(map), "r"(c0), "r"(rows.x), "r"(rows.y), "r"(rows.z), "r"(rows.w), "r"(bar), "l"(policy)
      : "memory");
}
// The same issued by either CTA of a pair, the bytes credited to `bar` in the shared::cluster window.
__device__ __forceinline__ void tma_gather4_pair(uint32_t dst, const CUtensorMap* map, int c0, const int4& rows,
                                                 uint32_t bar, uint64_t policy) {
  asm volatile(
      "cp.async.bulk.tensor.2d.shared::cluster.global.tile::gather4.mbarrier::complete_tx::bytes.cta_group::2.L2::cache_hint "
      "[%0], [%1, {%2, %3, %4, %5, %6}], [%7], %8;"
      ::"r"(dst), "l"(map), "r"(c0), "r"(rows.x), "r"(rows.y), "r"(rows.z), "r"(rows.w), "r"(bar), "l"(policy)
      : "memory");
}
// Plain 2-D tile load without a cache hint (epilogue side inputs).
__device__ __forceinline__ void tma_load_2d_plain(uint32_t dst, const CUtensorMap* map, int c0, int c1, uint32_t bar) {
  asm volatile(
      "cp.async.bulk.tensor.2d.shared::cta.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];"
      ::"r"(dst), "l"(map), "r"(c0), "r"(c1), "r"(bar)
      : "memory");
}
// 2-D tile store from shared memory (bulk async-group completion); parts of the box outside the tensor are dropped.
__device__ __forceinline__ void tma_store_2d(const CUtensorMap* map, int c0, int c1, uint32_t src) {
  asm volatile("cp.async.bulk.tensor.2d.global.shared::cta.tile.bulk_group [%0, {%1, %2}], [%3];"
               ::"l"(map), "r"(c0), "r"(c1), "r"(src)
               : "memory");
}
__device__ __forceinline__ void tma_store_3d(const CUtensorMap* map, int c0, int c1, int c2, uint32_t src) {
  asm volatile("cp.async.bulk.tensor.3d.global.shared::cta.tile.bulk_group [%0, {%1, %2, %3}], [%4];"
               ::"l"(map), "r"(c0), "r"(c1), "r"(c2), "r"(src)
               : "memory");
}
__device__ __forceinline__ void bulk_commit() { asm volatile("cp.async.bulk.commit_group;" ::: "memory"); }
// Wait until the bulk stores committed by this thread have finished READING shared memory (the buffer may be reused).
__device__ __forceinline__ void bulk_wait_read_all() { asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory"); }
// The same, all but the last committed group.
__device__ __forceinline__ void bulk_wait_read_one() { asm volatile("cp.async.bulk.wait_group.read 1;" ::: "memory"); }
// Wait until the bulk stores committed by this thread are complete.
__device__ __forceinline__ void bulk_wait_all() { asm volatile("cp.async.bulk.wait_group 0;" ::: "memory"); }
// Orders this thread's generic-proxy shared-memory writes before later async-proxy (TMA) reads of them.
__device__ __forceinline__ void fence_proxy_async_smem() { asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); }

// TMEM allocation (whole warp executes these).
__device__ __forceinline__ void tmem_alloc(uint32_t smem_slot, uint32_t ncols) {
  asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_slot), "r"(ncols)
               : "memory");
}
__device__ __forceinline__ void tmem_relinquish() {
  asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void tmem_dealloc(uint32_t taddr, uint32_t ncols) {
  asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(taddr), "r"(ncols) : "memory");
}
__device__ __forceinline__ void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }

// D[tmem] (+)= A[smem desc] * B[smem desc], 16-bit inputs, fp32 accumulate; one thread issues.
__device__ __forceinline__ void umma_f16(uint32_t d_tmem, uint64_t a_desc, uint64_t b_desc, uint32_t idesc,
                                         uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}"
      ::"r"(d_tmem), "l"(a_desc), "l"(b_desc), "r"(idesc), "r"(accumulate)
      : "memory");
}
// Arrive on an mbarrier once every MMA issued so far by this thread has completed.
__device__ __forceinline__ void umma_commit(uint32_t bar) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar) : "memory");
}

// ---- CTA-pair (cluster of 2) variants: one MMA spans the tensor cores of two SMs ----
__device__ __forceinline__ uint32_t cluster_ctarank() {
  uint32_t r;
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
  return r;
}
// Address of the same shared-memory location in CTA `rank` of this cluster (shared::cluster window).
__device__ __forceinline__ uint32_t mapa_shared(uint32_t addr, uint32_t rank) {
  uint32_t r;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(addr), "r"(rank));
  return r;
}
__device__ __forceinline__ void cluster_sync_all() {
  asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
__device__ __forceinline__ void mbar_arrive_cluster(uint32_t cluster_addr) {
  asm volatile("mbarrier.arrive.shared::cluster.b64 _, [%0];" ::"r"(cluster_addr) : "memory");
}
// Four words into either CTA's shared memory, their 16 bytes credited to that CTA's barrier when they are there (visible to whoever
// waits for it, as a copy's bytes are).
__device__ __forceinline__ void st_async_v4(uint32_t cluster_addr, int a, int b, int c, int d, uint32_t cluster_bar) {
  asm volatile("st.async.weak.shared::cluster.mbarrier::complete_tx::bytes.v4.b32 [%0], {%1, %2, %3, %4}, [%5];"
               ::"r"(cluster_addr), "r"(a), "r"(b), "r"(c), "r"(d), "r"(cluster_bar)
               : "memory");
}
__device__ __forceinline__ void mbar_arrive_expect_tx_cluster(uint32_t cluster_addr, uint32_t bytes) {
  // default (CTA-scope) ordering: the operand bytes are published by the copies' own complete_tx, not by this
  // arrive, and a cluster-scope release here would put a full fence in front of every stage
  asm volatile("mbarrier.arrive.expect_tx.shared::cluster.b64 _, [%0], %1;" ::"r"(cluster_addr), "r"(bytes)
               : "memory");
}
// Tile loads issued by either CTA of a pair: data lands in the issuing CTA's shared memory, the
// transaction bytes are credited to `bar`, an mbarrier address in the shared::cluster window (the
// pair leader's barrier).  Each CTA fetches its own tiles; nothing is broadcast.
__device__ __forceinline__ void tma_load_2d_pair(uint32_t dst, const CUtensorMap* map, int c0, int c1, uint32_t bar,
                                                 uint64_t policy) {
  asm volatile(
      "cp.async.bulk.tensor.2d.shared::cluster.global.tile.mbarrier::complete_tx::bytes.cta_group::2.L2::cache_hint "
      "[%0], [%1, {%2, %3}], [%4], %5;"
      ::"r"(dst), "l"(map), "r"(c0), "r"(c1), "r"(bar), "l"(policy)
      : "memory");
}
__device__ __forceinline__ void tma_load_3d_pair(uint32_t dst, const CUtensorMap* map, int c0, int c1, int c2,
                                                 uint32_t bar, uint64_t policy) {
  asm volatile(
      "cp.async.bulk.tensor.3d.shared::cluster.global.tile.mbarrier::complete_tx::bytes.cta_group::2.L2::cache_hint "
      "[%0], [%1, {%2, %3, %4}], [%5], %6;"
      ::"r"(dst), "l"(map), "r"(c0), "r"(c1), "r"(c2), "r"(bar), "l"(policy)
      : "memory");
}
__device__ __forceinline__ void tma_load_4d_pair(uint32_t dst, const CUtensorMap* map, int c0, int c1, int c2, int c3,
                                                 uint32_t bar, uint64_t policy) {
  asm volatile(
      "cp.async.bulk.tensor.4d.shared::cluster.global.tile.mbarrier::complete_tx::bytes.cta_group::2.L2::cache_hint "
      "[%0], [%1, {%2, %3, %4, %5}], [%6], %7;"
      ::"r"(dst), "l"(map), "r"(c0), "r"(c1), "r"(c2), "r"(c3), "r"(bar), "l"(policy)
      : "memory");
}
__device__ __forceinline__ void tmem_alloc_pair(uint32_t smem_slot, uint32_t ncols) {
  asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_slot), "r"(ncols)
               : "memory");
}
__device__ __forceinline__ void tmem_relinquish_pair() {
  asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void tmem_dealloc_pair(uint32_t taddr, uint32_t ncols) {
  asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(taddr), "r"(ncols) : "memory");
}
// One MMA over both CTAs of the pair: 256 accumulator rows (128 in each CTA's TMEM), A rows and B
// columns split between the two CTAs' shared memory.  Issued by one thread of the leader CTA.
__device__ __forceinline__ void umma_f16_pair(uint32_t d_tmem, uint64_t a_desc, uint64_t b_desc, uint32_t idesc,
                                              uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::2.kind::f16 [%0], %1, %2, %3, p;\n\t}"
      ::"r"(d_tmem), "l"(a_desc), "l"(b_desc), "r"(idesc), "r"(accumulate)
      : "memory");
}
// `bar` is an address in the shared::cluster window (own or peer CTA).
__device__ __forceinline__ void umma_commit_pair(uint32_t bar) {
  asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar) : "memory");
}

// One commit that arrives on the barrier at the same shared-memory offset in both CTAs of the pair
// (the arrival is broadcast by the commit itself; no operand load carries a cluster qualifier).
__device__ __forceinline__ void umma_commit_pair_both(uint32_t bar) {
  asm volatile(
      "tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;" ::"r"(bar),
      "h"(static_cast<uint16_t>(3))
      : "memory");
}

// 32 lanes x 32 consecutive fp32 columns: thread i of the warp receives lane (base+i).
__device__ __forceinline__ void tmem_ld_32x32(uint32_t taddr, uint32_t (&v)[32]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x32.b32 "
      "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, "
      "%16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%32];"
      : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]),
        "=r"(v[8]), "=r"(v[9]), "=r"(v[10]), "=r"(v[11]), "=r"(v[12]), "=r"(v[13]), "=r"(v[14]), "=r"(v[15]),
        "=r"(v[16]), "=r"(v[17]), "=r"(v[18]), "=r"(v[19]), "=r"(v[20]), "=r"(v[21]), "=r"(v[22]), "=r"(v[23]),
        "=r"(v[24]), "=r"(v[25]), "=r"(v[26]), "=r"(v[27]), "=r"(v[28]), "=r"(v[29]), "=r"(v[30]), "=r"(v[31])
      : "r"(taddr)
      : "memory");
}
__device__ __forceinline__ void tmem_ld_wait() { asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory"); }

// 16 bytes (eight 16-bit values) added to global memory element-wise, no return value.
template <typename T> __device__ __forceinline__ void red_add_v8(void* ptr, const uint4& v);
template <> __device__ __forceinline__ void red_add_v8<__nv_bfloat16>(void* ptr, const uint4& v) {
  asm volatile("red.global.add.noftz.v4.bf16x2 [%0], {%1, %2, %3, %4};" ::"l"(ptr), "r"(v.x), "r"(v.y), "r"(v.z), "r"(v.w)
               : "memory");
}
template <> __device__ __forceinline__ void red_add_v8<__half>(void* ptr, const uint4& v) {
  asm volatile("red.global.add.noftz.v4.f16x2 [%0], {%1, %2, %3, %4};" ::"l"(ptr), "r"(v.x), "r"(v.y), "r"(v.z), "r"(v.w)
               : "memory");
}

// Activation math (fp32).
// e^x = 2^(x log2 e), by the approximation that flushes: 0 below the normal range.
__device__ __forceinline__ float exp_flush(float x) {
  float r;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x * 1.4426950408889634f));
  return r;
}
// 1 / (1 + e^-x).  The reciprocal is one step of the Newton-Raphson iteration r' = r + r (1 - y r), whose relative error is the
// square of r's, from the hardware's approximation (relative error 2^-23: the step leaves the rounding of its last
// operation).  Straight-line code, because the elements of an epilogue row have to be interleaved: with two warps per scheduler
// that is the whole speed of the gated epilogues (dGLU at 16384 tokens x 4 slots, 60 experts, K 2048: 229 -> 204 us against the
// division operator).  y is a quarter of 1 + e^-x, so that the flushing forms serve: e^-x below the normal range adds nothing to 1,
// and 4 / (1 + e^-x) stays above it; the last product may then leave a result below (gates under -87).  The cap makes the step
// from r = 0 at y = infinity a finite one; r itself is taken of y, so that NaN comes out as it is.  Measured against the forms
// that do not flush: a 32 x 32 block of the gated backward 2093 -> 1743 cycles, of a forward SiLU 2450 -> 2330.
__device__ __forceinline__ float sigmoidf_fast(float x) {
  const float y = fmaf(0.25f, exp_flush(-x), 0.25f);
  float r;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(y));
  return 0.25f * fmaf(r, fmaf(-fminf(y, 1.0e38f), r, 1.0f), r);
}
__device__ __forceinline__ float silu_f(float x) { return x * sigmoidf_fast(x); }
__device__ __forceinline__ float gelu_f(float x) { return 0.5f * x * (1.0f + erff(x * 0.70710678118654752f)); }
// tanh form: 0.5 x (1 + tanh(sqrt(2/pi) (x + 0.044715 x^3)))
__device__ __forceinline__ float gelu_tanh_f(float x) {
  const float u = 0.7978845608028654f * (x + 0.044715f * x * x * x);
  return 0.5f * x * (1.0f + tanhf(u));
}
__device__ __forceinline__ float dgelu_tanh_f(float x) {
  const float u = 0.7978845608028654f * (x + 0.044715f * x * x * x);
  const float t = tanhf(u);
  const float du = 0.7978845608028654f * (1.0f + 3.0f * 0.044715f * x * x);
  return 0.5f * (1.0f + t) + 0.5f * x * (1.0f - t * t) * du;
}
__device__ __forceinline__ float dsilu_f(float x) {
  float s = sigmoidf_fast(x);
  return s * (1.0f + x * (1.0f - s));
}
__device__ __forceinline__ float dgelu_f(float x) {
  float cdf = 0.5f * (1.0f + erff(x * 0.70710678118654752f));
  float pdf = 0.3989422804014327f * __expf(-0.5f * x * x);
  return cdf + x * pdf;
}

}  // namespace moe
