// Host side of the grouped GEMMs: argument checks, tensor maps (cached), scheduling choices and the
// C entry points.  The kernel itself is in gemm_kernel.cuh; its variants are instantiated in gemm_inst_*.cu.
#include "gemm_t_kernel.cuh"

#include <mutex>

namespace moe {

#define MOE_EXTERN(T, CTAS, BN, A_K, B_K, EPI, KG, GATHER)                                                       \
  extern template int launch<T, BN, A_K, B_K, EPI, KG, CTAS, GATHER>(const CUtensorMap&, const CUtensorMap&,       \
                                                                     const CUtensorMap&, const CUtensorMap&, GemmArgs, \
                                                                     const LaunchParams&, const ShortStepsOf<KG>::type&);
// every variant without the row gather; with it, the variants the gathering entry points reach
#define MOE_EXTERN_BN(T, CTAS, BN)                                \
  MOE_EXTERN(T, CTAS, BN, true, false, EPI_ACT, false, false)     \
  MOE_EXTERN(T, CTAS, BN, true, false, EPI_GLU, false, false)     \
  MOE_EXTERN(T, CTAS, BN, true, false, EPI_ACT_AUX, false, false) \
  MOE_EXTERN(T, CTAS, BN, true, true, EPI_ACT, false, false)      \
  MOE_EXTERN(T, CTAS, BN, true, true, EPI_ACT_AUX, false, false)  \
  MOE_EXTERN(T, CTAS, BN, true, true, EPI_DGLU, false, false)     \
  MOE_EXTERN(T, CTAS, BN, false, false, EPI_ACT, true, false)     \
  MOE_EXTERN(T, CTAS, BN, true, false, EPI_ACT, false, true)      \
  MOE_EXTERN(T, CTAS, BN, true, false, EPI_GLU, false, true)      \
  MOE_EXTERN(T, CTAS, BN, true, false, EPI_ACT_AUX, false, true)  \
  MOE_EXTERN(T, CTAS, BN, true, true, EPI_ACT, false, true)       \
  MOE_EXTERN(T, CTAS, BN, false, false, EPI_ACT, true, true)
#define MOE_EXTERN_ALL(T, CTAS) MOE_EXTERN_BN(T, CTAS, 128) MOE_EXTERN_BN(T, CTAS, 256)
MOE_EXTERN_ALL(__nv_bfloat16, 2)
MOE_EXTERN_ALL(__nv_bfloat16, 1)
MOE_EXTERN_ALL(__half, 2)
MOE_EXTERN_ALL(__half, 1)

#define MOE_EXTERN_T(T, UNIT, W_K, EPI) \
  extern template int launch_t<T, UNIT, W_K, EPI>(const TMaps&, const GemmArgs&, const LaunchParams&);
#define MOE_EXTERN_T_ALL(T, UNIT)           \
  MOE_EXTERN_T(T, UNIT, false, EPI_ACT)     \
  MOE_EXTERN_T(T, UNIT, false, EPI_GLU)     \
  MOE_EXTERN_T(T, UNIT, false, EPI_ACT_AUX) \
  MOE_EXTERN_T(T, UNIT, true, EPI_ACT)      \
  MOE_EXTERN_T(T, UNIT, true, EPI_ACT_AUX)  \
  MOE_EXTERN_T(T, UNIT, true, EPI_DGLU)
MOE_EXTERN_T_ALL(__nv_bfloat16, 128)
MOE_EXTERN_T_ALL(__nv_bfloat16, 256)
MOE_EXTERN_T_ALL(__half, 128)
MOE_EXTERN_T_ALL(__half, 256)

typedef CUresult (*EncodeTiledFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                                  const cuuint64_t*, const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave,
                                  CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

static EncodeTiledFn encode_fn() {
  static std::atomic<EncodeTiledFn> cached{nullptr};
  EncodeTiledFn fn = cached.load(std::memory_order_acquire);
  if (fn == nullptr) {
    void* p = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q) == cudaSuccess &&
        q == cudaDriverEntryPointSuccess) {
      fn = reinterpret_cast<EncodeTiledFn>(p);
      cached.store(fn, std::memory_order_release);
    }
  }
  return fn;
}

// Tensor maps depend only on (address, element type, extents, box), never on the data, so they are kept: a training
// step of one layer uses the same 20 to 40 maps again and again, and the host is what small token counts are bound by.  A small
// table with round-robin replacement, shared by all threads.  (Layers that replace each other's maps in it, 16 or 32 of them in
// turn, cost the host no more each than two do.)
struct TmapKey {
  const void* ptr;
  int dtype;
  int rank;
  int swizzle;
  uint64_t dims[4];
  uint64_t strides[3];  // bytes, of dims 1..rank-1
  uint32_t box[4];
  bool operator==(const TmapKey& o) const {
    if (ptr != o.ptr || dtype != o.dtype || rank != o.rank || swizzle != o.swizzle) return false;
    for (int i = 0; i < rank; ++i)
      if (dims[i] != o.dims[i] || box[i] != o.box[i]) return false;
    for (int i = 0; i + 1 < rank; ++i)
      if (strides[i] != o.strides[i]) return false;
    return true;
  }
};
constexpr int kTmapCacheSize = 128;
static std::mutex g_tmap_mutex;
static TmapKey g_tmap_keys[kTmapCacheSize];
static CUtensorMap g_tmap_vals[kTmapCacheSize];
static int g_tmap_used = 0, g_tmap_next = 0;

// Tensor map (by default with the 128-byte swizzle); dims[0] is the contiguous dimension.  `strides` (bytes, for dims 1..rank-1)
// may be null for a dense row-major tensor.
static int make_tmap(CUtensorMap* map, int dtype, const void* ptr, int rank, const uint64_t* dims,
                     const uint32_t* box, const uint64_t* strides = nullptr, bool swizzle = true) {
  TmapKey key{};
  key.ptr = ptr;
  key.dtype = dtype;
  key.rank = rank;
  key.swizzle = swizzle;
  uint64_t dense = 2;
  for (int i = 0; i < rank; ++i) {
    key.dims[i] = dims[i];
    key.box[i] = box[i];
    dense *= dims[i];
    if (i < rank - 1) key.strides[i] = strides != nullptr ? strides[i] : dense;
  }
  {
    std::lock_guard<std::mutex> lock(g_tmap_mutex);
    for (int i = 0; i < g_tmap_used; ++i)
      if (g_tmap_keys[i] == key) {
        *map = g_tmap_vals[i];
        return MOE_OK;
      }
  }
  EncodeTiledFn fn = encode_fn();
  if (fn == nullptr) {
    set_error("cuTensorMapEncodeTiled is not available from the driver");
    return MOE_ERR_CUDA;
  }
  cuuint64_t gdim[4];
  cuuint64_t gstride[3];
  cuuint32_t bdim[4];
  cuuint32_t estr[4] = {1, 1, 1, 1};
  for (int i = 0; i < rank; ++i) {
    gdim[i] = dims[i];
    bdim[i] = box[i];
    if (i < rank - 1) gstride[i] = key.strides[i];
  }
  CUresult r = fn(map, dtype == MOE_DTYPE_BF16 ? CU_TENSOR_MAP_DATA_TYPE_BFLOAT16 : CU_TENSOR_MAP_DATA_TYPE_FLOAT16,
                  rank, const_cast<void*>(ptr), gdim, gstride, bdim, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
                  swizzle ? CU_TENSOR_MAP_SWIZZLE_128B : CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (r != CUDA_SUCCESS) {
    set_error("cuTensorMapEncodeTiled failed with CUresult %d (rank %d, dims %llu x %llu x %llu)", (int)r, rank,
              (unsigned long long)dims[0], (unsigned long long)(rank > 1 ? dims[1] : 1),
              (unsigned long long)(rank > 2 ? dims[2] : 1));
    return MOE_ERR_CUDA;
  }
  {
    std::lock_guard<std::mutex> lock(g_tmap_mutex);
    const int slot = g_tmap_used < kTmapCacheSize ? g_tmap_used++ : (g_tmap_next++ % kTmapCacheSize);
    g_tmap_keys[slot] = key;
    g_tmap_vals[slot] = *map;
  }
  return MOE_OK;
}

// Blocked view of a [rows, cols] (x batch) matrix whose contiguous extent is a multiple of 64 elements:
// dims {64, rows, cols / 64 (, batch)}, so that ONE copy with a {64, box_rows, blocks} box fetches `blocks` adjacent
// 64-column blocks, each landing as a box_rows x 128-byte swizzled tile (the layout of separate 64-wide copies).
static int make_tmap_blocked(CUtensorMap* map, int dtype, const void* ptr, uint64_t rows, uint64_t cols, uint64_t batch,
                             uint32_t box_rows, uint32_t blocks) {
  const uint64_t dims[4] = {64, rows, cols / 64, batch};
  const uint64_t strides[3] = {cols * 2, 128, rows * cols * 2};
  const uint32_t box[4] = {64, box_rows, blocks, 1};
  return make_tmap(map, dtype, ptr, batch > 0 ? 4 : 3, dims, box, strides);
}

static bool aligned16(const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15u) == 0; }

// Arrival counters of the wave barrier for callers that do not bring their own: a small ring in device memory;
// every launch that uses the barrier takes the next slot and zeroes it on its stream first.  A slot that another
// launch re-zeroes under a running kernel only costs that kernel its barrier (it falls back to the static stride).
constexpr int kWaveSlots = 256;
static __device__ uint32_t g_wave_counters[kWaveSlots];

static int ring_wave_counter(uint32_t** out) {
  static std::atomic<uint32_t*> base[64];
  static std::atomic<unsigned> next{0};
  int dev = 0;
  MOE_CUDA(cudaGetDevice(&dev));
  uint32_t* b = (dev >= 0 && dev < 64) ? base[dev].load(std::memory_order_acquire) : nullptr;
  if (b == nullptr) {
    void* p = nullptr;
    MOE_CUDA(cudaGetSymbolAddress(&p, g_wave_counters));
    b = static_cast<uint32_t*>(p);
    if (dev >= 0 && dev < 64) base[dev].store(b, std::memory_order_release);
  }
  *out = b + (next.fetch_add(1, std::memory_order_relaxed) % kWaveSlots);
  return MOE_OK;
}

static moe_gemm_options resolve(const moe_gemm_options* o) {
  moe_gemm_options r{};
  if (o != nullptr) r = *o;
  return r;
}

// 256-column tiles whenever there is more than one 128-column tile of work: with CTA pairs a 256 x 128 x 16 MMA
// takes ~144 cycles against ~158 for 256 x 256 x 16 (its operand reads from shared memory are the limit), so a
// half-empty last 256-column tile is far cheaper than narrow tiles throughout.
static int pick_bn(int N) { return N <= 128 ? 128 : 256; }

// Whether CTA pairs claim their work items (ItemQueue) or have them dealt out: the ring costs 1 to 2 us per launch, so from ten
// items per pair on.  Launches with 4 items per pair 30 -> 32 us and 7 items 86 -> 87, but with 14 items and uneven rows 183 -> 179,
// with 55 equal ones (weight gradients, 128 tokens) 107 -> 95 and 55 -> 51, and the whole 8192-token pass of 64 experts of
// 7168 x 2048 under Zipf routing 19.9 -> 18.9 ms.
static bool worth_claiming(int64_t items) { return items >= 10ll * (sm_count() / 2); }

// What an M-grouped call may add to the plain contraction.
struct MExtras {
  void* aux_out = nullptr;
  const void* aux_in = nullptr;
  void* const* push_bases = nullptr;   // EPI_ACT: rows go to other GPUs' buffers
  const int32_t* push_rank = nullptr;
  const int32_t* push_row = nullptr;
  const int32_t* gather_row_src = nullptr;  // A rows are gathered from a [gather_rows, K] tensor by the loads
  int gather_div = 1;
  int64_t gather_rows = 0;
  const int32_t* combine_row_src = nullptr;  // EPI_ACT: rows are scaled and added into token-order rows
  const void* combine_scores = nullptr;
  int combine_topk = 1;
  int chunk_index = 0;
  int chunk_count = 1;
  RowCounts counts;
};

template <typename T, int BN, int CTAS>
static int mgrouped_dispatch(const void* a, const void* w, int64_t a_rows, int64_t out_rows, int K, int N, int E, int w_transposed, int epi,
                             const GemmArgs& args, int dtype, const LaunchParams& lp) {
  CUtensorMap ta, tb;
  const bool gather = args.a_row_src != nullptr;  // selects the kernel variant whose operand loads gather rows
  {
    const uint64_t dims[2] = {(uint64_t)K, (uint64_t)a_rows};
    const uint32_t box[2] = {BK, args.a_row_src != nullptr ? 1u : (uint32_t)BM};
    int rc = make_tmap(&ta, dtype, a, 2, dims, box);
    if (rc != MOE_OK) return rc;
  }
  if (w_transposed) {
    const uint64_t dims[3] = {(uint64_t)K, (uint64_t)N, (uint64_t)E};
    const uint32_t box[3] = {BK, (uint32_t)(BN / CTAS), 1};
    int rc = make_tmap(&tb, dtype, w, 3, dims, box);
    if (rc != MOE_OK) return rc;
  } else if (args.b_blocked) {
    int rc = make_tmap_blocked(&tb, dtype, w, (uint64_t)K, (uint64_t)N, (uint64_t)E, BK, (uint32_t)(BN / CTAS / 64));
    if (rc != MOE_OK) return rc;
  } else {
    const uint64_t dims[3] = {(uint64_t)N, (uint64_t)K, (uint64_t)E};
    const uint32_t box[3] = {64, BK, 1};
    int rc = make_tmap(&tb, dtype, w, 3, dims, box);
    if (rc != MOE_OK) return rc;
  }
  if (epi == EPI_ACT) {
    CUtensorMap td = ta;
    if (args.out_tma) {
      const uint64_t dims[2] = {(uint64_t)N, (uint64_t)out_rows};
      const uint32_t box[2] = {64, 32};
      int rc = make_tmap(&td, dtype, args.out, 2, dims, box);
      if (rc != MOE_OK) return rc;
    }
    if (gather)
      return w_transposed ? launch<T, BN, true, true, EPI_ACT, false, CTAS, true>(ta, tb, ta, td, args, lp)
                          : launch<T, BN, true, false, EPI_ACT, false, CTAS, true>(ta, tb, ta, td, args, lp);
    return w_transposed ? launch<T, BN, true, true, EPI_ACT, false, CTAS, false>(ta, tb, ta, td, args, lp)
                        : launch<T, BN, true, false, EPI_ACT, false, CTAS, false>(ta, tb, ta, td, args, lp);
  } else if (epi == EPI_GLU) {
    return gather ? launch<T, BN, true, false, EPI_GLU, false, CTAS, true>(ta, tb, ta, ta, args, lp)
                  : launch<T, BN, true, false, EPI_GLU, false, CTAS, false>(ta, tb, ta, ta, args, lp);
  } else if (epi == EPI_ACT_AUX) {
    // the un-activated product (written in the forward pass, read in the backward pass) and the result: tensor copies of
    // 32-row x 64-column boxes
    CUtensorMap tc, td;
    const uint64_t dims[2] = {(uint64_t)N, (uint64_t)(args.mtiles_bound) * BM};
    const uint32_t box[2] = {64, 32};
    int rc = make_tmap(&tc, dtype, args.aux_in != nullptr ? args.aux_in : args.aux_out, 2, dims, box);
    if (rc != MOE_OK) return rc;
    rc = make_tmap(&td, dtype, args.out, 2, dims, box);
    if (rc != MOE_OK) return rc;
    if (gather) return launch<T, BN, true, false, EPI_ACT_AUX, false, CTAS, true>(ta, tb, tc, td, args, lp);  // forward only
    return w_transposed ? launch<T, BN, true, true, EPI_ACT_AUX, false, CTAS, false>(ta, tb, tc, td, args, lp)
                        : launch<T, BN, true, false, EPI_ACT_AUX, false, CTAS, false>(ta, tb, tc, td, args, lp);
  }
  // EPI_DGLU (always with the transposed weight: dAct = g @ W2^T): the saved product and the result are moved by
  // tensor copies of 32-row x 64-column boxes
  CUtensorMap tc, td;
  {
    const uint64_t dims[2] = {(uint64_t)(2 * N), (uint64_t)(args.mtiles_bound) * BM};
    const uint32_t box[2] = {64, 32};
    int rc = make_tmap(&tc, dtype, args.aux_in, 2, dims, box);
    if (rc != MOE_OK) return rc;
    rc = make_tmap(&td, dtype, args.out, 2, dims, box);
    if (rc != MOE_OK) return rc;
  }
  return launch<T, BN, true, true, EPI_DGLU, false, CTAS, false>(ta, tb, tc, td, args, lp);
}

// The same with transposed tiles (gemm_t_kernel.cuh).
template <typename T, int UNIT>
static int mgrouped_dispatch_t(const void* a, const void* w, int64_t a_rows, int64_t out_rows, int K, int N, int E, int w_transposed,
                               int epi, const GemmArgs& args, int dtype, const LaunchParams& lp) {
  TMaps m;
  int rc;
  if (w_transposed) {
    const uint64_t dims[3] = {(uint64_t)K, (uint64_t)N, (uint64_t)E};
    const uint32_t box[3] = {BK, 128, 1};
    rc = make_tmap(&m.w, dtype, w, 3, dims, box);
  } else if (args.b_blocked) {
    rc = make_tmap_blocked(&m.w, dtype, w, (uint64_t)K, (uint64_t)N, (uint64_t)E, BK, 2);
  } else {
    const uint64_t dims[3] = {(uint64_t)N, (uint64_t)K, (uint64_t)E};
    const uint32_t box[3] = {64, BK, 1};
    rc = make_tmap(&m.w, dtype, w, 3, dims, box);
  }
  if (rc != MOE_OK) return rc;
  for (int i = 0; i < 4; ++i) {
    if (i >= UNIT / 64) {
      m.r[i] = m.r[0];
      continue;
    }
    const uint64_t dims[2] = {(uint64_t)K, (uint64_t)a_rows};
    const uint32_t box[2] = {BK, 32u * (i + 1)};
    rc = make_tmap(&m.r[i], dtype, a, 2, dims, box);
    if (rc != MOE_OK) return rc;
  }
  // results and saved products: 32 rows x a warp's 32 weight columns (16 results of gated ones, 32 saved pairs)
  m.c = m.d = m.w;
  const uint64_t cols_d = epi == EPI_GLU ? N / 2 : epi == EPI_DGLU ? 2 * N : N;
  const uint32_t box_d[2] = {epi == EPI_GLU ? 16u : epi == EPI_DGLU ? 64u : 32u, 32};
  if (args.out_tma) {
    const uint64_t dims[2] = {cols_d, (uint64_t)out_rows};
    rc = make_tmap(&m.d, dtype, args.out, 2, dims, box_d, nullptr, epi == EPI_DGLU);
    if (rc != MOE_OK) return rc;
  }
  const void* side = args.aux_in != nullptr ? args.aux_in : args.aux_out;
  if (side != nullptr) {
    const uint64_t dims[2] = {epi == EPI_DGLU ? cols_d : (uint64_t)N, (uint64_t)args.mtiles_bound * BM};
    const uint32_t box[2] = {epi == EPI_DGLU ? 64u : 32u, 32};
    rc = make_tmap(&m.c, dtype, side, 2, dims, box, nullptr, epi == EPI_DGLU);
    if (rc != MOE_OK) return rc;
  }
  if (epi == EPI_ACT) return w_transposed ? launch_t<T, UNIT, true, EPI_ACT>(m, args, lp) : launch_t<T, UNIT, false, EPI_ACT>(m, args, lp);
  if (epi == EPI_GLU) return launch_t<T, UNIT, false, EPI_GLU>(m, args, lp);
  if (epi == EPI_DGLU) return launch_t<T, UNIT, true, EPI_DGLU>(m, args, lp);
  return w_transposed ? launch_t<T, UNIT, true, EPI_ACT_AUX>(m, args, lp) : launch_t<T, UNIT, false, EPI_ACT_AUX>(m, args, lp);
}

static int mgrouped_common(const char* name, const void* a, const void* w, void* out, const MExtras& x,
                           const int32_t* mtile_expert, const int32_t* tile_pairs, const int32_t* num_mtiles,
                           int64_t padded_rows, int K, int N, int E, int w_transposed, int epi, int act, int dtype,
                           const moe_gemm_options* options, int32_t* status, void* stream) {
  MOE_CHECK_ARG(a && w && (out || x.push_bases) && mtile_expert && num_mtiles, "%s: null pointer argument", name);
  MOE_CHECK_ARG(aligned16(a) && aligned16(w) && aligned16(out) && aligned16(x.aux_out) && aligned16(x.aux_in),
                "%s: pointers must be 16-byte aligned", name);
  MOE_CHECK_ARG(padded_rows > 0 && padded_rows % BM == 0, "%s: padded_rows=%lld must be a positive multiple of %d", name,
                (long long)padded_rows, BM);
  MOE_CHECK_ARG(K > 0 && N > 0 && E > 0, "%s: K=%d N=%d E=%d must be positive", name, K, N, E);
  if (K % 8 != 0 || N % 8 != 0 || (epi == EPI_GLU && N % 16 != 0)) {
    set_error("%s: K=%d and N=%d must be multiples of 8 (16 for GLU outputs): rows must be 16-byte aligned", name, K, N);
    return MOE_ERR_UNSUPPORTED;
  }
  MOE_CHECK_ARG(dtype == MOE_DTYPE_BF16 || dtype == MOE_DTYPE_F16, "%s: unknown dtype %d", name, dtype);
  MOE_CHECK_ARG(x.chunk_count <= 1 || (tile_pairs != nullptr && x.chunk_index >= 0 && x.chunk_index < x.chunk_count),
                "%s: chunk %d of %d needs tile_pairs and 0 <= index < count", name, x.chunk_index, x.chunk_count);
  MOE_CHECK_ARG(x.gather_row_src == nullptr || (x.gather_rows > 0 && x.gather_rows < (1ll << 31) && x.gather_div > 0),
                "%s: gathered A needs 0 < rows < 2^31 and div > 0", name);
  MOE_CHECK_ARG(x.combine_row_src == nullptr || x.combine_topk > 0, "%s: topk must be positive", name);
  const moe_gemm_options o = resolve(options);
  GemmArgs args{};
  args.chunk_index = x.chunk_index;
  args.chunk_count = x.chunk_count;
  MOE_CHECK_ARG(o.expert_end <= o.expert_begin || (tile_pairs != nullptr && o.expert_begin >= 0 && o.expert_begin < E),
                "%s: the expert range [%d, %d) needs tile_pairs and 0 <= begin < num_experts", name, o.expert_begin,
                o.expert_end);
  args.expert_begin = o.expert_begin;
  args.expert_end = o.expert_end;
  MOE_CHECK_ARG(o.pair_end <= o.pair_begin || (tile_pairs != nullptr && o.pair_begin >= 0),
                "%s: the pair range [%d, %d) needs tile_pairs and begin >= 0", name, o.pair_begin, o.pair_end);
  args.pair_begin = o.pair_begin;
  args.pair_end = o.pair_end;
  args.mtile_expert = mtile_expert;
  args.tile_pairs = tile_pairs;
  args.mtiles_bound = static_cast<int32_t>(padded_rows / BM);
  args.pair_prefix = tile_pairs != nullptr ? tile_pairs + padded_rows / BM : nullptr;
  {
    // Expert-aligned groups pay off when an expert has enough row-tile pairs to fill a group by itself
    // (measured: -36 % DRAM reads, +4 % speed at 8 pairs per expert; slower at ~4 pairs per expert, where
    // groups spanning several experts keep more CTA pairs on the same row tiles).
    const long long mean_rows = (padded_rows - static_cast<long long>(E) * (BM - 1)) / E;
    args.align_experts = tile_pairs == nullptr ? 0 : (o.align_experts != 0 ? (o.align_experts > 0 ? 1 : 0)
                                                                          : (mean_rows >= 6 * 2 * BM ? 1 : 0));
  }
  args.pad_offsets = x.counts.pad_offsets;
  args.group_indices = x.counts.pad_offsets != nullptr ? x.counts.group_indices : nullptr;
  args.a_compact = x.counts.a_rows >= 0 ? 1 : 0;
  args.num_mtiles = num_mtiles;
  args.num_experts = E;
  args.n_dim = N;
  args.k_dim = K;
  args.a_row_src = x.gather_row_src;
  args.a_div = x.gather_div;
  args.a_rows = static_cast<int32_t>(x.gather_rows);
  args.b_blocked = (!w_transposed && N % 64 == 0 && o.separate_copies == 0) ? 1 : 0;
  // plain stores in the padded layout leave through bulk tensor stores (the copy engine clips the 64-column boxes at N)
  args.out_tma = (epi == EPI_ACT && x.push_row == nullptr && x.combine_row_src == nullptr && out != nullptr &&
                  o.lane_stores == 0) ? 1 : 0;
  args.out = out;
  args.aux_out = x.aux_out;
  args.aux_in = x.aux_in;
  args.push_bases = x.push_bases;
  args.push_rank = x.push_rank;
  args.push_row = x.push_row;
  args.combine_row_src = x.combine_row_src;
  args.combine_scores = x.combine_scores;
  args.combine_topk = x.combine_topk;
  args.act = act;
  args.group_m = o.group_m > 0 ? o.group_m : kDefaultGroupM;
  args.wait_limit = wait_limit_cycles();
  args.status = status;
  LaunchParams lp;
  lp.stream = static_cast<cudaStream_t>(stream);
  lp.max_ctas = o.max_ctas > 0 ? o.max_ctas : 0;
  lp.chained = chained_launches();
  const long long mean_rows_per_expert = (padded_rows - static_cast<long long>(E) * (BM - 1)) / E;
  const int64_t a_rows = x.gather_row_src != nullptr ? x.gather_rows : (x.counts.a_rows >= 0 ? x.counts.a_rows : padded_rows);
  const int64_t out_rows = x.counts.out_rows >= 0 ? x.counts.out_rows : padded_rows;
  // Inside a pass (the routed counts are known): transposed tiles while an expert has few enough rows for its last tile to
  // matter; from six pairs of tiles on (2048 rows of the widest layer: equal within the power-bound spread of 4 %) the
  // expert-aligned, wave-synchronised walk of the other kernel.  Row units of one tile up to 112 rows per expert (160 in the gated
  // backward, whose second staging tile costs the large units a stage), of two from there on: a unit of two tiles shares each
  // weight step among up to 256 rows, one of a single tile keeps eight stages in flight instead of six and wastes less on rare
  // experts.  64 experts, d 2048, I 1024, us, one / two tiles; even, moderately uneven, Zipf routing: forward pass's two
  // contractions, 96 rows 159 / 162, 162 / 173, 177 / 182; 128 rows 178 / 170, 180 / 180, 195 / 189; 192 rows 213 / 188, 213 / 196,
  // 229 / 218; 320 rows 301 / 277, 309 / 268, 320 / 276.  Gated backward, 128 rows 93 / 90, 90 / 85, 89 / 101; 160 rows 90 / 86,
  // 92 / 93, 90 / 91; 224 rows 97 / 94, 102 / 98, 106 / 103.
  // Where units of two tiles would occupy less than half of the pairs, units of one tile again: 8 experts, d 256, I 512, per
  // contraction, 300 rows 16-21 / 18-25, 600 rows 12-20 / 16-26; at three quarters of the pairs either may be ahead (28 / 26 even,
  // 23 / 27 Zipf).
  // One expert has no rare ones and its rows are known exactly: units of two tiles from 129 rows on.  d 7168, I 2048, whole passes out
  // of a graph, one / two where the rule says so, forward and training: 300 rows 53 / 53, 158 / 154; 520 rows 77 / 69, 197 / 198; 768
  // rows 84 / 72, 225 / 213; 1024 rows 92 / 79, 262 / 242; 1500 rows 120 / 118, 345 / 342.  d 4096, I 14336: 200 rows 122 / 106, 359 /
  // 345; 300 rows 134 / 141, 402 / 406; 768 rows 302 / 234, 818 / 668.  d 2048, I 1408: one tile up to 768 rows, 1024 rows 35.6 / 34.4.
  if (x.counts.group_indices != nullptr && tile_pairs != nullptr && x.gather_row_src == nullptr && x.push_bases == nullptr &&
      options == nullptr && mean_rows_per_expert < 6 * 2 * BM) {
    MOE_CHECK_ARG(x.counts.routed_rows >= 0, "%s: the number of routed rows is not set", name);
    args.out_tma = x.push_row == nullptr && x.combine_row_src == nullptr;
    args.settled = x.counts.settled ? 1 : 0;
    // about a unit per expert that has rows, and for every further `unit` rows one; with one expert the rows are known
    const int64_t hit = x.counts.routed_rows < E ? x.counts.routed_rows : E;
    const auto items = [&](int64_t unit) {
      const int64_t units = E == 1 ? (x.counts.routed_rows + unit - 1) / unit : x.counts.routed_rows / unit + hit / 2;
      return (units > hit ? units : hit) * ((N + 255) / 256);
    };
    const int64_t one_tile_rows = epi == EPI_DGLU ? 160 : E == 1 ? BM : 112;
    const int64_t unit =
        (E == 1 ? x.counts.routed_rows : mean_rows_per_expert) > one_tile_rows && items(256) * 4 >= sm_count() ? 256 : 128;
    if (worth_claiming(items(unit))) args.work_counter = x.counts.work_counter;
#define MOE_MG_T(TYPE)                                                                                                 \
  (unit == 256                                                                                                         \
       ? mgrouped_dispatch_t<TYPE, 256>(a, w, a_rows, out_rows, K, N, E, w_transposed, epi, args, dtype, lp)           \
       : mgrouped_dispatch_t<TYPE, 128>(a, w, a_rows, out_rows, K, N, E, w_transposed, epi, args, dtype, lp))
    return dtype == MOE_DTYPE_BF16 ? MOE_MG_T(__nv_bfloat16) : MOE_MG_T(__half);
#undef MOE_MG_T
  }
  {
    // The wave barrier cuts the DRAM reads of every M-grouped GEMM to about the algorithmic bytes (gate/up at
    // the Mixtral shape: 6.4 -> 2.1 GB), but only long contractions get faster (K = 14336: -1.2 %, K = 28672:
    // -2 %); at K = 4096 the synchronised bursts on shared tiles cost more than the re-reads (+6 %).  Hence
    // on for K >= 8192 unless the caller says otherwise.
    const bool on = o.wave_sync != 0 ? o.wave_sync > 0 : K >= 8192;
    args.wave_counter = nullptr;
    args.wave_workers = o.wave_workers > 0 ? o.wave_workers : 0;  // 0: the launcher fills in its worker count
    if (on) {
      args.wave_counter = o.wave_counter;
      if (args.wave_counter == nullptr) {
        const int rc = ring_wave_counter(&args.wave_counter);
        if (rc != MOE_OK) return rc;
      }
      MOE_CUDA(cudaMemsetAsync(args.wave_counter, 0, sizeof(uint32_t), lp.stream));
      lp.chained = false;  // the memset stands between this kernel and the one before
    }
  }
  const int bn = pick_bn(N);
  // CTA pairs, unless the experts average at most one 128-row tile: a pair then has nothing for its second CTA, and
  // a work item streams half as many weight columns per tensor-core cycle as two independent CTAs do (measured at
  // 64 rows per expert, DeepSeek-V3 shape: gate/up 4.10 -> 2.69 ms, down 2.01 -> 1.38; at 16 rows per expert,
  // OLMoE shape: -6..12 %; at 128 rows per expert 0..5 %).
  // (Even routing at 144-192 rows is 6-17 % slower on one CTA: 64 experts, K 2048, 160 rows: 140 / 124 and 85 / 77 us.)  A pass
  // that gathers its rows in the loads stays with one CTA up to 192 where the epilogue moves only the result.
  const bool light = x.counts.group_indices != nullptr && x.gather_row_src != nullptr &&
                     (epi == EPI_ACT || (epi == EPI_GLU && x.aux_out == nullptr));
  const bool pairs = tile_pairs != nullptr &&
                     (o.single_cta == 0 ? mean_rows_per_expert > (light ? BM + BM / 2 : BM) : o.single_cta < 0);
#define MOE_MG(TYPE)                                                                                              \
  (pairs ? (bn == 256 ? mgrouped_dispatch<TYPE, 256, 2>(a, w, a_rows, out_rows, K, N, E, w_transposed, epi, args, dtype, lp) \
                      : mgrouped_dispatch<TYPE, 128, 2>(a, w, a_rows, out_rows, K, N, E, w_transposed, epi, args, dtype, lp)) \
         : (bn == 256 ? mgrouped_dispatch<TYPE, 256, 1>(a, w, a_rows, out_rows, K, N, E, w_transposed, epi, args, dtype, lp) \
                      : mgrouped_dispatch<TYPE, 128, 1>(a, w, a_rows, out_rows, K, N, E, w_transposed, epi, args, dtype, lp)))
  if (dtype == MOE_DTYPE_BF16) return MOE_MG(__nv_bfloat16);
  return MOE_MG(__half);
#undef MOE_MG
}

template <typename T, int BN, int CTAS>
static int kgrouped_dispatch(const void* a, const void* b, int64_t a_rows, int64_t b_rows, int M, int N,
                             const GemmArgs& args, int dtype, const LaunchParams& lp) {
  // operands in boxes of BK contracted rows, and of 16 and 32 for an expert's last step (without routed counts there is none)
  CUtensorMap ta, tb;
  ShortSteps small;
  const auto operand = [&](CUtensorMap* map, const void* p, bool blocked, int64_t rows, int cols, int block_cols, uint32_t depth) {
    if (blocked) return make_tmap_blocked(map, dtype, p, (uint64_t)rows, (uint64_t)cols, 0, depth, (uint32_t)(block_cols / 64));
    const uint64_t dims[2] = {(uint64_t)cols, (uint64_t)rows};
    const uint32_t box[2] = {64, depth};
    return make_tmap(map, dtype, p, 2, dims, box);
  };
  const bool gather = args.a_row_src != nullptr;
  const bool short_steps = args.short_steps != 0;
  int rc = operand(&ta, a, args.a_blocked, a_rows, M, BM, gather ? 1 : BK);
  if (rc == MOE_OK) rc = operand(&tb, b, args.b_blocked, b_rows, N, BN / CTAS, BK);
  for (int i = 0; i < 2 && rc == MOE_OK; ++i) {
    small.a[i] = ta;
    small.b[i] = tb;
    if (!short_steps) continue;
    rc = operand(&small.a[i], a, args.a_blocked, a_rows, M, BM, 16 << i);
    if (rc == MOE_OK) rc = operand(&small.b[i], b, args.b_blocked, b_rows, N, BN / CTAS, 16 << i);
  }
  if (rc != MOE_OK) return rc;
  CUtensorMap td = ta;
  if (args.out_tma) {
    const uint64_t dims[3] = {(uint64_t)N, (uint64_t)M, (uint64_t)args.num_experts};
    const uint32_t box[3] = {64, 32, 1};
    rc = make_tmap(&td, dtype, args.out, 3, dims, box);
    if (rc != MOE_OK) return rc;
  }
  return gather ? launch<T, BN, false, false, EPI_ACT, true, CTAS, true>(ta, tb, ta, td, args, lp, small)
                                   : launch<T, BN, false, false, EPI_ACT, true, CTAS, false>(ta, tb, ta, td, args, lp, small);
}

static int kgrouped_common(const char* name, const void* a, int64_t gather_rows, const int32_t* gather_row_src,
                           int gather_div, const void* b, void* dw, const int32_t* pad_offsets, int64_t padded_rows, int M,
                           int N, int num_experts, int dtype, const moe_gemm_options* options, int32_t* status,
                           void* stream, const RowCounts& counts) {
  MOE_CHECK_ARG(a && b && dw && pad_offsets, "%s: null pointer argument", name);
  MOE_CHECK_ARG(aligned16(a) && aligned16(b) && aligned16(dw), "%s: pointers must be 16-byte aligned", name);
  MOE_CHECK_ARG(padded_rows > 0 && padded_rows % BM == 0, "%s: padded_rows=%lld must be a positive multiple of %d", name,
                (long long)padded_rows, BM);
  MOE_CHECK_ARG(M > 0 && N > 0 && num_experts > 0, "%s: M=%d N=%d E=%d must be positive", name, M, N, num_experts);
  if (M % 8 != 0 || N % 8 != 0) {
    set_error("%s: M=%d and N=%d must be multiples of 8", name, M, N);
    return MOE_ERR_UNSUPPORTED;
  }
  MOE_CHECK_ARG(dtype == MOE_DTYPE_BF16 || dtype == MOE_DTYPE_F16, "%s: unknown dtype %d", name, dtype);
  MOE_CHECK_ARG(gather_row_src == nullptr || (gather_rows > 0 && gather_rows < (1ll << 31) && gather_div > 0),
                "%s: gathered A needs 0 < rows < 2^31 and div > 0", name);
  const moe_gemm_options o = resolve(options);
  GemmArgs args{};
  args.pad_offsets = pad_offsets;
  args.group_indices = counts.group_indices;
  args.num_experts = num_experts;
  args.m_dim = M;
  args.n_dim = N;
  args.a_row_src = gather_row_src;
  args.a_div = gather_div;
  args.a_rows = static_cast<int32_t>(gather_rows);
  args.a_blocked = (gather_row_src == nullptr && M % 64 == 0 && o.separate_copies == 0) ? 1 : 0;
  args.b_blocked = (N % 64 == 0 && o.separate_copies == 0) ? 1 : 0;
  args.out_tma = o.lane_stores == 0 ? 1 : 0;
  args.out = dw;
  args.act = MOE_ACT_NONE;
  args.group_m = o.group_m > 0 ? o.group_m : kDefaultGroupM;
  args.wait_limit = wait_limit_cycles();
  args.status = status;
  LaunchParams lp;
  lp.stream = static_cast<cudaStream_t>(stream);
  lp.max_ctas = o.max_ctas > 0 ? o.max_ctas : 0;
  lp.chained = chained_launches();
  const int bn = pick_bn(N);
  // CTA pairs unless the contraction is at most one 64-row step per expert on average (measured at 64 rows per
  // expert, DeepSeek-V3 shape: weight1 gradient 4.00 -> 3.48 ms; at 128 rows per expert pairs are 9 % faster)
  const long long mean_rows_per_expert = (padded_rows - static_cast<long long>(num_experts) * (BM - 1)) / num_experts;
  // ... unless the pairs claim their work items (at most one step: 106.0 / 105.5 us dealt out, 64 experts x 2048 x 2048)
  const int64_t items = static_cast<int64_t>(num_experts) * ((M + 2 * BM - 1) / (2 * BM)) * ((N + bn - 1) / bn);
  args.work_counter = gather_row_src == nullptr && worth_claiming(items) ? counts.work_counter : nullptr;
  const bool pairs = o.single_cta == 0 ? mean_rows_per_expert > 64 || args.work_counter != nullptr : o.single_cta < 0;
  // (above four steps an eighth of the loads at most is saved, for four more tensor maps per call)
  args.short_steps = counts.group_indices != nullptr && gather_row_src == nullptr && mean_rows_per_expert <= 4 * BK ? 1 : 0;
  const int64_t a_rows = gather_row_src != nullptr ? gather_rows : (counts.a_rows >= 0 ? counts.a_rows : padded_rows);
  const int64_t b_rows = counts.b_rows >= 0 ? counts.b_rows : padded_rows;
#define MOE_KG(TYPE)                                                                                      \
  (pairs ? (bn == 256 ? kgrouped_dispatch<TYPE, 256, 2>(a, b, a_rows, b_rows, M, N, args, dtype, lp)  \
                      : kgrouped_dispatch<TYPE, 128, 2>(a, b, a_rows, b_rows, M, N, args, dtype, lp)) \
         : (bn == 256 ? kgrouped_dispatch<TYPE, 256, 1>(a, b, a_rows, b_rows, M, N, args, dtype, lp)  \
                      : kgrouped_dispatch<TYPE, 128, 1>(a, b, a_rows, b_rows, M, N, args, dtype, lp)))
  if (dtype == MOE_DTYPE_BF16) return MOE_KG(__nv_bfloat16);
  return MOE_KG(__half);
#undef MOE_KG
}

static bool act_is_glu(int act) { return act == MOE_ACT_SWIGLU || act == MOE_ACT_GEGLU; }


int mgrouped_gemm(const void* a, const void* w, void* out, void* pre_act, const int32_t* mtile_expert, const int32_t*
                  tile_pairs, const int32_t* num_mtiles, int64_t padded_rows, int K, int N, int num_experts, int
                  w_transposed, int act, int dtype, int chunk_index, int chunk_count, const moe_gemm_options* options,
                  int32_t* status, void* stream, const RowCounts& counts) {
  MOE_CHECK_ARG(act >= MOE_ACT_NONE && act <= MOE_ACT_GELU_TANH, "moe_mgrouped_gemm: unknown activation %d", act);
  const bool glu = act_is_glu(act);
  MOE_CHECK_ARG(!(glu && w_transposed), "moe_mgrouped_gemm: gated activations need w as [E, K, N]");
  if (!glu && (act == MOE_ACT_NONE || pre_act == nullptr)) pre_act = nullptr;  // nothing to save without an activation
  MExtras x;
  x.counts = counts;
  x.aux_out = pre_act;
  x.chunk_index = chunk_index;
  x.chunk_count = chunk_count;
  const int epi = glu ? EPI_GLU : (pre_act != nullptr ? EPI_ACT_AUX : EPI_ACT);
  return mgrouped_common("moe_mgrouped_gemm", a, w, out, x, mtile_expert, tile_pairs, num_mtiles, padded_rows, K, N,
                         num_experts, w_transposed, epi, act, dtype, options, status, stream);
}

int mgrouped_gemm_gather(const void* src, int64_t src_rows, const int32_t* row_src, int div, const void* w, void* out,
                         void* pre_act, const int32_t* mtile_expert, const int32_t* tile_pairs, const int32_t* num_mtiles,
                         int64_t padded_rows, int K, int N, int num_experts, int act, int dtype, const moe_gemm_options*
                         options, int32_t* status, void* stream, const RowCounts& counts) {
  MOE_CHECK_ARG(act >= MOE_ACT_NONE && act <= MOE_ACT_GELU_TANH, "moe_mgrouped_gemm_gather: unknown activation %d", act);
  MOE_CHECK_ARG(row_src != nullptr, "moe_mgrouped_gemm_gather: row_src is null");
  const bool glu = act_is_glu(act);
  if (!glu && (act == MOE_ACT_NONE || pre_act == nullptr)) pre_act = nullptr;
  MExtras x;
  x.counts = counts;
  x.aux_out = pre_act;
  x.gather_row_src = row_src;
  x.gather_div = div;
  x.gather_rows = src_rows;
  const int epi = glu ? EPI_GLU : (pre_act != nullptr ? EPI_ACT_AUX : EPI_ACT);
  return mgrouped_common("moe_mgrouped_gemm_gather", src, w, out, x, mtile_expert, tile_pairs, num_mtiles, padded_rows, K,
                         N, num_experts, 0, epi, act, dtype, options, status, stream);
}

int mgrouped_gemm_combine(const void* a, const void* w, void* out, const int32_t* row_src, const void* scores, int topk,
                          const int32_t* mtile_expert, const int32_t* tile_pairs, const int32_t* num_mtiles, int64_t
                          padded_rows, int K, int N, int num_experts, int w_transposed, int dtype, const moe_gemm_options*
                          options, int32_t* status, void* stream, const RowCounts& counts) {
  MOE_CHECK_ARG(row_src != nullptr && out != nullptr, "moe_mgrouped_gemm_combine: null pointer argument");
  MExtras x;
  x.counts = counts;
  x.combine_row_src = row_src;
  x.combine_scores = scores;
  x.combine_topk = topk;
  return mgrouped_common("moe_mgrouped_gemm_combine", a, w, out, x, mtile_expert, tile_pairs, num_mtiles, padded_rows, K,
                         N, num_experts, w_transposed, EPI_ACT, MOE_ACT_NONE, dtype, options, status, stream);
}

int mgrouped_gemm_dglu(const void* g, const void* w, const void* pre_act, void* d_pre, const int32_t* mtile_expert, const
                       int32_t* tile_pairs, const int32_t* num_mtiles, int64_t padded_rows, int K, int N, int num_experts,
                       int act, int dtype, int chunk_index, int chunk_count, const moe_gemm_options* options, int32_t*
                       status, void* stream, const RowCounts& counts) {
  MOE_CHECK_ARG(act >= MOE_ACT_SILU && act <= MOE_ACT_GELU_TANH, "moe_mgrouped_gemm_dglu: activation %d has no derivative here",
                act);
  MOE_CHECK_ARG(pre_act != nullptr, "moe_mgrouped_gemm_dglu: pre_act is null");
  MExtras x;
  x.counts = counts;
  x.aux_in = pre_act;
  x.chunk_index = chunk_index;
  x.chunk_count = chunk_count;
  return mgrouped_common("moe_mgrouped_gemm_dglu", g, w, d_pre, x, mtile_expert, tile_pairs, num_mtiles, padded_rows, K, N,
                         num_experts, 1, act_is_glu(act) ? EPI_DGLU : EPI_ACT_AUX, act, dtype, options, status, stream);
}

int kgrouped_gemm(const void* a, const void* b, void* dw, const int32_t* pad_offsets, int64_t padded_rows, int M, int N,
                  int num_experts, int dtype, const moe_gemm_options* options, int32_t* status, void* stream, const
                  RowCounts& counts) {
  return kgrouped_common("moe_kgrouped_gemm", a, 0, nullptr, 1, b, dw, pad_offsets, padded_rows, M, N, num_experts, dtype,
                         options, status, stream, counts);
}

int kgrouped_gemm_gather(const void* src, int64_t src_rows, const int32_t* row_src, int div, const void* b, void* dw,
                         const int32_t* pad_offsets, int64_t padded_rows, int M, int N, int num_experts, int dtype, const
                         moe_gemm_options* options, int32_t* status, void* stream, const RowCounts& counts) {
  MOE_CHECK_ARG(row_src != nullptr, "moe_kgrouped_gemm_gather: row_src is null");
  return kgrouped_common("moe_kgrouped_gemm_gather", src, src_rows, row_src, div, b, dw, pad_offsets, padded_rows, M, N,
                         num_experts, dtype, options, status, stream, counts);
}

int mgrouped_gemm_rows(const void* a, int64_t compact_rows, const void* w, void* out, const int32_t* out_rows,
                       const int32_t* mtile_expert, const int32_t* tile_pairs, const int32_t* num_mtiles, int64_t padded_rows,
                       int K, int N, int num_experts, int act, int dtype, int32_t* status, void* stream,
                       const RowCounts& counts) {
  MExtras x;
  x.counts = counts;
  x.counts.a_rows = compact_rows;
  x.push_row = out_rows;
  return mgrouped_common("moe_rows_gemm", a, w, out, x, mtile_expert, tile_pairs, num_mtiles, padded_rows, K, N, num_experts, 0,
                         act_is_glu(act) ? EPI_GLU : EPI_ACT, act, dtype, nullptr, status, stream);
}

}  // namespace moe

using namespace moe;

extern "C" int moe_mgrouped_gemm(const void* a, const void* w, void* out, void* pre_act, const int32_t* mtile_expert,
                                 const int32_t* tile_pairs, const int32_t* num_mtiles, int64_t padded_rows, int K, int N,
                                 int num_experts, int w_transposed, int act, int dtype, int chunk_index, int chunk_count,
                                 const moe_gemm_options* options, int32_t* status, void* stream) {
  return mgrouped_gemm(a, w, out, pre_act, mtile_expert, tile_pairs, num_mtiles, padded_rows, K, N, num_experts,
                       w_transposed, act, dtype, chunk_index, chunk_count, options, status, stream, RowCounts{});
}

extern "C" int moe_mgrouped_gemm_gather(const void* src, int64_t src_rows, const int32_t* row_src, int div, const void* w,
                                        void* out, void* pre_act, const int32_t* mtile_expert, const int32_t* tile_pairs,
                                        const int32_t* num_mtiles, int64_t padded_rows, int K, int N, int num_experts, int
                                        act, int dtype, const moe_gemm_options* options, int32_t* status, void* stream) {
  return mgrouped_gemm_gather(src, src_rows, row_src, div, w, out, pre_act, mtile_expert, tile_pairs, num_mtiles,
                              padded_rows, K, N, num_experts, act, dtype, options, status, stream, RowCounts{});
}

extern "C" int moe_mgrouped_gemm_combine(const void* a, const void* w, void* out, const int32_t* row_src, const void*
                                         scores, int topk, const int32_t* mtile_expert, const int32_t* tile_pairs, const
                                         int32_t* num_mtiles, int64_t padded_rows, int K, int N, int num_experts, int
                                         w_transposed, int dtype, const moe_gemm_options* options, int32_t* status, void*
                                         stream) {
  return mgrouped_gemm_combine(a, w, out, row_src, scores, topk, mtile_expert, tile_pairs, num_mtiles, padded_rows, K, N,
                               num_experts, w_transposed, dtype, options, status, stream, RowCounts{});
}

extern "C" int moe_mgrouped_gemm_dglu(const void* g, const void* w, const void* pre_act, void* d_pre, const int32_t*
                                      mtile_expert, const int32_t* tile_pairs, const int32_t* num_mtiles, int64_t
                                      padded_rows, int K, int N, int num_experts, int act, int dtype, int chunk_index, int
                                      chunk_count, const moe_gemm_options* options, int32_t* status, void* stream) {
  return mgrouped_gemm_dglu(g, w, pre_act, d_pre, mtile_expert, tile_pairs, num_mtiles, padded_rows, K, N, num_experts,
                            act, dtype, chunk_index, chunk_count, options, status, stream, RowCounts{});
}

extern "C" int moe_kgrouped_gemm(const void* a, const void* b, void* dw, const int32_t* pad_offsets, int64_t padded_rows,
                                 int M, int N, int num_experts, int dtype, const moe_gemm_options* options, int32_t*
                                 status, void* stream) {
  return kgrouped_gemm(a, b, dw, pad_offsets, padded_rows, M, N, num_experts, dtype, options, status, stream, RowCounts{});
}

extern "C" int moe_kgrouped_gemm_gather(const void* src, int64_t src_rows, const int32_t* row_src, int div, const void* b,
                                        void* dw, const int32_t* pad_offsets, int64_t padded_rows, int M, int N, int
                                        num_experts, int dtype, const moe_gemm_options* options, int32_t* status, void*
                                        stream) {
  return kgrouped_gemm_gather(src, src_rows, row_src, div, b, dw, pad_offsets, padded_rows, M, N, num_experts, dtype,
                              options, status, stream, RowCounts{});
}

extern "C" int moe_mgrouped_gemm_push(const void* a, const void* w, void* const* peer_bases, const int32_t* dest_rank,
                                      const int32_t* dest_row, const int32_t* mtile_expert, const int32_t* tile_pairs,
                                      const int32_t* num_mtiles, int64_t padded_rows, int K, int N, int num_experts,
                                      int w_transposed, int dtype, int chunk_index, int chunk_count,
                                      const moe_gemm_options* options, int32_t* status, void* stream) {
  MOE_CHECK_ARG(peer_bases && dest_rank && dest_row, "moe_mgrouped_gemm_push: null pointer argument");
  MExtras x;
  x.push_bases = peer_bases;
  x.push_rank = dest_rank;
  x.push_row = dest_row;
  x.chunk_index = chunk_index;
  x.chunk_count = chunk_count;
  return mgrouped_common("moe_mgrouped_gemm_push", a, w, nullptr, x, mtile_expert, tile_pairs, num_mtiles, padded_rows, K,
                         N, num_experts, w_transposed, EPI_ACT, MOE_ACT_NONE, dtype, options, status, stream);
}

extern "C" int moe_mgrouped_gemm_scatter(const void* a, int64_t a_rows, const int32_t* a_row_src, int a_div,
                                         const void* w, void* out, const int32_t* out_rows, const int32_t* mtile_expert,
                                         const int32_t* tile_pairs, const int32_t* num_mtiles, int64_t padded_rows, int K,
                                         int N, int num_experts, int w_transposed, int act, int dtype,
                                         const moe_gemm_options* options, int32_t* status, void* stream) {
  MOE_CHECK_ARG(out != nullptr && out_rows != nullptr, "moe_mgrouped_gemm_scatter: null pointer argument");
  MOE_CHECK_ARG(act == MOE_ACT_NONE || act == MOE_ACT_SILU || act == MOE_ACT_GELU || act == MOE_ACT_GELU_TANH,
                "moe_mgrouped_gemm_scatter: activation %d is not an element-wise one", act);
  MExtras x;
  x.push_row = out_rows;
  if (a_row_src != nullptr) {
    x.gather_row_src = a_row_src;
    x.gather_div = a_div;
    x.gather_rows = a_rows;
  }
  return mgrouped_common("moe_mgrouped_gemm_scatter", a, w, out, x, mtile_expert, tile_pairs, num_mtiles, padded_rows, K,
                         N, num_experts, w_transposed, EPI_ACT, act, dtype, options, status, stream);
}
