// The grouped-GEMM kernel of the MoE expert path on B200 tensor cores, and its launcher.
//
// One persistent, warp-specialised kernel template covers every contraction of the layer:
//
//   M-grouped (ragged rows, one weight matrix per expert), padded expert-sorted layout:
//     gate/up  : H = Xs @ W1[e]            A K-major, B MN-major ([E,K,N], N contiguous)
//     down     : Y = Act @ W2[e]           A K-major, B MN-major
//     dAct     : dA = Gs @ W2[e]^T         A K-major, B K-major  ([E,N,K], K contiguous)
//     dX       : dXs = dH @ W1[e]^T        A K-major, B K-major
//   K-grouped (contraction over an expert's rows, one output matrix per expert):
//     dW1[e] = Xs_e^T @ dH_e, dW2[e] = Act_e^T @ Gs_e      A and B both MN-major
//
// Roles inside a CTA (320 threads, one CTA per SM):
//   warp 0      : TMA producer  -- cp.async.bulk.tensor tile loads into a ring of shared-memory
//                 stages (128-byte swizzle), signalled by mbarriers.  In the GATHER variants of the
//                 template (a row map `a_row_src` is given) the A rows are GATHERED by the loads themselves:
//                 the 32 lanes issue one tile::gather4 copy each (4 rows x 128 bytes), so the token rows of
//                 an expert never have to be copied into the expert-sorted layout first.  A compile-time
//                 variant because this loop has no slack for branches it does not take;
//   warp 1      : MMA issuer    -- tcgen05.mma (128 x BN x 16 per CTA, fp32 accumulators in TMEM,
//                 two accumulator stages) and tcgen05.commit;
//                 both warps walk their loops with all 32 lanes (uniform control flow) and let one
//                 ELECTED lane issue; each probes the next stage's barrier one stage ahead.  (Issuing
//                 from a single lane inside a divergent branch cost ~100 cycles per tcgen05 instruction
//                 and left the tensor pipe idle 15 % of the time.)
//   warps 2..9  : epilogue      -- tcgen05.ld the accumulator (each warp its 32-lane quadrant and
//                 half of the columns), apply the fused epilogue and store through a swizzled
//                 shared-memory tile per warp, so that every global store covers whole row segments,
//                 locally or into another GPU's buffer.  The dGLU epilogue moves its rows with TMA:
//                 the saved product arrives by cp.async.bulk.tensor loads into the warp's staging tile
//                 (one chunk ahead) and the result leaves by a bulk tensor store from the same tile.
// The accumulator of tile i+1 is produced while tile i is being drained.
//
// CTA pairs (template parameter CTAS = 2, launched as clusters of two): the two CTAs of a pair work
// on two row tiles of the same expert against the same weight tile.  Each CTA loads its own 128 A
// rows and HALF of the B columns; one tcgen05.mma.cta_group::2 issued by the pair's leader spans
// both SMs (256 x BN accumulator, 128 rows in each CTA's TMEM) and reads the B halves from both
// CTAs' shared memory.  That halves the B bytes each SM pulls from L2 and reads from shared memory
// per FLOP.  Every CTA fetches its own tiles with its own loads; nothing is broadcast.  Operand
// arrival is credited to the leader's mbarriers, stage release and accumulator-ready signals go to
// both CTAs (one tcgen05.commit whose arrival is broadcast to the pair), accumulator-drained arrivals
// come back to the leader.
//
// Replaces the Triton kernels m_grouped_gemm_persistent_kernel / m_grouped_gemm_inner_kernel
// (reference: src/moe_explore/triton_kernels/m_grouped_gemm.py:33-267) and their epilogues
// (epilogue_split.py:4-44, triton_kernels/activation.py:5-45).
#pragma once

#include "common.cuh"

#include <atomic>

namespace moe {

constexpr int BM = 128;       // accumulator rows per CTA (= TMEM lanes)
constexpr int BK = 64;        // K extent of one shared-memory stage: 64 x 2 bytes = one 128-byte swizzle row
constexpr int UMMA_K = 16;    // K extent of one tcgen05.mma for 16-bit inputs
constexpr int kEpilogueWarps = 8;
constexpr int kThreads = 64 + 32 * kEpilogueWarps;
constexpr int kWaveLead = 8;   // stages before the end of an item at which a worker announces the next wave
constexpr int kDefaultGroupM = 12;  // consecutive row units that share a sweep over column tiles (L2 reuse)
constexpr uint32_t kTmemCols = 512;
constexpr long long kWaveWaitLimitCycles = 1ll << 21;  // ~1 ms: the wave barrier is an optimisation, not a dependency

// EPI_ACT_AUX is EPI_ACT plus either a second output (aux_out: the un-activated product, saved for backward)
// or a second input (aux_in: the saved product; the accumulator is multiplied by the activation's derivative
// there).  A separate instantiation, so that the plain-store kernels of the hot path carry none of it.
enum Epilogue : int { EPI_ACT = 0, EPI_GLU = 1, EPI_DGLU = 2, EPI_ACT_AUX = 3 };

struct GemmArgs {
  // scheduling
  const int32_t* mtile_expert;  // M-grouped: expert of each 128-row tile
  const int32_t* tile_pairs;    // M-grouped, CTA pairs: first tile | expert << 20 | (pair has a second tile) << 31
  const int32_t* pair_prefix;   // M-grouped: exclusive prefix of the per-expert pair counts [E+1]
  const int32_t* num_mtiles;    // M-grouped: device int32[4] = {tiles in use, tile pairs in use, tile bound, 0}
  const int32_t* pad_offsets;   // K-grouped, and with group_indices: padded row offsets [E+1]
  // Optional prefix of the routed rows per expert [E+1].  With it, only the 64-row blocks of an expert's padded range that
  // hold a routed row exist: M-grouped kernels store nothing into the others, K-grouped kernels contract over the others' rows not
  // at all.
  const int32_t* group_indices;
  int32_t settled;              // transposed tiles: RowCounts::settled
  int32_t short_steps;          // K-grouped: the last step may be 16 or 32 deep (ShortSteps)
  int32_t a_compact;            // M-grouped, with group_indices: A holds the routed rows without padding, expert by expert
  int32_t mtiles_bound;         // M-grouped: padded_rows / 128 as the caller sees it (checked against num_mtiles[2])
  int32_t num_experts;
  int32_t m_dim;  // K-grouped: rows of each output matrix
  int32_t n_dim;  // accumulator columns (N of the contraction)
  int32_t k_dim;  // M-grouped: K of the contraction
  // MN-major operands whose contiguous extent is a multiple of 64 are described to the copy engine as
  // [blocks of 64][rows][64]: ONE copy per stage then fetches all the 64-element-wide column blocks of the tile
  // (one instruction instead of two to four; the blocks land exactly where separate copies put them).
  int32_t a_blocked;  // K-grouped A
  int32_t b_blocked;  // B, when it is MN-major
  // A rows gathered by the loads (null: A is stored in the padded layout).  Padded row p reads row
  // a_row_src[p] / a_div of the A tensor, zeros where a_row_src[p] < 0.  a_rows = rows of the A tensor.
  const int32_t* a_row_src;
  int32_t a_div;
  int32_t a_rows;
  // epilogue
  int32_t out_tma;     // EPI_ACT without a row map: tiles leave through bulk tensor stores (tmap_d covers `out`)
  void* out;           // EPI_ACT: [rows, N]; EPI_GLU: [rows, N/2]; EPI_DGLU: [rows, 2N]
  void* aux_out;       // EPI_GLU, EPI_ACT_AUX: un-activated product [rows, N] or null
  const void* aux_in;  // EPI_DGLU: saved un-activated product [rows, 2N]; EPI_ACT_AUX: the same, [rows, N], or null
  // EPI_ACT (EPI_GLU without push_bases), M-grouped only: when push_row != null, accumulator row p is stored at row push_row[p] (skipped when
  // negative) instead of row p -- of `out`, or, when push_bases != null, of the [*, N] matrix based at
  // push_bases[push_rank[p]] (another GPU's buffer, peer-mapped; rows with push_rank[p] < 0 are not stored).
  void* const* push_bases;
  const int32_t* push_rank;
  const int32_t* push_row;
  // EPI_ACT, M-grouped only: when combine_row_src != null, accumulator row p is multiplied by
  // combine_scores[j] (j = combine_row_src[p], or by 1 when combine_scores is null) and ADDED to row j / combine_topk
  // of `out` with vector reductions; rows with j < 0 are skipped.  `out` must start at zero.
  const int32_t* combine_row_src;
  const void* combine_scores;
  int32_t combine_topk;
  int32_t act;
  int32_t chunk_index;  // M-grouped: process only the experts [E*index/count, E*(index+1)/count) (lets a caller
  int32_t chunk_count;  // pipeline row movement against the GEMM); count <= 1 = everything
  int32_t expert_begin;  // M-grouped: when expert_end > expert_begin, process exactly the experts [begin, end)
  int32_t expert_end;    // instead (slices of unequal size, e.g. chosen by row counts)
  int32_t pair_begin;    // M-grouped: when pair_end > pair_begin, process exactly the row-tile pairs [begin, end) of
  int32_t pair_end;      // the pair list instead (slices that may cut through an expert)
  int32_t align_experts;  // M-grouped CTA pairs: scheduling groups never span two experts
  uint32_t* wave_counter;  // non-null: workers start every work item together (grid-wide arrival counter, zeroed
                           // by the host before the launch)
  int32_t wave_workers;    // arrivals per wave the barrier waits for (the number of workers of the launch)
  // Non-null: work items after a worker's first are claimed from this word (0 before the launch and again after it), see
  // ItemQueue.  CTA pairs of the K-grouped and of the transposed kernels.
  uint32_t* work_counter;
  int32_t group_m;  // row units per scheduling group
  long long wait_limit;  // cycles after which a device-side wait gives up
  int32_t* status;
};

struct TileCoord {
  int m0;       // first accumulator row of THIS CTA: padded row (M-grouped) or output-matrix row (K-grouped)
  int n0;       // first accumulator column of the tile
  int expert;
  int k_row0;   // K-grouped: first padded row of the contraction
  int kiters;   // number of BK-deep stages to contract
  int k_last;   // K-grouped: depth of the last of them (16, 32 or BK)
  bool active;  // false for the second CTA of a pair whose expert has an odd number of row tiles
  int a_row;    // M-grouped: row of A the tile begins at (m0, or its unpadded counterpart; the rows after the expert's last
                // one are then the next expert's, and nothing is stored for them)
  int live;     // M-grouped: rows of the tile that exist (64 or 128, see GemmArgs::group_indices)
  int unit_rows;  // M-grouped: rows of the whole row unit that exist, in 64-row blocks (the tile's, or the pair's)
  bool valid;     // false: there is no further item
};

// A word of the row maps and counts (mtile_expert, tile_pairs, num_mtiles, pad_offsets, group_indices).  From the device's point
// of coherence and not from L1: with RowCounts::settled they are read before this kernel's wait for the one before, which is what
// would make an earlier kernel's writes visible to loads that may hit a line of L1.
__device__ __forceinline__ int32_t map_word(const int32_t* p) {
  int32_t v;
  asm volatile("ld.relaxed.gpu.global.s32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
  return v;
}

// K-grouped: rows of expert e to contract over, in steps of 16 (what follows an expert's last row up to the end of its 64-row
// block is zero), at most its padded range.
__device__ __forceinline__ int contracted_rows(const GemmArgs& args, int e, int padded) {
  if (args.group_indices == nullptr) return padded;
  const int rows = (map_word(args.group_indices + e + 1) - map_word(args.group_indices + e) + 15) & ~15;
  return rows < padded ? (rows > 0 ? rows : 0) : padded;
}

// Rows of expert e that exist, in whole 64-row blocks, at most its padded range (whatever the prefix says).
__device__ __forceinline__ int live_rows(const GemmArgs& args, int e, int padded) {
  if (args.group_indices == nullptr) return padded;
  const int rows = (map_word(args.group_indices + e + 1) - map_word(args.group_indices + e) + 63) & ~63;
  return rows < padded ? (rows > 0 ? rows : 0) : padded;
}

// ----------------------------------------------------------------------------------
// Shared-memory matrix descriptors (64-bit) for tcgen05.mma.
//   bits  0-13  start address >> 4
//   bits 16-29  leading-dimension byte offset >> 4
//   bits 32-45  stride-dimension byte offset >> 4
//   bits 46-47  descriptor version (1 on sm_100)
//   bits 61-63  swizzle mode (2 = 128-byte)
// K-major operand tile as TMA writes it with a {64 x rows} box: row r sits at r*128 bytes, 16-byte
// chunks XOR-swizzled by (r % 8); 8-row groups are 1024 bytes apart (stride offset); the
// leading offset is unused for swizzled K-major layouts.
// MN-major operand tile: each TMA box is {64 MN-elements x BK k-rows}: k-row at k*128 bytes;
// 8-k-row groups are 1024 bytes apart (stride offset); the next 64 MN-elements live in the
// next box, BK*128 bytes further (leading offset).
// ----------------------------------------------------------------------------------
__device__ __forceinline__ uint64_t make_desc(uint32_t smem_addr, uint32_t lbo_bytes, uint32_t sbo_bytes) {
  uint64_t d = 0;
  d |= static_cast<uint64_t>((smem_addr & 0x3FFFFu) >> 4);
  d |= static_cast<uint64_t>((lbo_bytes >> 4) & 0x3FFFu) << 16;
  d |= static_cast<uint64_t>((sbo_bytes >> 4) & 0x3FFFu) << 32;
  d |= 1ull << 46;
  d |= 2ull << 61;
  return d;
}

// Instruction descriptor (32-bit): fp32 accumulate, 16-bit A/B format, operand majorness, N>>3, M>>4.
// With a CTA pair the instruction covers M = 256 rows (128 per CTA).
template <typename T, int BN, bool A_K, bool B_K, int CTAS>
__device__ __forceinline__ constexpr uint32_t make_idesc() {
  uint32_t d = 0;
  d |= 1u << 4;                       // D format: F32
  d |= Elem<T>::kUmmaFormat << 7;     // A format
  d |= Elem<T>::kUmmaFormat << 10;    // B format
  d |= (A_K ? 0u : 1u) << 15;         // A major: 0 = K, 1 = MN
  d |= (B_K ? 0u : 1u) << 16;         // B major
  d |= static_cast<uint32_t>(BN >> 3) << 17;
  d |= static_cast<uint32_t>((BM * CTAS) >> 4) << 24;
  return d;
}

// Shared-memory plan: [operand stages][epilogue staging][barriers].  The staging area holds, per epilogue warp,
// swizzled 32-row x 128-byte tiles: one for the plain-store and GLU epilogues, two for the dGLU and the ungated AUX
// epilogues (the saved product of the next chunk lands in one while the other is computed on and stored from; or the
// un-activated and the activated product are stored side by side), which costs those kernels one operand stage.
// One-CTA kernels have 48 KB stages and stream weights past few rows, so what they keep in flight is their speed: the dGLU
// epilogue takes one staging tile there (its copies in and out then alternate, hidden by the next item) and keeps a
// fourth stage: 1001 tokens x 8 slots, 64 experts, K 2048 95 -> 90 us, 64 tokens on 8 wide experts 224 -> 211.  (A second
// tile and three stages for their weight-gradient kernels: 113 -> 122 us at two steps per item, 0.6 % of a pass at one; not
// taken.)
template <int BN, int CTAS, int EPI>
struct SmemPlan {
  static constexpr int kABytes = BM * BK * 2;
  static constexpr int kBCols = BN / CTAS;        // B columns held by one CTA
  static constexpr int kBBytes = kBCols * BK * 2;
  static constexpr int kStageBytes = kABytes + kBBytes;
  static constexpr int kStagingTile = 32 * 128;
  static constexpr int kTilesPerWarp = ((EPI == EPI_DGLU && CTAS == 2) || EPI == EPI_ACT_AUX) ? 2 : 1;
  static constexpr int kStagingBytes = kEpilogueWarps * kTilesPerWarp * kStagingTile;
  static constexpr int kBarrierBytes = 1024;
  static constexpr int kBudget = 232448 - 1024 - kBarrierBytes - kStagingBytes;  // 227 KB minus alignment slack
  static constexpr int kStages = (kBudget / kStageBytes) > 8 ? 8 : (kBudget / kStageBytes);
  static constexpr int kTotal = kStages * kStageBytes + kStagingBytes + kBarrierBytes + 1024;
};

// The slice of the work a launch covers.
struct Window {
  int m_begin;  // first row unit (pair or tile) of the window
  int e0, e1;   // experts of the window (M-grouped)
  int p_end;    // CTA pairs: one past the last pair of the window (a window may begin and end inside an expert)
};

// Before the wait for the kernels before: the translations of the index arrays, which the first loads after the wait would miss
// (a prefetch into L2 is no read: what the arrays hold may still be about to change).
__device__ __forceinline__ void prefetch_maps(const GemmArgs& args) {
  const void* p = nullptr;
  if (threadIdx.x == 32) p = args.num_mtiles;
  else if (threadIdx.x == 33) p = args.tile_pairs;
  else if (threadIdx.x == 34) p = args.mtile_expert;
  else if (threadIdx.x == 35) p = args.group_indices;
  else if (threadIdx.x == 36) p = args.pad_offsets;
  if (p != nullptr) asm volatile("prefetch.global.L2 [%0];" ::"l"(p));
}

// Number of (row unit, column tile) work items and the row-unit / column-tile counts.  A row unit is
// one 128-row tile (one CTA) or a pair of them (CTA pair).
template <bool KG, int CTAS>
__device__ __forceinline__ int total_tiles(const GemmArgs& args, int& mt, int& nt, Window& win, int BN) {
  nt = (args.n_dim + BN - 1) / BN;
  win.m_begin = 0;
  win.e0 = 0;
  win.e1 = args.num_experts;
  win.p_end = 0x7FFFFFFF;
  if (KG) {
    mt = (args.m_dim + BM * CTAS - 1) / (BM * CTAS);
    return args.num_experts * mt * nt;
  }
  // (the three words are asked for together: a load that follows another's result waits 0.5 to 1 us more for the first tile)
  const int tiles = map_word(args.num_mtiles), pairs = map_word(args.num_mtiles + 1), bound = map_word(args.num_mtiles + 2);
  mt = CTAS == 2 ? pairs : tiles;
  if (args.pair_prefix != nullptr) {
    if (bound != args.mtiles_bound) {
      // the pair prefix sits at tile_pairs[bound]: metadata built for another bound cannot be walked
      if (threadIdx.x == 0 && args.status != nullptr) atomicCAS(args.status, 0, DS_BAD_LAYOUT);
      mt = 0;
      return 0;
    }
    int p0, p1;
    if (args.pair_end > args.pair_begin) {
      // an explicit range of the pair list; the experts it touches are found by the search in decode_tile
      p0 = args.pair_begin < pairs ? args.pair_begin : pairs;
      p1 = args.pair_end < pairs ? args.pair_end : pairs;
    } else if (args.expert_end <= args.expert_begin && args.chunk_count <= 1) {
      p0 = 0;
      p1 = pairs;
    } else {
      if (args.expert_end > args.expert_begin) {
        win.e0 = args.expert_begin;
        win.e1 = args.expert_end < args.num_experts ? args.expert_end : args.num_experts;
      } else {
        win.e0 = static_cast<int>(static_cast<long long>(args.num_experts) * args.chunk_index / args.chunk_count);
        win.e1 = static_cast<int>(static_cast<long long>(args.num_experts) * (args.chunk_index + 1) / args.chunk_count);
      }
      p0 = map_word(args.pair_prefix + win.e0);
      p1 = map_word(args.pair_prefix + win.e1);
    }
    win.p_end = p1;
    if (CTAS == 2) {
      win.m_begin = p0;
      mt = p1 - p0;
    } else {  // one-CTA kernels: the same window expressed in tiles
      win.m_begin = p0 == 0 ? 0 : p0 < pairs ? (map_word(args.tile_pairs + p0) & 0xFFFFF) : tiles;
      mt = (p1 < pairs ? (map_word(args.tile_pairs + p1) & 0xFFFFF) : tiles) - win.m_begin;
    }
  }
  return mt * nt;
}

// Order of the work items.  CTA pairs (M-grouped): expert by expert; inside an expert its pairs are walked in
// groups of `group_m`, and inside a group every column tile is visited for all pairs of the group before moving
// on.  The CTA pairs running at one time then share ONE expert's weight tiles and a small set of row tiles, which
// keeps both in L2 (groups that straddle experts doubled the weight tiles in flight and cost 1.5x the DRAM reads).
// One-CTA kernels and the K-grouped kernels use the same grouped walk without the expert alignment.
template <bool KG, int CTAS>
__device__ __forceinline__ TileCoord decode_tile(int t, int mt, int nt, const Window& win, const GemmArgs& args, int BN,
                                                 int rank) {
  TileCoord c;
  int expert = 0;
  int span = mt;       // row units the grouped walk below runs over
  int span_begin = win.m_begin;
  if (KG) {
    expert = t / (mt * nt);
    t -= expert * (mt * nt);
  } else if (CTAS == 2 && args.align_experts != 0) {
    // binary search: the expert whose pairs contain work item t
    const int base = win.m_begin;
    int lo = win.e0, hi = win.e1;
    while (hi - lo > 1) {
      const int mid = (lo + hi) >> 1;
      if ((map_word(args.pair_prefix + mid) - base) * nt <= t) lo = mid; else hi = mid;
    }
    span_begin = map_word(args.pair_prefix + lo);
    int span_end = map_word(args.pair_prefix + lo + 1);
    // a window given as a pair range may begin or end inside this expert: walk only its part of the expert
    if (span_begin < base) span_begin = base;
    if (span_end > win.p_end) span_end = win.p_end;
    span = span_end - span_begin;
    t -= (span_begin - base) * nt;
  }
  // split the span into equal groups of at most args.group_m row units
  const int num_groups = (span + args.group_m - 1) / args.group_m;
  const int group_m = num_groups > 0 ? (span + num_groups - 1) / num_groups : 1;
  const int per_group = group_m * nt;
  const int g = t / per_group;
  const int rem = t - g * per_group;
  const int m_first = g * group_m;
  const int gm = min(group_m, span - m_first);
  const int n_idx = rem / gm;
  const int m_idx = span_begin + m_first + (rem - n_idx * gm);
  c.n0 = n_idx * BN;
  c.active = true;
  if (KG) {
    c.m0 = (m_idx * CTAS + rank) * BM;
    c.expert = expert;
    c.k_row0 = map_word(args.pad_offsets + expert);
    const int rows = contracted_rows(args, expert, map_word(args.pad_offsets + expert + 1) - c.k_row0);
    c.kiters = (rows + BK - 1) / BK;
    const int rest = rows & (BK - 1);
    c.k_last = rest == 0 || rest > 32 || args.short_steps == 0 ? BK : rest > 16 ? 32 : 16;
    c.live = BM;
    c.unit_rows = BM;
    c.a_row = 0;
  } else {
    int tile = m_idx;
    c.unit_rows = BM;
    if (CTAS == 2) {
      // one load: first tile (bits 0-19), expert (bits 20-30), "has a second tile" (bit 31)
      const uint32_t info = static_cast<uint32_t>(map_word(args.tile_pairs + m_idx));
      const bool second = (info >> 31) != 0;
      tile = static_cast<int>(info & 0xFFFFFu);
      c.expert = static_cast<int>((info >> 20) & 0x7FFu);
      c.active = rank == 0 || second;
      c.unit_rows = second ? 2 * BM : BM;
      if (rank == 1 && second) tile += 1;  // an inactive second CTA re-reads the first tile and stores nothing
    } else {
      c.expert = map_word(args.mtile_expert + tile);
    }
    c.m0 = tile * BM;
    c.a_row = c.m0;
    c.live = BM;
    if (args.group_indices != nullptr) {
      const int base = map_word(args.pad_offsets + c.expert);
      const int left = live_rows(args, c.expert, 1 << 30) - (c.m0 - base);
      c.live = left < BM ? (left > 64 ? left : 64) : BM;
      if (left < c.unit_rows) c.unit_rows = left > 64 ? left : 64;
      if (args.a_compact) c.a_row = c.m0 - base + map_word(args.group_indices + c.expert);
    }
    c.k_row0 = 0;
    c.kiters = (args.k_dim + BK - 1) / BK;
    c.k_last = BK;
  }
  return c;
}

// The work items of one worker, as a warp walks them: every lane decodes one of the next 32 items, and the warp takes them from
// its lanes in turn.  Decoding is a chain of two dependent loads (the unit, then its expert's row counts), 1000 to 2000 cycles
// under load in an in-order warp; item by item it left the copy engine and the tensor cores without instructions for that
// long per item, whatever was still queued.
template <bool KG, int CTAS>
struct ItemWalk {
  TileCoord mine;
  int first, stride, count, mt, nt, BN, rank;  // of the worker's items, `count` items in the launch
  __device__ __forceinline__ ItemWalk(int unit, int num_units, int ntiles, int mt_, int nt_, int BN_, int rank_)
      : mine{}, first(unit), stride(num_units), count(ntiles), mt(mt_), nt(nt_), BN(BN_), rank(rank_) {}
  // The i-th item; i = 0, 1, 2, ... in this order, by all lanes of the warp.
  __device__ __forceinline__ TileCoord get(int i, const Window& win, const GemmArgs& args) {
    if ((i & 31) == 0) {
      const int t = first + (i + static_cast<int>(threadIdx.x & 31)) * stride;
      // (an item that does not exist is not decoded: when no row tile is in use the maps hold nothing to decode)
      if (t < count) mine = decode_tile<KG, CTAS>(t, mt, nt, win, args, BN, rank);
      __syncwarp();
    }
    const int src = i & 31;
    TileCoord c;
    c.valid = first + i * stride < count;
    c.m0 = __shfl_sync(0xFFFFFFFFu, mine.m0, src);
    c.n0 = __shfl_sync(0xFFFFFFFFu, mine.n0, src);
    c.expert = __shfl_sync(0xFFFFFFFFu, mine.expert, src);
    c.k_row0 = __shfl_sync(0xFFFFFFFFu, mine.k_row0, src);
    c.kiters = KG ? __shfl_sync(0xFFFFFFFFu, mine.kiters, src) : (args.k_dim + BK - 1) / BK;
    c.k_last = KG ? __shfl_sync(0xFFFFFFFFu, mine.k_last, src) : BK;
    c.active = __shfl_sync(0xFFFFFFFFu, mine.active ? 1 : 0, src) != 0;
    c.a_row = __shfl_sync(0xFFFFFFFFu, mine.a_row, src);
    c.live = __shfl_sync(0xFFFFFFFFu, mine.live, src);
    c.unit_rows = __shfl_sync(0xFFFFFFFFu, mine.unit_rows, src);
    return c;
  }
};

// Work items claimed one by one instead of dealt out: with a fixed stride the slowest worker is 5 to 11 % behind the mean where
// rows fall unevenly (simulated with the stage costs measured; claimed 1 to 5 %), and where the items are equal the SMs are not --
// storing weight gradients, some were done after 68 us and others after 100.  The second CTA's idle MMA warp is the scheduler: it
// claims an item with one atomic addition, decodes it and writes it into a ring of five slots in both CTAs' shared memory; the other
// nineteen roles read it there.  A worker's first item is its index; M-grouped workers claim the next one when the leader's producer
// has begun the last one claimed, so that at most one unbegun item is held.  Every worker's claims end with one that
// finds nothing left; the claim that is the last of all puts the word back to zero.
// A role hands a slot back when it asks for the item after it.  Handing back goes to the other CTA, by an arrival that orders nothing
// beyond this CTA, so what keeps the scheduler from rewriting a slot under a load is that the load's value is there: everything the
// role did with the item (its copies, instructions and branches depend on the words it read) was issued before, and a word that
// it does not use may be any.  Handed back right after the load, the arrival overtook it now and then: one item in a million was
// another one.  A release at cluster scope waits for all of the warp's memory traffic instead (weight gradients of 128 tokens
// 95 -> 155 us).
constexpr int kQueueSlots = 5;
constexpr int kQueueBarrierBytes = (16 * kQueueSlots + 8 + 15) / 16 * 16;
struct ItemQueue {
  uint32_t full, empty, taken;  // barriers: [slots] in each CTA; [slots] and one in the second CTA
  uint32_t slots;               // [slots][8] words in each CTA

  __device__ __forceinline__ explicit ItemQueue(uint32_t area)
      : full(area), empty(area + 8 * kQueueSlots), taken(area + 16 * kQueueSlots), slots(area + kQueueBarrierBytes) {}
  __device__ __forceinline__ void init() const {  // by one thread of each CTA
    for (int s = 0; s < kQueueSlots; ++s) {
      mbar_init(full + 8 * s, 1);
      mbar_init(empty + 8 * s, 2 * (1 + kEpilogueWarps) + 1);
    }
    mbar_init(taken, 1);
  }
  // The i-th item, by all lanes of a warp of either CTA that is done with the one before; an item that is not valid where the wait
  // gave up (then the abort flag is set).
  template <bool KG>
  __device__ __forceinline__ TileCoord get(int i, const GemmArgs& args, bool mark_taken, const WaitCtx& w, int code) const {
    const int s = i % kQueueSlots;
    if (i > 0 && (threadIdx.x & 31) == 0) mbar_arrive_cluster(mapa_shared(empty + 8 * ((i - 1) % kQueueSlots), 1));
    TileCoord c{};
    if (!__all_sync(0xFFFFFFFFu, mbar_wait(full + 8 * s, (i / kQueueSlots) & 1, w, code))) return c;
    uint32_t mine;
    asm volatile("ld.shared.b32 %0, [%1];" : "=r"(mine) : "r"(slots + 32 * s + 4 * (threadIdx.x & 7)) : "memory");
    int word[8];
#pragma unroll
    for (int j = 0; j < 8; ++j) word[j] = static_cast<int>(__shfl_sync(0xFFFFFFFFu, mine, j));
    __syncwarp();
    if (!KG && mark_taken && (threadIdx.x & 31) == 0) mbar_arrive_cluster(mapa_shared(taken, 1));
    c.m0 = word[0];
    c.n0 = word[1];
    c.expert = word[2];
    c.k_row0 = KG ? word[3] : 0;
    c.a_row = KG ? 0 : word[3];
    c.kiters = KG ? word[4] : (args.k_dim + BK - 1) / BK;
    c.unit_rows = KG ? BM : word[4];
    c.live = BM;
    c.k_last = KG ? word[5] : BK;
    c.active = true;
    c.valid = word[7] != 0;
    return c;
  }
  // The scheduler, by all lanes of a warp of the second CTA.
  template <bool KG, int CTAS>
  __device__ __forceinline__ void serve(int unit, int num_units, int ntiles, int mt, int nt, int BN, const Window& win, const GemmArgs& args,
                                        const WaitCtx& w) const {
    const int lane = threadIdx.x & 31;
    uint32_t claimed = 0;
    const auto claim = [&]() {
      if (lane == 0) {
        claimed = atomicAdd(args.work_counter, 1u);
        if (claimed == static_cast<uint32_t>(ntiles) - 1) *args.work_counter = 0;
      }
    };
    int t = unit;
    for (int i = 0;; ++i) {
      const int s = i % kQueueSlots;
      if (i > 0) {
        if (!KG) {
          if (i == 1) grid_wait();  // the counter was set to zero by a kernel before this one
          if (!__all_sync(0xFFFFFFFFu, mbar_wait(taken, (i - 1) & 1, w, DS_TIMEOUT_PRODUCER))) return;
          claim();
        }
        const uint32_t n = __shfl_sync(0xFFFFFFFFu, claimed, 0);
        t = n < static_cast<uint32_t>(ntiles) ? num_units + static_cast<int>(n) : ntiles;
      }
      const bool valid = t < ntiles;
      if (KG && valid) claim();  // items are short: the next claim is under way while this one waits for its slot
      TileCoord c{};
      if (valid) c = decode_tile<KG, CTAS>(t, mt, nt, win, args, BN, KG ? lane & 1 : 0);
      if (i >= kQueueSlots &&
          !__all_sync(0xFFFFFFFFu, mbar_wait(empty + 8 * s, (i / kQueueSlots - 1) & 1, w, DS_TIMEOUT_PRODUCER))) return;
      if (lane < 2) {
        const uint32_t to = mapa_shared(slots + 32 * s, static_cast<uint32_t>(lane));
        const uint32_t bar = mapa_shared(full + 8 * s, static_cast<uint32_t>(lane));
        mbar_arrive_expect_tx_cluster(bar, 32);
        st_async_v4(to, c.m0, c.n0, c.expert, KG ? c.k_row0 : c.a_row, bar);
        st_async_v4(to + 16, KG ? c.kiters : c.unit_rows, KG ? c.k_last : 0, 0, valid ? 1 : 0, bar);
      }
      __syncwarp();
      if (!valid) return;
    }
  }
};
constexpr int kQueueOffset = 512;  // of the queue in the barrier area

// Wave barrier of the persistent workers.  With a static stride every worker's i-th work item belongs to the same
// "wave" of neighbouring tiles; workers that share operand tiles only hit in L2 while they stream through them
// together, and they drift apart after a few tiles (measured: DRAM reads of a long-K GEMM equal the algorithmic
// bytes for one wave, 1.4x for two, 3.9x for eight).  The leader's producer thread of every worker therefore
// arrives on a global counter a few stages BEFORE it finishes the items of wave i-1 and waits at the start
// of wave i until all workers have arrived: split like this the wait is short and the operand pipeline does not
// drain, while workers still stay within a few stages of each other.
//
// The barrier is only an optimisation, and it presumes that all workers are resident at the same time, which
// nothing guarantees when another kernel holds SMs.  So the wait is short (~1 ms) and a worker whose wait runs
// out does NOT abort: it records DS_WAVE_FALLBACK, stops waiting for the rest of the launch (it keeps arriving,
// so that the others are not held up by it) and carries on with the static stride.  Returns false on that.
__device__ __forceinline__ bool wave_wait(uint32_t* counter, uint32_t target, const WaitCtx& w) {
  const long long t0 = clock64();
  // a quarter of the general limit at most: the other roles of the CTA wait (bounded by the general limit) for
  // what this producer will load only after it has given up here
  const long long limit = (w.limit >> 2) < kWaveWaitLimitCycles ? (w.limit >> 2) : kWaveWaitLimitCycles;
  int spins = 0;
  while (true) {
    uint32_t seen;
    asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(seen) : "l"(counter) : "memory");
    if (seen >= target) return true;
    if (((++spins) & 15) == 0) {
      if (*w.abort_flag) return false;
      if (clock64() - t0 > limit) {
        if (w.status != nullptr) atomicCAS(w.status, 0, DS_WAVE_FALLBACK);
        return false;
      }
    }
    __nanosleep(64);
  }
}

// 8 consecutive output elements (16 bytes) from 8 fp32 values.
template <typename T>
__device__ __forceinline__ uint4 pack8(const float* v) {
  uint4 r;
  r.x = Elem<T>::pack2(v[0], v[1]);
  r.y = Elem<T>::pack2(v[2], v[3]);
  r.z = Elem<T>::pack2(v[4], v[5]);
  r.w = Elem<T>::pack2(v[6], v[7]);
  return r;
}

// Element-wise activation of a register row, and its derivative as a factor.  The choice is made once per row: inside the
// element loop its branches kept the elements from being interleaved.
__device__ __forceinline__ void apply_act(float (&v)[32], int act) {
  if (act == MOE_ACT_SILU) {
#pragma unroll
    for (int i = 0; i < 32; ++i) v[i] = silu_f(v[i]);
  } else if (act == MOE_ACT_GELU) {
#pragma unroll
    for (int i = 0; i < 32; ++i) v[i] = gelu_f(v[i]);
  } else if (act != MOE_ACT_NONE) {
#pragma unroll
    for (int i = 0; i < 32; ++i) v[i] = gelu_tanh_f(v[i]);
  }
}
__device__ __forceinline__ void mul_dact(float (&v)[32], const float (&x)[32], int act) {
  if (act == MOE_ACT_SILU) {
#pragma unroll
    for (int i = 0; i < 32; ++i) v[i] *= dsilu_f(x[i]);
  } else if (act == MOE_ACT_GELU) {
#pragma unroll
    for (int i = 0; i < 32; ++i) v[i] *= dgelu_f(x[i]);
  } else {
#pragma unroll
    for (int i = 0; i < 32; ++i) v[i] *= dgelu_tanh_f(x[i]);
  }
}
template <typename T>
__device__ __forceinline__ void mul_dact(float (&v)[32], const uint4 (&pre)[4], int act) {
  float x[32];
#pragma unroll
  for (int qq = 0; qq < 4; ++qq) {
    const uint32_t w[4] = {pre[qq].x, pre[qq].y, pre[qq].z, pre[qq].w};
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const float2 f = Elem<T>::unpack2(w[i]);
      x[qq * 8 + 2 * i] = f.x;
      x[qq * 8 + 2 * i + 1] = f.y;
    }
  }
  mul_dact(v, x, act);
}

// Gated backward of one register row: da = gradient of the activated value, h = the saved (gate, up) pairs, replaced by
// (d_gate, d_up).
template <typename T, bool GEGLU>
__device__ __forceinline__ void dglu_row(const float (&da)[32], uint4 (&h)[8]) {
#pragma unroll
  for (int qq = 0; qq < 8; ++qq) {  // 8 elements = 4 (gate, up) pairs per 16 bytes
    const uint32_t hw[4] = {h[qq].x, h[qq].y, h[qq].z, h[qq].w};
    float o[8];
#pragma unroll
    for (int p = 0; p < 4; ++p) {
      const float2 gu = Elem<T>::unpack2(hw[p]);
      float act_g, dact_g;
      if (GEGLU) {
        act_g = gelu_f(gu.x);
        dact_g = dgelu_f(gu.x);
      } else {
        const float sg = sigmoidf_fast(gu.x);
        act_g = gu.x * sg;
        dact_g = sg * (1.0f + gu.x * (1.0f - sg));
      }
      o[2 * p] = da[qq * 4 + p] * gu.y * dact_g;
      o[2 * p + 1] = da[qq * 4 + p] * act_g;
    }
    h[qq] = pack8<T>(o);
  }
}

// Source rows of four consecutive padded rows, as the gather4 copy wants them: row_src / div, or `oob` (a row
// index outside the tensor, which the copy fills with zeros) for padding rows.
__device__ __forceinline__ int4 gather_rows4(const int32_t* row_src, int first, int div, int oob) {
  const int4 j = *reinterpret_cast<const int4*>(row_src + first);
  int4 r;
  r.x = j.x < 0 ? oob : j.x / div;
  r.y = j.y < 0 ? oob : j.y / div;
  r.z = j.z < 0 ? oob : j.z / div;
  r.w = j.w < 0 ? oob : j.w / div;
  return r;
}

// K-grouped: the operands again, in boxes of 16 and 32 contracted rows, for the last step of an expert with few rows left.  With 16
// rows per expert three quarters of what a 64-row step loads are zeros, and these kernels then move little else than their
// result (weight1 gradient of 64 experts x 2048 x 2048, 128 tokens x 8: 114.6 -> 106 us; 64 x 7168 x 4096: 872 -> 802).
struct ShortSteps {
  CUtensorMap a[2], b[2];
};
struct NoShortSteps {};
template <bool KG> struct ShortStepsOf { typedef NoShortSteps type; };
template <> struct ShortStepsOf<true> { typedef ShortSteps type; };

// tmap_a / tmap_b: the operands.  tmap_c / tmap_d (EPI_DGLU): the saved product and the output, both
// [rows, 2N] with a {64 columns, 32 rows} box; EPI_ACT_AUX: the un-activated product (saved or read) and the output, both
// [rows, N], same box.  tmap_d (EPI_ACT with out_tma): the output, [rows, N] or
// [E, M, N], same box.
template <typename T, int BN, bool A_K, bool B_K, int EPI, bool KG, int CTAS, bool GATHER>
__global__ void __launch_bounds__(kThreads, 1)
grouped_gemm_kernel(const __grid_constant__ CUtensorMap tmap_a, const __grid_constant__ CUtensorMap tmap_b,
                    const __grid_constant__ CUtensorMap tmap_c, const __grid_constant__ CUtensorMap tmap_d,
                    const GemmArgs args, const __grid_constant__ typename ShortStepsOf<KG>::type short_steps) {
  using Plan = SmemPlan<BN, CTAS, EPI>;
  constexpr int kStages = Plan::kStages;
  constexpr bool kPair = CTAS == 2;
  extern __shared__ uint8_t smem_raw[];
  const uint32_t raw_addr = smem_u32(smem_raw);
  const uint32_t tiles_addr = (raw_addr + 1023u) & ~1023u;  // 128-byte swizzle atoms need 1024-byte alignment
  uint8_t* tiles = smem_raw + (tiles_addr - raw_addr);
  const uint32_t staging_addr = tiles_addr + kStages * Plan::kStageBytes;  // 1024-byte aligned as well
  uint64_t* bars = reinterpret_cast<uint64_t*>(tiles + kStages * Plan::kStageBytes + Plan::kStagingBytes);
  const uint32_t full_bar = smem_u32(bars);                     // [kStages]  (used in the leader CTA)
  const uint32_t empty_bar = smem_u32(bars + kStages);          // [kStages]  (one set per CTA)
  const uint32_t tfull_bar = smem_u32(bars + 2 * kStages);      // [2]        (one set per CTA)
  const uint32_t tempty_bar = smem_u32(bars + 2 * kStages + 2); // [2]        (used in the leader CTA)
  const uint32_t epi_bar = smem_u32(bars + 2 * kStages + 4);    // [kEpilogueWarps][2]  (dGLU side-input tiles)
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 2 * kStages + 4 + 2 * kEpilogueWarps);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);
  static_assert((2 * 8 + 4 + 2 * kEpilogueWarps) * 8 + 8 <= kQueueOffset && kQueueOffset + kQueueBarrierBytes + kQueueSlots * 32 <= Plan::kBarrierBytes,
                "barrier area too small");
  // items claimed at run time (K-grouped pairs): a compile-time possibility, the other kernels' loops carry none of it
  constexpr bool kQueue = KG && kPair && !GATHER;
  const ItemQueue queue(smem_u32(bars) + kQueueOffset);
  const bool queued = kQueue && args.work_counter != nullptr;

  const int warp = threadIdx.x >> 5;
  const int lane = threadIdx.x & 31;
  const int rank = kPair ? static_cast<int>(cluster_ctarank()) : 0;  // 0 = leader of the pair
  const int unit = blockIdx.x / CTAS;        // persistent worker index (CTA or CTA pair)
  const int num_units = gridDim.x / CTAS;

  WaitCtx wctx;
  wctx.abort_flag = abort_flag;
  wctx.peer_abort = kPair ? mapa_shared(smem_u32(const_cast<int*>(abort_flag)), static_cast<uint32_t>(rank ^ 1)) : 0u;
  wctx.status = args.status;
  wctx.limit = args.wait_limit;

  if (threadIdx.x == 0) {
    for (int s = 0; s < kStages; ++s) {
      mbar_init(full_bar + 8 * s, CTAS);   // one arrive.expect_tx per CTA
      mbar_init(empty_bar + 8 * s, 1);
    }
    for (int a = 0; a < 2; ++a) {
      mbar_init(tfull_bar + 8 * a, 1);
      mbar_init(tempty_bar + 8 * a, kEpilogueWarps * CTAS);
    }
    for (int i = 0; i < 2 * kEpilogueWarps; ++i) mbar_init(epi_bar + 8 * i, 1);
    if (kQueue) queue.init();
    *abort_flag = 0;
    mbar_fence_init();
    tma_prefetch_desc(&tmap_a);
    tma_prefetch_desc(&tmap_b);
    if (EPI == EPI_DGLU || EPI == EPI_ACT_AUX) tma_prefetch_desc(&tmap_c);
    if (EPI == EPI_DGLU || EPI == EPI_ACT_AUX || (EPI == EPI_ACT && args.out_tma)) tma_prefetch_desc(&tmap_d);
  }
  if (warp == 1) {
    if (kPair) {
      tmem_alloc_pair(smem_u32(tmem_slot), kTmemCols);
      tmem_relinquish_pair();
    } else {
      tmem_alloc(smem_u32(tmem_slot), kTmemCols);
      tmem_relinquish();
    }
  }
  prefetch_maps(args);
  tc_fence_before();
  __syncthreads();
  if (kPair) cluster_sync_all();  // the peer's barriers must be initialised before anything arrives on them
  tc_fence_after();
  grid_wait();  // nothing above reads or writes global memory
  const uint32_t tmem_base = *tmem_slot;

  int mt, nt;
  Window win;
  const int ntiles = total_tiles<KG, CTAS>(args, mt, nt, win, BN);
  ItemWalk<KG, CTAS> walk(unit, num_units, ntiles, mt, nt, BN, rank);
  const auto item = [&](int i, bool mark_taken, int code) {
    if (kQueue && queued) return queue.template get<KG>(i, args, mark_taken, wctx, code);
    return walk.get(i, win, args);
  };

  if (warp == 0) {
    // ------------------------------ TMA producer ------------------------------
    // The whole warp walks the loop (uniform control flow); one elected lane issues the tile copies, and with
    // gathered A rows every lane issues one gather4 copy.
    {
      int stage = 0;
      uint32_t phase = 0;
      bool ok = true;
      bool freed = false;  // the stage about to be filled was already seen free (probed one stage ahead)
      const int bcol = rank * Plan::kBCols;  // this CTA's share of the tile's B columns
      const uint64_t pol = l2_policy_evict_normal();
      // Gathered A rows are a compile-time variant: the mere presence of the gather branches in this loop (taken or
      // not) cost every kernel 15-25 % (measured: gate/up 3.30 -> 3.00 ms, weight1 gradient 3.43 -> 2.75 ms at the
      // Mixtral shape with the branches compiled out), because the loop then no longer is the short elected-lane
      // sequence the operand pipeline needs once per 512 tensor-core cycles.
      constexpr bool gather = GATHER;
      TileCoord c_next = item(0, rank == 0, DS_TIMEOUT_PRODUCER);
      // M-grouped gather: lane l owns rows 4l..4l+3 of the tile for all of its stages
      int4 rows_next = make_int4(0, 0, 0, 0);
      if (gather && !KG && unit < ntiles) rows_next = gather_rows4(args.a_row_src, c_next.m0 + 4 * lane, args.a_div, args.a_rows);
      bool wave_sync = !KG && args.wave_counter != nullptr && rank == 0;
      int wave = 0;
      for (; c_next.valid && ok; ++wave) {
        const TileCoord c = c_next;
        const int4 rows_m = rows_next;
        if (gather) {
          // the next work item's rows: their indices are loaded while this tile streams
          c_next = item(wave + 1, false, DS_TIMEOUT_PRODUCER);
          if (!KG && c_next.valid) rows_next = gather_rows4(args.a_row_src, c_next.m0 + 4 * lane, args.a_div, args.a_rows);
        }
        if (wave_sync && wave > 0 &&
            !__all_sync(0xFFFFFFFFu, wave_wait(args.wave_counter, static_cast<uint32_t>(args.wave_workers) * wave, wctx))) {
          if (*abort_flag) {
            ok = false;
            break;
          }
          wave_sync = false;  // the barrier ran out: static stride from here on (arrivals below continue)
        }
        // this worker's arrival for the NEXT wave goes out kWaveLead stages before this item ends
        const bool arrive_here = !KG && args.wave_counter != nullptr && rank == 0;
        const int arrive_kb = c.kiters > kWaveLead ? c.kiters - kWaveLead : 0;
        // K-grouped gather: lane l owns k-rows 4(l % 16)..+3 of box l / 16; the indices change every stage and are
        // fetched one stage ahead
        int4 rows_k = make_int4(0, 0, 0, 0);
        if (gather && KG && c.kiters > 0) rows_k = gather_rows4(args.a_row_src, c.k_row0 + 4 * (lane & 15), args.a_div, args.a_rows);
        for (int kb = 0; kb < c.kiters; ++kb) {
          if (arrive_here && kb == arrive_kb && lane == 0) atomicAdd(args.wave_counter, 1u);
          int4 rows_k_next = rows_k;
          if (gather && KG && kb + 1 < c.kiters)
            rows_k_next = gather_rows4(args.a_row_src, c.k_row0 + (kb + 1) * BK + 4 * (lane & 15), args.a_div, args.a_rows);
          if (!freed && !__all_sync(0xFFFFFFFFu, mbar_wait(empty_bar + 8 * stage, phase ^ 1, wctx, DS_TIMEOUT_PRODUCER))) {
            ok = false;
            break;
          }
          {
            const int ns = stage + 1 == kStages ? 0 : stage + 1;
            freed = __all_sync(0xFFFFFFFFu, mbar_test_wait(empty_bar + 8 * ns, stage + 1 == kStages ? phase : phase ^ 1));
          }
          const uint32_t sa = tiles_addr + stage * Plan::kStageBytes;
          const uint32_t sb = sa + Plan::kABytes;
          const CUtensorMap* map_a = &tmap_a;
          const CUtensorMap* map_b = &tmap_b;
          uint32_t stage_bytes = Plan::kStageBytes;
          int block = BK * 128;  // bytes of one 64-element-wide block of an MN-major operand
          if constexpr (KG && !GATHER) {
            if (kb + 1 == c.kiters && c.k_last != BK) {
              map_a = &short_steps.a[c.k_last >> 5];
              map_b = &short_steps.b[c.k_last >> 5];
              block = c.k_last * 128;
              stage_bytes = (BM + Plan::kBCols) * 2 * c.k_last;
            }
          }
          // the second CTA of a pair credits the LEADER's barrier: the leader issues the MMA that reads both halves
          const bool remote = kPair && rank != 0;
          const uint32_t fb = remote ? mapa_shared(full_bar + 8 * stage, 0) : full_bar + 8 * stage;
          const bool leader_lane = elect_one();
          if (leader_lane) {
            if (remote) mbar_arrive_expect_tx_cluster(fb, stage_bytes);
            else mbar_arrive_expect_tx(fb, stage_bytes);
          }
          if (gather) {
            // all 32 lanes: 4 rows x 128 bytes each = the whole 128 x 64 (or 64 x 128) A tile of the stage
            if (KG) {
              const uint32_t dst = sa + (lane >> 4) * (BK * 128) + (lane & 15) * 512;
              if (remote) tma_gather4_pair(dst, &tmap_a, c.m0 + 64 * (lane >> 4), rows_k, fb, pol);
              else tma_gather4(dst, &tmap_a, c.m0 + 64 * (lane >> 4), rows_k, fb, pol);
            } else {
              const uint32_t dst = sa + lane * 512;
              if (remote) tma_gather4_pair(dst, &tmap_a, kb * BK, rows_m, fb, pol);
              else tma_gather4(dst, &tmap_a, kb * BK, rows_m, fb, pol);
            }
          }
          if (!leader_lane) {
            // the other lanes only keep step
          } else if (remote) {
            if (KG) {
              const int krow = c.k_row0 + kb * BK;
              if (gather) {
              } else if (args.a_blocked) {
                tma_load_3d_pair(sa, map_a, 0, krow, c.m0 >> 6, fb, pol);
              } else {
#pragma unroll
                for (int j = 0; j < BM / 64; ++j) tma_load_2d_pair(sa + j * block, map_a, c.m0 + 64 * j, krow, fb, pol);
              }
              if (args.b_blocked) {
                tma_load_3d_pair(sb, map_b, 0, krow, (c.n0 + bcol) >> 6, fb, pol);
              } else {
#pragma unroll
                for (int j = 0; j < Plan::kBCols / 64; ++j)
                  tma_load_2d_pair(sb + j * block, map_b, c.n0 + bcol + 64 * j, krow, fb, pol);
              }
            } else {
              if (!gather) tma_load_2d_pair(sa, &tmap_a, kb * BK, c.a_row, fb, pol);
              if (B_K) {
                tma_load_3d_pair(sb, &tmap_b, kb * BK, c.n0 + bcol, c.expert, fb, pol);
              } else if (args.b_blocked) {
                tma_load_4d_pair(sb, &tmap_b, 0, kb * BK, (c.n0 + bcol) >> 6, c.expert, fb, pol);
              } else {
#pragma unroll
                for (int j = 0; j < Plan::kBCols / 64; ++j)
                  tma_load_3d_pair(sb + j * (BK * 128), &tmap_b, c.n0 + bcol + 64 * j, kb * BK, c.expert, fb, pol);
              }
            }
          } else {
            // single CTA, or the leader of a pair: everything is local
            if (KG) {
              const int krow = c.k_row0 + kb * BK;
              if (gather) {
              } else if (args.a_blocked) {
                tma_load_3d(sa, map_a, 0, krow, c.m0 >> 6, fb, pol);
              } else {
#pragma unroll
                for (int j = 0; j < BM / 64; ++j) tma_load_2d(sa + j * block, map_a, c.m0 + 64 * j, krow, fb, pol);
              }
              if (args.b_blocked) {
                tma_load_3d(sb, map_b, 0, krow, (c.n0 + bcol) >> 6, fb, pol);
              } else {
#pragma unroll
                for (int j = 0; j < Plan::kBCols / 64; ++j)
                  tma_load_2d(sb + j * block, map_b, c.n0 + bcol + 64 * j, krow, fb, pol);
              }
            } else {
              if (!gather) tma_load_2d(sa, &tmap_a, kb * BK, c.a_row, fb, pol);
              if (B_K) {
                tma_load_3d(sb, &tmap_b, kb * BK, c.n0 + bcol, c.expert, fb, pol);
              } else if (args.b_blocked) {
                tma_load_4d(sb, &tmap_b, 0, kb * BK, (c.n0 + bcol) >> 6, c.expert, fb, pol);
              } else {
#pragma unroll
                for (int j = 0; j < Plan::kBCols / 64; ++j)
                  tma_load_3d(sb + j * (BK * 128), &tmap_b, c.n0 + bcol + 64 * j, kb * BK, c.expert, fb, pol);
              }
            }
          }
          __syncwarp();
          rows_k = rows_k_next;
          if (++stage == kStages) { stage = 0; phase ^= 1; }
        }
        if (!gather) c_next = item(wave + 1, rank == 0, DS_TIMEOUT_PRODUCER);
      }
      // all operand loads are issued: the next chained kernel may come up beside the last tile's contraction and epilogue (from
      // the start of this kernel on, its waiting CTAs cost more than they hid)
      grid_release();
      if (!KG && args.wave_counter != nullptr && rank == 0 && lane == 0) {
        // workers without an item in the remaining waves still count, so that the others do not wait for them
        // (arrivals for waves up to `wave` were made inside the items that preceded them)
        const int waves = (ntiles + num_units - 1) / num_units;
        for (int w = wave + 1; w < waves; ++w) atomicAdd(args.wave_counter, 1u);
      }
      if (!ok || *abort_flag) {
        // Let copies that were already issued land before the CTA releases its shared memory.
        for (int i = 0; i < 2000; ++i) __nanosleep(1000);
      }
    }
  } else if (warp == 1) {
    // ------------------------------ MMA issuer (leader CTA only) --------------
    // The whole warp walks the tile / stage loop (uniform control flow and operands); one elected lane issues
    // the tensor-core instructions.
    if (rank == 0) {
      constexpr uint32_t idesc = make_idesc<T, BN, A_K, B_K, CTAS>();
      int stage = 0;
      uint32_t phase = 0;
      int acc = 0;
      uint32_t acc_phase = 0;
      bool ok = true;
      bool ready = false;  // the stage about to be consumed was already seen full
      for (int i = 0; ok; ++i) {
        const TileCoord c = item(i, false, DS_TIMEOUT_MMA);
        if (!c.valid) break;
        if (c.kiters == 0) continue;  // empty expert: the epilogue writes zeros on its own
        if (!__all_sync(0xFFFFFFFFu, mbar_wait(tempty_bar + 8 * acc, acc_phase ^ 1, wctx, DS_TIMEOUT_MMA))) {
          ok = false;
          break;
        }
        tc_fence_after();
        const uint32_t d_tmem = tmem_base + acc * BN;
        for (int kb = 0; kb < c.kiters; ++kb) {
          // `ready` was probed one stage ahead (below), so that the barrier's round trip to shared memory
          // overlaps the issue of the previous stage's MMAs; only a stage that was not there yet is waited for.
          if (!ready && !__all_sync(0xFFFFFFFFu, mbar_wait(full_bar + 8 * stage, phase, wctx, DS_TIMEOUT_MMA))) {
            ok = false;
            break;
          }
          tc_fence_after();
          {
            const int ns = stage + 1 == kStages ? 0 : stage + 1;
            ready = __all_sync(0xFFFFFFFFu, mbar_test_wait(full_bar + 8 * ns, stage + 1 == kStages ? phase ^ 1 : phase));
          }
          const uint32_t sa = tiles_addr + stage * Plan::kStageBytes;
          const uint32_t sb = sa + Plan::kABytes;
          const int depth = KG && !GATHER && kb + 1 == c.kiters ? c.k_last : BK;
          const uint32_t block = KG ? depth * 128 : BK * 128;  // see the producer
          if (elect_one()) {
#pragma unroll
            for (int k = 0; k < BK / UMMA_K; ++k) {
              if (KG && k * UMMA_K >= depth) break;
              // K-major: step 16 elements (32 bytes) along the swizzled 128-byte row.
              // MN-major: step 16 k-rows of 128 bytes.
              const uint64_t da = A_K ? make_desc(sa + k * (UMMA_K * 2), 16, 1024)
                                      : make_desc(sa + k * (UMMA_K * 128), block, 1024);
              const uint64_t db = B_K ? make_desc(sb + k * (UMMA_K * 2), 16, 1024)
                                      : make_desc(sb + k * (UMMA_K * 128), block, 1024);
              if (kPair) umma_f16_pair(d_tmem, da, db, idesc, (kb | k) != 0 ? 1u : 0u);
              else umma_f16(d_tmem, da, db, idesc, (kb | k) != 0 ? 1u : 0u);
            }
            // free the stage in every CTA whose shared memory these MMAs read (one broadcast arrival)
            if (kPair) umma_commit_pair_both(empty_bar + 8 * stage);
            else umma_commit(empty_bar + 8 * stage);
          }
          __syncwarp();
          if (++stage == kStages) { stage = 0; phase ^= 1; }
        }
        if (!ok) break;
        // accumulator complete: tell the epilogue warps of every CTA holding a part of it
        if (elect_one()) {
          if (kPair) umma_commit_pair_both(tfull_bar + 8 * acc);
          else umma_commit(tfull_bar + 8 * acc);
        }
        __syncwarp();
        if (++acc == 2) { acc = 0; acc_phase ^= 1; }
      }
      if (!ok || *abort_flag) {
        for (int i = 0; i < 2000; ++i) __nanosleep(1000);
      }
    } else if (kQueue && queued) {
      queue.template serve<KG, CTAS>(unit, num_units, ntiles, mt, nt, BN, win, args, wctx);
    }
  } else {
    // ------------------------------ epilogue ----------------------------------
    // Warp w reads TMEM lane quadrant (w % 4); the two warps of a quadrant split the columns.
    const int quad = warp & 3;
    const int half = (warp - 2) >> 2;
    constexpr int kChunksPerWarp = BN / 32 / 2;
    const int chunk_begin = half * kChunksPerWarp;
    const int row_in_tile = quad * 32 + lane;
    int acc = 0;
    uint32_t acc_phase = 0;
    T* out = reinterpret_cast<T*>(args.out);
    T* aux_out = reinterpret_cast<T*>(args.aux_out);
    const int N = args.n_dim;
    const uint32_t tempty_leader = kPair ? mapa_shared(tempty_bar, 0) : tempty_bar;
    // this warp's staging tile(s): 32 rows x 128 bytes, 16-byte pieces XOR-swizzled by (row % 8), i.e. the layout
    // the 128-byte-swizzle tensor copies read and write
    const uint32_t stage_base = staging_addr + (warp - 2) * (Plan::kTilesPerWarp * Plan::kStagingTile);
    const uint32_t my_epi_bar = epi_bar + (warp - 2) * 16;
    // running count of side-input tiles this warp has received; two staging tiles are used in turn
    uint32_t q = 0;
    const auto side_buf = [](uint32_t n) { return Plan::kTilesPerWarp == 2 ? (n & 1) : 0u; };
    const auto side_parity = [](uint32_t n) { return Plan::kTilesPerWarp == 2 ? (n >> 1) & 1 : n & 1; };
    const int co_row = lane >> 3;  // coalesced access: row within a group of four
    const int co_ck = lane & 7;    // and 16-byte piece of the row's 128 bytes
    for (int i = 0;; ++i) {
      const TileCoord c = item(i, false, DS_TIMEOUT_EPILOGUE);
      if (!c.valid) break;
      const bool have_acc = c.kiters != 0;
      const int row = c.m0 + row_in_tile;
      const bool quad_live = KG || (c.active && quad * 32 < c.live);  // this warp's 32 rows exist
      bool row_ok = quad_live;
      long long out_row;  // row index into the output matrix
      T* row_out = out;  // base of the matrix this lane's row is stored into
      float row_scale = 1.0f;
      if (KG) {
        row_ok = row_ok && row < args.m_dim;
        out_row = static_cast<long long>(c.expert) * args.m_dim + row;
      } else {
        out_row = row;
        if ((EPI == EPI_ACT || EPI == EPI_GLU) && args.push_row != nullptr) {
          int32_t r = -1;
          if (row_ok) {
            if (args.push_bases != nullptr) {
              const int32_t rk = args.push_rank[row];
              if (rk >= 0) {
                row_out = reinterpret_cast<T*>(args.push_bases[rk]);
                r = args.push_row[row];
              }
            } else {
              r = args.push_row[row];
            }
          }
          row_ok = r >= 0;
          if (row_ok) out_row = r;
        } else if (EPI == EPI_ACT && args.combine_row_src != nullptr) {
          const int32_t j = row_ok ? args.combine_row_src[row] : -1;
          row_ok = j >= 0;
          if (row_ok) {
            out_row = j / args.combine_topk;
            if (args.combine_scores != nullptr) row_scale = Elem<T>::to_float(reinterpret_cast<const T*>(args.combine_scores)[j]);
          }
        }
      }
      const long long warp_row0 = static_cast<long long>(c.m0) + quad * 32;
      const bool side_input = EPI == EPI_DGLU || (EPI == EPI_ACT_AUX && args.aux_in != nullptr);
      if (side_input) {
        // The saved product does not depend on the accumulator: request the first chunk's tile before waiting
        // for the MMAs.  The buffer it lands in was last read by the store issued two chunks ago.
        const int col0 = c.n0 + chunk_begin * 32;
        if (quad_live && col0 < N && lane == 0) {
          bulk_wait_read_all();
          const uint32_t bar = my_epi_bar + 8 * side_buf(q);
          mbar_arrive_expect_tx(bar, Plan::kStagingTile);
          tma_load_2d_plain(stage_base + side_buf(q) * Plan::kStagingTile, &tmap_c, EPI == EPI_DGLU ? 2 * col0 : col0,
                            static_cast<int>(warp_row0), bar);
        }
        __syncwarp();
      }
      if (have_acc) {
        if (!__all_sync(0xFFFFFFFFu, mbar_wait(tfull_bar + 8 * acc, acc_phase, wctx, DS_TIMEOUT_EPILOGUE))) break;
        tc_fence_after();
      }
      const uint32_t taddr = tmem_base + (static_cast<uint32_t>(quad * 32) << 16) + acc * BN;
      if (!quad_live) {
        // nothing to store
      } else if (EPI == EPI_ACT) {
        // Plain store (optionally with an activation, optionally into another GPU's buffer, optionally scaled and
        // added into token-order rows): two 32-column chunks at a time go through the swizzled shared-memory tile so
        // that every store instruction of the warp writes four 128-byte row segments instead of 32 scattered
        // 16-byte pieces.
        const unsigned long long my_base = reinterpret_cast<unsigned long long>(row_out + out_row * N);
        const bool accumulate = !KG && args.combine_row_src != nullptr;
        // Without a row map the 32-row x 64-column piece this warp has staged leaves as ONE bulk tensor store (the copy
        // engine clips it at the edges of the matrix) instead of eight 16-byte stores per lane; the staging tile is
        // written again only after that store has read it.
        const bool tma_out = args.out_tma != 0;
        const bool tile_stored = !KG || c.m0 + quad * 32 < args.m_dim;
#pragma unroll 1
        for (int chunk = chunk_begin; chunk < chunk_begin + kChunksPerWarp; chunk += 2) {
#pragma unroll
          for (int hc = 0; hc < 2; ++hc) {
            float v[32];
            if (have_acc) {
              uint32_t raw[32];
              tmem_ld_32x32(taddr + (chunk + hc) * 32, raw);
              tmem_ld_wait();
#pragma unroll
              for (int i = 0; i < 32; ++i) v[i] = __uint_as_float(raw[i]);
            } else {
#pragma unroll
              for (int i = 0; i < 32; ++i) v[i] = 0.0f;
            }
            apply_act(v, args.act);
            if (accumulate) {
#pragma unroll
              for (int i = 0; i < 32; ++i) v[i] *= row_scale;
            }
            if (tma_out && hc == 0) {
              if (lane == 0) bulk_wait_read_all();  // the previous round's store has read the staging tile
              __syncwarp();
            }
#pragma unroll
            for (int qq = 0; qq < 4; ++qq) {
              const uint4 u = pack8<T>(v + qq * 8);
              const uint32_t addr = stage_base + lane * 128 + (((hc * 4 + qq) ^ (lane & 7)) << 4);
              asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(addr), "r"(u.x), "r"(u.y), "r"(u.z), "r"(u.w)
                           : "memory");
            }
          }
          const int col_pair0 = c.n0 + chunk * 32;  // first of the 64 columns staged
          if (tma_out) {
            fence_proxy_async_smem();
            __syncwarp();
            if (lane == 0 && tile_stored && col_pair0 < N) {
              if (KG) tma_store_3d(&tmap_d, col_pair0, c.m0 + quad * 32, c.expert, stage_base);
              else tma_store_2d(&tmap_d, col_pair0, static_cast<int>(warp_row0), stage_base);
              bulk_commit();
            }
            continue;
          }
          __syncwarp();
#pragma unroll
          for (int j = 0; j < 8; ++j) {
            const int r = j * 4 + co_row;  // row of the warp's 32 this lane writes in this step
            const unsigned long long base = __shfl_sync(0xFFFFFFFFu, my_base, r);
            const int ok = __shfl_sync(0xFFFFFFFFu, row_ok ? 1 : 0, r);
            uint4 u;
            const uint32_t addr = stage_base + r * 128 + ((co_ck ^ (r & 7)) << 4);
            asm volatile("ld.shared.v4.b32 {%0, %1, %2, %3}, [%4];" : "=r"(u.x), "=r"(u.y), "=r"(u.z), "=r"(u.w) : "r"(addr));
            const int col = col_pair0 + co_ck * 8;
            if (ok && col < N) {
              if (accumulate) red_add_v8<T>(reinterpret_cast<T*>(base) + col, u);
              else *reinterpret_cast<uint4*>(reinterpret_cast<T*>(base) + col) = u;
            }
          }
          __syncwarp();
        }
      } else if (EPI == EPI_ACT_AUX) {
        // Ungated experts in training, 64 columns per round, moved by tensor copies of the warp's 32-row tiles:
        // with aux_out the un-activated and the activated product leave from one tile each; with aux_in the saved
        // product comes in one round ahead (as in the dGLU epilogue) and the row is replaced in place.  The accumulator is
        // read once.
        bool failed = false;
#pragma unroll 1
        for (int chunk = chunk_begin; chunk < chunk_begin + kChunksPerWarp; chunk += 2) {
          const int col0 = c.n0 + chunk * 32;
          const bool live = col0 < N;  // uniform over the warp
          const uint32_t buf = side_input ? stage_base + (q & 1) * Plan::kStagingTile : stage_base;
          if (side_input) {
            if (live) {
              const int ncol0 = col0 + 64;
              if (chunk + 2 < chunk_begin + kChunksPerWarp && ncol0 < N && lane == 0) {
                bulk_wait_read_all();
                const uint32_t nbar = my_epi_bar + 8 * ((q + 1) & 1);
                mbar_arrive_expect_tx(nbar, Plan::kStagingTile);
                tma_load_2d_plain(stage_base + ((q + 1) & 1) * Plan::kStagingTile, &tmap_c, ncol0,
                                  static_cast<int>(warp_row0), nbar);
              }
              __syncwarp();
              if (!__all_sync(0xFFFFFFFFu, mbar_wait(my_epi_bar + 8 * (q & 1), (q >> 1) & 1, wctx, DS_TIMEOUT_EPILOGUE))) {
                failed = true;
                break;
              }
            }
          } else if (lane == 0) {
            bulk_wait_read_all();  // the previous round's stores have read both tiles
          }
          __syncwarp();
#pragma unroll 1
          for (int hc = 0; hc < 2; ++hc) {
            uint32_t raw[32];
            tmem_ld_32x32(taddr + (chunk + hc) * 32, raw);
            tmem_ld_wait();
            float v[32];
#pragma unroll
            for (int i = 0; i < 32; ++i) v[i] = __uint_as_float(raw[i]);
            if (!live) continue;
            const uint32_t row_addr = buf + lane * 128;
            if (side_input) {
              uint4 pre[4];
#pragma unroll
              for (int qq = 0; qq < 4; ++qq)
                asm volatile("ld.shared.v4.b32 {%0, %1, %2, %3}, [%4];"
                             : "=r"(pre[qq].x), "=r"(pre[qq].y), "=r"(pre[qq].z), "=r"(pre[qq].w)
                             : "r"(row_addr + (((hc * 4 + qq) ^ (lane & 7)) << 4)));
              mul_dact<T>(v, pre, args.act);
            } else {
#pragma unroll
              for (int qq = 0; qq < 4; ++qq) {
                const uint4 u = pack8<T>(v + qq * 8);
                asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(row_addr + Plan::kStagingTile +
                                                                             (((hc * 4 + qq) ^ (lane & 7)) << 4)),
                             "r"(u.x), "r"(u.y), "r"(u.z), "r"(u.w)
                             : "memory");
              }
              apply_act(v, args.act);
            }
#pragma unroll
            for (int qq = 0; qq < 4; ++qq) {
              const uint4 u = pack8<T>(v + qq * 8);
              asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(row_addr + (((hc * 4 + qq) ^ (lane & 7)) << 4)),
                           "r"(u.x), "r"(u.y), "r"(u.z), "r"(u.w)
                           : "memory");
            }
          }
          fence_proxy_async_smem();
          __syncwarp();
          if (live) {
            if (lane == 0) {
              tma_store_2d(&tmap_d, col0, static_cast<int>(warp_row0), buf);
              if (!side_input) tma_store_2d(&tmap_c, col0, static_cast<int>(warp_row0), buf + Plan::kStagingTile);
              bulk_commit();
            }
            if (side_input) ++q;
          }
        }
        if (failed) break;
      } else if (EPI == EPI_GLU) {
        // Two 32-column chunks per round.  The un-activated product (128 bytes per row) and the activated
        // half (64 bytes per row) each go through the warp's swizzled shared-memory tile, so that every store
        // instruction writes whole row segments (4 rows x 128 bytes, then 8 rows x 64 bytes) instead of 32
        // scattered 16-byte pieces.
        const int half_n = N >> 1;
        const int glu_row = row_ok ? static_cast<int>(out_row) : -1;
#pragma unroll 1
        for (int chunk = chunk_begin; chunk < chunk_begin + kChunksPerWarp; chunk += 2) {
          uint4 act_pk[4];  // this lane's 32 activated values of the round
          const int col0 = c.n0 + chunk * 32;
#pragma unroll
          for (int hc = 0; hc < 2; ++hc) {
            float v[32];
            if (have_acc) {
              uint32_t raw[32];
              tmem_ld_32x32(taddr + (chunk + hc) * 32, raw);
              tmem_ld_wait();
#pragma unroll
              for (int i = 0; i < 32; ++i) v[i] = __uint_as_float(raw[i]);
            } else {
#pragma unroll
              for (int i = 0; i < 32; ++i) v[i] = 0.0f;
            }
            if (aux_out != nullptr) {
#pragma unroll
              for (int qq = 0; qq < 4; ++qq) {
                const uint4 u = pack8<T>(v + qq * 8);
                const uint32_t addr = stage_base + lane * 128 + (((hc * 4 + qq) ^ (lane & 7)) << 4);
                asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(addr), "r"(u.x), "r"(u.y), "r"(u.z), "r"(u.w)
                             : "memory");
              }
            }
            float g[16];
            if (args.act == MOE_ACT_GEGLU) {
#pragma unroll
              for (int i = 0; i < 16; ++i) g[i] = gelu_f(v[2 * i]) * v[2 * i + 1];
            } else {
#pragma unroll
              for (int i = 0; i < 16; ++i) g[i] = silu_f(v[2 * i]) * v[2 * i + 1];
            }
            act_pk[hc * 2] = pack8<T>(g);
            act_pk[hc * 2 + 1] = pack8<T>(g + 8);
          }
          if (aux_out != nullptr) {
            __syncwarp();
            const bool ok = col0 + co_ck * 8 < N;  // all 32 rows exist (aux_out does not go with a row map)
            T* dst = aux_out + (warp_row0 + co_row) * N + col0 + co_ck * 8;
#pragma unroll
            for (int j = 0; j < 8; ++j) {
              const int r = j * 4 + co_row;
              uint4 u;
              const uint32_t addr = stage_base + r * 128 + ((co_ck ^ (r & 7)) << 4);
              asm volatile("ld.shared.v4.b32 {%0, %1, %2, %3}, [%4];" : "=r"(u.x), "=r"(u.y), "=r"(u.z), "=r"(u.w) : "r"(addr));
              if (ok) *reinterpret_cast<uint4*>(dst + static_cast<long long>(j) * 4 * N) = u;
            }
            __syncwarp();
          }
          // activated half: 4 pieces per row; slot = (piece | odd row << 2) ^ (row >> 1 & 3) keeps both the
          // row-per-lane writes and the 8-rows-per-instruction reads free of bank conflicts
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            const int slot = (i | ((lane & 1) << 2)) ^ ((lane >> 1) & 3);
            const uint32_t addr = stage_base + lane * 128 + (slot << 4);
            asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(addr), "r"(act_pk[i].x), "r"(act_pk[i].y),
                         "r"(act_pk[i].z), "r"(act_pk[i].w)
                         : "memory");
          }
          __syncwarp();
          {
            const int hr = lane >> 2;  // row within a group of eight
            const int hk = lane & 3;   // 16-byte piece of the row's 64 bytes
            const int hcol = (col0 >> 1) + hk * 8;
            const bool ok = hcol < half_n;
#pragma unroll
            for (int j = 0; j < 4; ++j) {
              const int r = j * 8 + hr;
              // row of the output, negative: not stored (each lane holds its own row's; without a row map they are consecutive)
              const int dst_row = __shfl_sync(0xFFFFFFFFu, glu_row, r);
              const int slot = (hk | ((r & 1) << 2)) ^ ((r >> 1) & 3);
              uint4 u;
              const uint32_t addr = stage_base + r * 128 + (slot << 4);
              asm volatile("ld.shared.v4.b32 {%0, %1, %2, %3}, [%4];" : "=r"(u.x), "=r"(u.y), "=r"(u.z), "=r"(u.w) : "r"(addr));
              if (ok && dst_row >= 0) *reinterpret_cast<uint4*>(out + static_cast<long long>(dst_row) * half_n + hcol) = u;
            }
          }
          __syncwarp();
        }
      } else {
        // EPI_DGLU: per 32 accumulator columns, 64 columns (128 bytes per row) of the saved product come in and as
        // many of the result go out, both as tensor copies of this warp's 32 x 128-byte tile; the lanes only read
        // their row from shared memory, do the math on the accumulator and write the row back in place.
        bool failed = false;
#pragma unroll 1
        for (int chunk = chunk_begin; chunk < chunk_begin + kChunksPerWarp; ++chunk) {
          const int col0 = c.n0 + chunk * 32;
          const bool live = col0 < N;  // uniform over the warp
          const uint32_t buf = stage_base + side_buf(q) * Plan::kStagingTile;
          uint4 h_cur[8];
          if (live) {
            const int ncol0 = col0 + 32;
            if (Plan::kTilesPerWarp == 2 && chunk + 1 < chunk_begin + kChunksPerWarp && ncol0 < N && lane == 0) {
              // next chunk's tile into the other buffer, once the store that last read it is done with it
              bulk_wait_read_all();
              const uint32_t nbar = my_epi_bar + 8 * ((q + 1) & 1);
              mbar_arrive_expect_tx(nbar, Plan::kStagingTile);
              tma_load_2d_plain(stage_base + ((q + 1) & 1) * Plan::kStagingTile, &tmap_c, 2 * ncol0,
                                static_cast<int>(warp_row0), nbar);
            }
            __syncwarp();
            if (!__all_sync(0xFFFFFFFFu, mbar_wait(my_epi_bar + 8 * side_buf(q), side_parity(q), wctx, DS_TIMEOUT_EPILOGUE))) {
              failed = true;
              break;
            }
#pragma unroll
            for (int qq = 0; qq < 8; ++qq) {
              const uint32_t addr = buf + lane * 128 + ((qq ^ (lane & 7)) << 4);
              asm volatile("ld.shared.v4.b32 {%0, %1, %2, %3}, [%4];"
                           : "=r"(h_cur[qq].x), "=r"(h_cur[qq].y), "=r"(h_cur[qq].z), "=r"(h_cur[qq].w)
                           : "r"(addr));
            }
          }
          __syncwarp();  // tcgen05.ld is warp-collective
          float v[32];
          if (have_acc) {
            uint32_t raw[32];
            tmem_ld_32x32(taddr + chunk * 32, raw);
            tmem_ld_wait();
#pragma unroll
            for (int i = 0; i < 32; ++i) v[i] = __uint_as_float(raw[i]);
          } else {
#pragma unroll
            for (int i = 0; i < 32; ++i) v[i] = 0.0f;
          }
          if (live) {
            // v = d(activated)[row, col0..col0+32); pre-activation (gate, up) pairs at columns 2*col
            if (args.act == MOE_ACT_GEGLU) dglu_row<T, true>(v, h_cur);
            else dglu_row<T, false>(v, h_cur);
#pragma unroll
            for (int qq = 0; qq < 8; ++qq) {
              const uint32_t addr = buf + lane * 128 + ((qq ^ (lane & 7)) << 4);
              asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(addr), "r"(h_cur[qq].x), "r"(h_cur[qq].y),
                           "r"(h_cur[qq].z), "r"(h_cur[qq].w)
                           : "memory");
            }
            fence_proxy_async_smem();
            __syncwarp();
            if (lane == 0) {
              tma_store_2d(&tmap_d, 2 * col0, static_cast<int>(warp_row0), buf);
              bulk_commit();
              if (Plan::kTilesPerWarp == 1 && chunk + 1 < chunk_begin + kChunksPerWarp && col0 + 32 < N) {
                // the only tile: the next chunk comes in when this one has been read
                bulk_wait_read_all();
                mbar_arrive_expect_tx(my_epi_bar, Plan::kStagingTile);
                tma_load_2d_plain(buf, &tmap_c, 2 * (col0 + 32), static_cast<int>(warp_row0), my_epi_bar);
              }
            }
            ++q;
          }
        }
        if (failed) break;
      }
      if (have_acc) {
        // this warp has read its part of the accumulator: one arrival per warp on the leader's barrier
        tc_fence_before();
        __syncwarp();
        if (lane == 0) {
          if (kPair && rank != 0) mbar_arrive_cluster(tempty_leader + 8 * acc);
          else mbar_arrive(tempty_bar + 8 * acc);
        }
        if (++acc == 2) { acc = 0; acc_phase ^= 1; }
      }
    }
    if ((EPI == EPI_DGLU || EPI == EPI_ACT || EPI == EPI_ACT_AUX) && lane == 0) bulk_wait_all();  // this warp's bulk stores are complete
  }

  tc_fence_before();
  __syncthreads();
  if (kPair) cluster_sync_all();  // neither CTA may exit while its peer can still touch its memory or barriers
  if (warp == 1) {
    __syncwarp();
    tc_fence_after();
    if (kPair) tmem_dealloc_pair(tmem_base, kTmemCols);
    else tmem_dealloc(tmem_base, kTmemCols);
  }
}

// ----------------------------------------------------------------------------------
// launcher (one explicit instantiation per kernel variant, spread over the gemm_inst_*.cu files)
// ----------------------------------------------------------------------------------
struct LaunchParams {
  int max_ctas;  // 0 = one CTA per SM
  bool chained;  // launched with programmatic stream serialization (chained_launches)
  cudaStream_t stream;
};

// Launches one kernel variant with as many persistent workers as fit the current device (capped by lp.max_ctas).
template <typename T, int BN, bool A_K, bool B_K, int EPI, bool KG, int CTAS, bool GATHER>
int launch(const CUtensorMap& ta, const CUtensorMap& tb, const CUtensorMap& tc, const CUtensorMap& td, GemmArgs args,
           const LaunchParams& lp, const typename ShortStepsOf<KG>::type& short_steps = {});

#ifdef MOE_GEMM_DEFINE_LAUNCH
// Launch configuration of a persistent kernel with as many workers as fit the current device (capped by lp.max_ctas), kept per
// device in `grids` (0 = not configured yet; two threads racing at the first launch compute the same value twice).
struct PersistentLaunch {
  cudaLaunchConfig_t cfg = {};
  cudaLaunchAttribute attr[2];
};
template <int CTAS, typename Kernel>
int configure(PersistentLaunch& l, Kernel kernel, int smem, std::atomic<int> (&grids)[64], const LaunchParams& lp) {
  int dev = 0;
  MOE_CUDA(cudaGetDevice(&dev));
  cudaLaunchConfig_t& cfg = l.cfg;
  cfg.blockDim = dim3(kThreads, 1, 1);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = lp.stream;
  l.attr[0].id = cudaLaunchAttributeClusterDimension;
  l.attr[0].val.clusterDim.x = CTAS;
  l.attr[0].val.clusterDim.y = 1;
  l.attr[0].val.clusterDim.z = 1;
  constexpr int kClusterAttrs = CTAS > 1 ? 1 : 0;
  l.attr[kClusterAttrs].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  l.attr[kClusterAttrs].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = l.attr;
  cfg.numAttrs = kClusterAttrs;
  int grid = (dev >= 0 && dev < 64) ? grids[dev].load(std::memory_order_acquire) : 0;
  if (grid == 0) {
    MOE_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
    grid = sm_count() / CTAS * CTAS;
    if (CTAS > 1) {
      // The tile loop is statically strided over the resident workers, so launch exactly as many
      // CTA pairs as can be resident at once (a GPC with an odd SM count cannot host a last pair).
      cfg.gridDim = dim3(static_cast<unsigned>(grid), 1, 1);
      int clusters = 0;
      MOE_CUDA(cudaOccupancyMaxActiveClusters(&clusters, kernel, &cfg));
      if (clusters <= 0) {
        set_error("grouped GEMM: no CTA pair of this kernel fits on the device");
        return MOE_ERR_UNSUPPORTED;
      }
      if (clusters * CTAS < grid) grid = clusters * CTAS;
    }
    if (dev >= 0 && dev < 64) grids[dev].store(grid, std::memory_order_release);
  }
  const int limit = lp.max_ctas / CTAS * CTAS;
  if (limit >= CTAS && limit < grid) grid = limit;
  cfg.gridDim = dim3(static_cast<unsigned>(grid), 1, 1);
  cfg.numAttrs = kClusterAttrs + (lp.chained ? 1 : 0);
  return MOE_OK;
}

template <typename T, int BN, bool A_K, bool B_K, int EPI, bool KG, int CTAS, bool GATHER>
int launch(const CUtensorMap& ta, const CUtensorMap& tb, const CUtensorMap& tc, const CUtensorMap& td, GemmArgs args,
           const LaunchParams& lp, const typename ShortStepsOf<KG>::type& short_steps) {
  auto kernel = grouped_gemm_kernel<T, BN, A_K, B_K, EPI, KG, CTAS, GATHER>;
  constexpr int smem = SmemPlan<BN, CTAS, EPI>::kTotal;
  static_assert(SmemPlan<BN, CTAS, EPI>::kStages >= 3, "too few operand stages");
  static std::atomic<int> grids[64];
  PersistentLaunch l;
  const int rc = configure<CTAS>(l, kernel, smem, grids, lp);
  if (rc != MOE_OK) return rc;
  if (args.wave_workers <= 0) args.wave_workers = static_cast<int>(l.cfg.gridDim.x) / CTAS;
  MOE_CUDA(cudaLaunchKernelEx(&l.cfg, kernel, ta, tb, tc, td, args, short_steps));
  return MOE_OK;
}
#endif  // MOE_GEMM_DEFINE_LAUNCH

}  // namespace moe
