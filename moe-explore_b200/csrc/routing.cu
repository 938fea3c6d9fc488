// Routing metadata: per-expert histogram, prefix sums, STABLE permutation by expert and its
// inverse, plus the padded expert-sorted row layout the grouped GEMMs consume.
//
// Replaces get_token_indices (reference: src/moe_explore/expert_permute.py:19-41), which runs
// torch.argsort + torch.histc + torch.cumsum as three or more launches.  Here it is a counting sort (the number of
// distinct keys, E, is small): one launch of one cluster (route_cluster_kernel) up to kClusterRows rows (fewer where the device
// takes only smaller clusters: max_route_cluster), and for
// more rows the chip-wide form:
//   1. chunk_histogram : each warp owns a contiguous chunk of kChunk flat positions and counts
//                        its ids per expert in shared memory (warp-aggregated via match.any);
//   2. scan_chunks     : a CTA per expert turns its column of the [chunks, E] histogram into exclusive
//                        offsets; scan_offsets: one CTA derives the per-expert prefix sums (unpadded and
//                        padded to 128-row tiles) and the tile -> expert map;
//   3. place_rows      : each warp walks its chunk again in order, ranks equal ids with
//                        match.any + popc (which preserves flat-position order) and writes
//                        perm / row_src / dst_row.
// All arithmetic is integer; results are bit-exact with torch.sort(stable=True).
// HBM traffic: 8R bytes read (ids; twice in the chip-wide form) + 8R (perm) + 4R (dst_row) + 4RP (row_src) written.
#include "common.cuh"

#include <atomic>

namespace moe {

constexpr int kChunk = 1024;        // flat positions per warp
constexpr int kWarpsPerBlock = 8;
constexpr int kMaxExperts = 1024;   // scan kernel uses one thread per expert

__host__ __device__ inline int64_t num_chunks(int64_t R) { return (R + kChunk - 1) / kChunk; }

// Peers of this lane holding the same key (full-warp, inactive lanes pass key = -1 - lane so they match nobody).
__device__ __forceinline__ unsigned match_key(int key) { return __match_any_sync(0xFFFFFFFFu, key); }

// Lane `lane` of the warp that owns [begin, begin + kChunk) loads its 32 ids (positions begin + 32*i + lane)
// with independent loads so their latencies overlap.  Positions past R and ids outside [0, E) become
// negative keys that match no other lane.
__device__ __forceinline__ void load_keys(const int64_t* __restrict__ ids, int64_t begin, int64_t R, int E, int lane,
                                          int (&keys)[kChunk / 32], int32_t* status) {
  int64_t raw[kChunk / 32];
#pragma unroll
  for (int i = 0; i < kChunk / 32; ++i) {
    const int64_t j = begin + 32 * i + lane;
    raw[i] = j < R ? ids[j] : -1;
  }
  bool bad = false;
#pragma unroll
  for (int i = 0; i < kChunk / 32; ++i) {
    const int64_t j = begin + 32 * i + lane;
    const bool ok = raw[i] >= 0 && raw[i] < E;
    bad |= (j < R) && !ok;
    keys[i] = ok ? static_cast<int>(raw[i]) : -1 - lane;
  }
  if (bad && status != nullptr) atomicCAS(status, 0, DS_BAD_EXPERT_ID);  // id out of range: dropped from every output
}

__global__ void __launch_bounds__(kWarpsPerBlock * 32)
chunk_histogram_kernel(const int64_t* __restrict__ ids, int64_t R, int E, int32_t* __restrict__ chunk_hist,
                       int32_t* status) {
  extern __shared__ int32_t sh_cnt[];  // [kWarpsPerBlock][E]
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  int32_t* cnt = sh_cnt + warp * E;
  for (int e = lane; e < E; e += 32) cnt[e] = 0;
  __syncwarp();
  const int64_t chunk = static_cast<int64_t>(blockIdx.x) * kWarpsPerBlock + warp;
  const int64_t begin = chunk * kChunk;
  if (begin >= R) return;
  int keys[kChunk / 32];
  load_keys(ids, begin, R, E, lane, keys, status);
#pragma unroll
  for (int i = 0; i < kChunk / 32; ++i) {
    const int key = keys[i];
    const unsigned peers = match_key(key);
    if (key >= 0 && (peers & ((1u << lane) - 1)) == 0) cnt[key] += __popc(peers);  // lowest peer adds for the group
    __syncwarp();
  }
  for (int e = lane; e < E; e += 32) chunk_hist[chunk * E + e] = cnt[e];
}

// Pair entry layout: bits 0-19 first tile, bits 20-30 expert, bit 31 "the pair has a second tile"
// (so one load tells a CTA pair everything about its next work item).  The per-expert exclusive prefix of
// the pair counts follows the pair list in the same buffer, at index `mtiles_bound` ([E+1] entries).
// Tile -> expert map and the pair list for expert e, whose padded rows start at `row_begin` and span
// `padded` rows; its pairs start at index `pair_begin`.
__device__ __forceinline__ void write_tile_maps(int e, int32_t row_begin, int32_t padded, int32_t pair_begin,
                                                int32_t* __restrict__ mtile_expert, int32_t* __restrict__ tile_pairs,
                                                int32_t* __restrict__ pair_prefix) {
  const int first = row_begin / MOE_TILE_M;
  const int last = first + padded / MOE_TILE_M;
  for (int m = first; m < last; ++m) mtile_expert[m] = e;
  if (tile_pairs != nullptr) {
    pair_prefix[e] = pair_begin;  // exclusive prefix of pair counts: expert e's pairs are [prefix[e], prefix[e+1])
    for (int m = first, p = pair_begin; m < last; m += 2, ++p)
      tile_pairs[p] = static_cast<int32_t>(static_cast<uint32_t>(m) | (static_cast<uint32_t>(e) << 20) |
                                           (m + 1 < last ? 0x80000000u : 0u));
  }
}

// One CTA per expert turns its column of the [chunks, E] histogram into exclusive offsets (every
// thread owns a contiguous run of chunks; block-wide scan of the run sums) and leaves the expert's row count in
// group_indices[e + 1] for the single-CTA pass below.
constexpr int kScanThreads = 256;
__global__ void __launch_bounds__(kScanThreads)
scan_chunks_kernel(const int32_t* __restrict__ chunk_hist, int32_t* __restrict__ chunk_off, int64_t nchunks, int E,
                   int32_t* __restrict__ group_indices) {
  __shared__ int32_t warp_sum[kScanThreads / 32];
  const int e = blockIdx.x;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int64_t per = (nchunks + kScanThreads - 1) / kScanThreads;
  const int64_t c0 = tid * per;
  const int64_t c1 = c0 + per < nchunks ? c0 + per : nchunks;
  int32_t mine = 0;
  for (int64_t c = c0; c < c1; ++c) mine += chunk_hist[c * E + e];
  int32_t incl = mine;
#pragma unroll
  for (int off = 1; off < 32; off <<= 1) {
    const int32_t v = __shfl_up_sync(0xFFFFFFFFu, incl, off);
    if (lane >= off) incl += v;
  }
  if (lane == 31) warp_sum[warp] = incl;
  __syncthreads();
  int32_t before = 0, total = 0;
#pragma unroll
  for (int w = 0; w < kScanThreads / 32; ++w) {
    if (w < warp) before += warp_sum[w];
    total += warp_sum[w];
  }
  int32_t run = before + incl - mine;
  for (int64_t c = c0; c < c1; ++c) {
    chunk_off[c * E + e] = run;
    run += chunk_hist[c * E + e];
  }
  if (tid == 0) group_indices[e + 1] = total;
}

// One CTA, one thread per expert (E <= 1024); the per-expert row counts are in group_indices[1..E] (scan_chunks_kernel).
// num_mtiles receives {tiles in use, tile pairs in use, mtiles_bound, 0}; perm entries past the rows that were
// kept (ids out of range are dropped) are set to -1.
__global__ void __launch_bounds__(kMaxExperts)
scan_offsets_kernel(int E, int32_t* __restrict__ group_indices,
                    int32_t* __restrict__ pad_offsets, int32_t* __restrict__ mtile_expert,
                    int32_t* __restrict__ tile_pairs, int32_t* __restrict__ num_mtiles, int mtiles_bound,
                    int64_t* __restrict__ perm, int64_t R) {
  __shared__ int32_t sh_a[kMaxExperts];
  __shared__ int32_t sh_b[kMaxExperts];
  __shared__ int32_t sh_c[kMaxExperts];
  const int e = threadIdx.x;
  const int32_t total = e < E ? group_indices[e + 1] : 0;
  const int32_t padded = (total + MOE_TILE_M - 1) / MOE_TILE_M * MOE_TILE_M;
  const int32_t pairs = (padded / MOE_TILE_M + 1) / 2;  // row tiles of one expert, two at a time
  sh_a[e] = e < E ? total : 0;
  sh_b[e] = e < E ? padded : 0;
  sh_c[e] = e < E ? pairs : 0;
  __syncthreads();
  // Hillis-Steele inclusive scan over experts for the three sequences.
  for (int off = 1; off < kMaxExperts; off <<= 1) {
    int32_t a = 0, b = 0, c = 0;
    if (e >= off) { a = sh_a[e - off]; b = sh_b[e - off]; c = sh_c[e - off]; }
    __syncthreads();
    sh_a[e] += a;
    sh_b[e] += b;
    sh_c[e] += c;
    __syncthreads();
  }
  if (e < E) {
    group_indices[e + 1] = sh_a[e];
    pad_offsets[e + 1] = sh_b[e];
    if (e == 0) { group_indices[0] = 0; pad_offsets[0] = 0; }
    int32_t* pair_prefix = tile_pairs != nullptr ? tile_pairs + mtiles_bound : nullptr;
    if (mtile_expert != nullptr) write_tile_maps(e, sh_b[e] - padded, padded, sh_c[e] - pairs, mtile_expert, tile_pairs, pair_prefix);
    if (num_mtiles != nullptr && e == E - 1) {
      num_mtiles[0] = sh_b[e] / MOE_TILE_M;
      num_mtiles[1] = sh_c[e];
      num_mtiles[2] = mtiles_bound;
      num_mtiles[3] = 0;
      if (pair_prefix != nullptr) pair_prefix[E] = sh_c[e];
    }
  }
  if (perm != nullptr) {
    const int64_t kept = sh_a[E - 1];
    for (int64_t r = kept + threadIdx.x; r < R; r += kMaxExperts) perm[r] = -1;
  }
}

__global__ void __launch_bounds__(kWarpsPerBlock * 32)
place_rows_kernel(const int64_t* __restrict__ ids, int64_t R, int E, const int32_t* __restrict__ chunk_off,
                  const int32_t* __restrict__ group_indices, const int32_t* __restrict__ pad_offsets,
                  int64_t* __restrict__ perm, int32_t* __restrict__ row_src, int32_t* __restrict__ dst_row) {
  extern __shared__ int32_t sh_cnt[];  // [kWarpsPerBlock][E]: rank of the next row of expert e inside the expert
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  int32_t* cnt = sh_cnt + warp * E;
  const int64_t chunk = static_cast<int64_t>(blockIdx.x) * kWarpsPerBlock + warp;
  const int64_t begin = chunk * kChunk;
  if (begin >= R) return;
  for (int e = lane; e < E; e += 32) cnt[e] = chunk_off[chunk * E + e];
  __syncwarp();
  int keys[kChunk / 32];
  load_keys(ids, begin, R, E, lane, keys, nullptr);
#pragma unroll
  for (int i = 0; i < kChunk / 32; ++i) {
    const int key = keys[i];
    const int64_t j = begin + 32 * i + lane;
    const unsigned peers = match_key(key);
    const unsigned before = peers & ((1u << lane) - 1);
    int32_t rank = 0;
    if (key >= 0) rank = cnt[key] + __popc(before);  // lanes are in flat-position order: stable
    __syncwarp();
    if (key >= 0 && before == 0) cnt[key] += __popc(peers);
    __syncwarp();
    if (key >= 0) {
      if (perm != nullptr) perm[group_indices[key] + rank] = j;
      const int32_t p = pad_offsets[key] + rank;
      if (row_src != nullptr) row_src[p] = static_cast<int32_t>(j);
      if (dst_row != nullptr) dst_row[j] = p;
    } else if (j < R && dst_row != nullptr) {
      dst_row[j] = -1;  // id out of range: the row is in no expert's segment; consumers skip negative rows
    }
  }
}

// ----------------------------------------------------------------------------------
// One launch for everything (the usual case): a single cluster of up to 16 CTAs.
//
// The work is latency, not bytes (28 bytes per row): histogram, prefix sums and placement used to be a memset and
// three or four launches, in which one warp walked 1024 positions through 32 dependent match.any / shared-memory
// steps (27-50 us per layer pass at 4 ... 65536 rows).  Here every lane keeps at most kHeld ids and their ranks in
// registers, the per-warp counts are scanned in shared memory, the per-CTA counts cross the cluster through
// distributed shared memory, and the same threads then place their rows: ids are read once, nothing is staged in
// global memory and there is one launch.  B200, E = 64, us per call in a captured graph, before -> now:
// 4 rows 24.0 -> 6.1, 8008 rows 31.9 -> 7.2, 65536 rows 35.2 -> 13.3, 131072 rows 34.4 -> 20.8.  From there on the
// scattered stores of 16 SMs are the limit (the time doubles with the rows) while the chip-wide kernels above stay
// almost flat (524288 rows: 38.8), hence the line at kClusterRows, which is also what kHeld ids per lane hold.
// ----------------------------------------------------------------------------------
constexpr int kRouteThreads = 1024;
constexpr int kRouteWarps = kRouteThreads / 32;
constexpr int kMaxCluster = 16;
constexpr int kHeld = 8;                                                     // ids per lane kept in registers
constexpr int64_t kClusterRows = int64_t(kMaxCluster) * kRouteThreads * kHeld;  // 131072

struct RouteOut {
  int32_t* group_indices;
  int64_t* perm;
  int32_t* pad_offsets;
  int32_t* row_src;
  int32_t* dst_row;
  int32_t* mtile_expert;
  int32_t* tile_pairs;
  int32_t* num_mtiles;
  int32_t mtiles_bound;
  int32_t padded_bound;
};

__device__ __forceinline__ int32_t ld_cluster(const int32_t* p, uint32_t rank) {
  int32_t v;
  asm volatile("ld.shared::cluster.s32 %0, [%1];" : "=r"(v) : "r"(mapa_shared(smem_u32(p), rank)) : "memory");
  return v;
}

__global__ void __launch_bounds__(kRouteThreads)
route_cluster_kernel(const int64_t* __restrict__ ids, int64_t R, int E, int held, RouteOut out, int32_t* status) {
  extern __shared__ int32_t route_smem[];
  int32_t* const warp_cnt = route_smem;                  // [kRouteWarps][E]: counts, then offsets of the warp in the CTA
  int32_t* const cta_cnt = warp_cnt + kRouteWarps * E;   // [E] rows of this CTA (read by the whole cluster)
  int32_t* const sh_group = cta_cnt + E;                 // [E]   first sorted position of this CTA's rows of expert e
  int32_t* const sh_place = sh_group + E;                // [E]   first padded row of this CTA's rows
  int32_t* const sh_pad = sh_place + E;                  // [E+1] padded row offsets
  int32_t* const sh_pair = sh_pad + E + 1;               // [E+1] pair prefix
  int32_t* const sh_end = sh_pair + E + 1;               // [E]   one past the last routed row of expert e (padded rows)
  __shared__ int32_t sums[3][32];
  __shared__ int32_t kept;  // rows with a valid id
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int rank = static_cast<int>(cluster_ctarank());
  const int ctas = gridDim.x;
  grid_release();
  for (int i = tid; i < kRouteWarps * E; i += kRouteThreads) warp_cnt[i] = 0;
  __syncthreads();

  // 1. count, and rank every id inside its warp's run of 32 * held positions (lanes are in position order: stable)
  const int64_t begin = (static_cast<int64_t>(rank) * kRouteWarps + warp) * 32 * held + lane;
  int32_t* const cnt = warp_cnt + warp * E;
  int key[kHeld];
  int32_t pos[kHeld];
  bool bad = false;
#pragma unroll
  for (int g = 0; g < kHeld; ++g) {
    const int64_t j = begin + 32 * g;
    const bool in = g < held && j < R;
    const int64_t raw = in ? ids[j] : -1;
    const bool ok = raw >= 0 && raw < E;
    bad |= in && !ok;
    key[g] = ok ? static_cast<int>(raw) : -1 - lane;
  }
#pragma unroll
  for (int g = 0; g < kHeld; ++g) {
    pos[g] = 0;
    if (g >= held) break;
    const unsigned peers = match_key(key[g]);
    const unsigned before = peers & ((1u << lane) - 1);
    if (key[g] >= 0) pos[g] = cnt[key[g]] + __popc(before);
    __syncwarp();
    if (key[g] >= 0 && before == 0) cnt[key[g]] += __popc(peers);
    __syncwarp();
  }
  if (bad && status != nullptr) atomicCAS(status, 0, DS_BAD_EXPERT_ID);
  __syncthreads();

  // 2. offsets of the warps inside the CTA (one thread per expert), then of the CTAs inside the cluster
  const int e = tid;
  if (e < E) {
    int32_t run = 0;
#pragma unroll 8
    for (int w = 0; w < kRouteWarps; ++w) {
      const int32_t c = warp_cnt[w * E + e];
      warp_cnt[w * E + e] = run;
      run += c;
    }
    cta_cnt[e] = run;
  }
  __syncwarp();  // the cluster barriers below are .aligned: every warp reaches them as a whole
  cluster_sync_all();
  int32_t total = 0, before = 0;
  if (e < E) {
    for (int c = 0; c < ctas; ++c) {
      const int32_t v = ld_cluster(cta_cnt + e, static_cast<uint32_t>(c));
      before += c < rank ? v : 0;
      total += v;
    }
  }
  // no CTA may exit while another still reads its counts: arrive here, wait at the end
  __syncwarp();
  asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");

  // 3. prefix sums over the experts (every CTA for itself): rows, padded rows, row-tile pairs
  const int32_t padded = (total + MOE_TILE_M - 1) / MOE_TILE_M * MOE_TILE_M;
  const int32_t pairs = (padded / MOE_TILE_M + 1) / 2;
  int32_t in_g = total, in_p = padded, in_q = pairs;
#pragma unroll
  for (int off = 1; off < 32; off <<= 1) {
    const int32_t a = __shfl_up_sync(0xFFFFFFFFu, in_g, off);
    const int32_t b = __shfl_up_sync(0xFFFFFFFFu, in_p, off);
    const int32_t c = __shfl_up_sync(0xFFFFFFFFu, in_q, off);
    if (lane >= off) { in_g += a; in_p += b; in_q += c; }
  }
  if (lane == 31) { sums[0][warp] = in_g; sums[1][warp] = in_p; sums[2][warp] = in_q; }
  __syncthreads();
  if (warp < 3) {
    int32_t v = sums[warp][lane];
    const int32_t own = v;
#pragma unroll
    for (int off = 1; off < 32; off <<= 1) {
      const int32_t a = __shfl_up_sync(0xFFFFFFFFu, v, off);
      if (lane >= off) v += a;
    }
    sums[warp][lane] = v - own;
  }
  __syncthreads();
  if (e < E) {
    const int32_t g1 = in_g + sums[0][warp], p1 = in_p + sums[1][warp], q1 = in_q + sums[2][warp];
    sh_group[e] = g1 - total + before;
    sh_place[e] = p1 - padded + before;
    sh_pad[e] = p1 - padded;
    sh_pair[e] = q1 - pairs;
    sh_end[e] = p1 - padded + total;
    if (e == E - 1) {
      sh_pad[E] = p1;
      sh_pair[E] = q1;
      kept = g1;
    }
    if (rank == 0) {
      out.group_indices[e + 1] = g1;
      out.pad_offsets[e + 1] = p1;
      if (e == 0) { out.group_indices[0] = 0; out.pad_offsets[0] = 0; }
      if (out.tile_pairs != nullptr) {
        out.tile_pairs[out.mtiles_bound + e] = q1 - pairs;
        if (e == E - 1) out.tile_pairs[out.mtiles_bound + E] = q1;
      }
      if (out.num_mtiles != nullptr && e == E - 1) {
        out.num_mtiles[0] = p1 / MOE_TILE_M;
        out.num_mtiles[1] = q1;
        out.num_mtiles[2] = out.mtiles_bound;
        out.num_mtiles[3] = 0;
      }
    }
  }
  __syncthreads();

  // 4. place this CTA's rows
#pragma unroll
  for (int g = 0; g < kHeld; ++g) {
    const int64_t j = begin + 32 * g;
    if (g >= held || j >= R) break;
    if (key[g] >= 0) {
      const int32_t r = cnt[key[g]] + pos[g];
      if (out.perm != nullptr) out.perm[sh_group[key[g]] + r] = j;
      const int32_t p = sh_place[key[g]] + r;
      if (out.row_src != nullptr) out.row_src[p] = static_cast<int32_t>(j);
      if (out.dst_row != nullptr) out.dst_row[j] = p;
    } else if (out.dst_row != nullptr) {
      out.dst_row[j] = -1;  // id out of range: the row is in no expert's segment; consumers skip negative rows
    }
  }

  // 5. what no row wrote: padding rows, the tail of the row map, dropped positions, the tile maps
  const int gw = rank * kRouteWarps + warp, gws = ctas * kRouteWarps;
  const int gt = rank * kRouteThreads + tid, gts = ctas * kRouteThreads;
  if (out.row_src != nullptr) {
    for (int x = gw; x < E; x += gws)
      for (int32_t p = sh_end[x] + lane; p < sh_pad[x + 1]; p += 32) out.row_src[p] = -1;
    for (int32_t p = sh_pad[E] + gt; p < out.padded_bound; p += gts) out.row_src[p] = -1;
  }
  if (out.perm != nullptr)
    for (int64_t r = kept + gt; r < R; r += gts) out.perm[r] = -1;
  if (out.mtile_expert != nullptr) {
    const int tiles = sh_pad[E] / MOE_TILE_M;
    for (int m = gt; m < tiles; m += gts) {
      int lo = 0, hi = E;  // the expert whose padded rows hold tile m: last one that starts at or before it
      while (hi - lo > 1) {
        const int mid = (lo + hi) >> 1;
        if (sh_pad[mid] <= m * MOE_TILE_M) lo = mid; else hi = mid;
      }
      out.mtile_expert[m] = lo;
      const int in_expert = m - sh_pad[lo] / MOE_TILE_M;
      if (out.tile_pairs != nullptr && (in_expert & 1) == 0)
        out.tile_pairs[sh_pair[lo] + in_expert / 2] =
            static_cast<int32_t>(static_cast<uint32_t>(m) | (static_cast<uint32_t>(lo) << 20) |
                                 ((m + 1) * MOE_TILE_M < sh_pad[lo + 1] ? 0x80000000u : 0u));
    }
  }
  __syncwarp();
  asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
}

static size_t route_smem_bytes(int E) {
  return (static_cast<size_t>(kRouteWarps) * E + 6 * static_cast<size_t>(E) + 2) * sizeof(int32_t);
}

// The largest cluster (a power of two up to kMaxCluster) that can run on the current device.  A whole B200 takes all 16 CTAs in
// a GPC; a device with fewer SMs to a GPC may not, and a launch of a cluster that fits nowhere fails.  Asked once per
// device, for at most 256 experts and for more (39 and 155 KB of shared memory per CTA).
static int max_route_cluster(int E, int* out) {
  static std::atomic<int> known[64][2];
  const int wide = E > 256 ? 1 : 0;
  int dev = 0;
  MOE_CUDA(cudaGetDevice(&dev));
  const bool keep = dev >= 0 && dev < 64;
  int ctas = keep ? known[dev][wide].load(std::memory_order_acquire) : 0;
  if (ctas == 0) {
    MOE_CUDA(cudaFuncSetAttribute(route_cluster_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                  static_cast<int>(route_smem_bytes(kMaxExperts))));
    MOE_CUDA(cudaFuncSetAttribute(route_cluster_kernel, cudaFuncAttributeNonPortableClusterSizeAllowed, 1));
    for (ctas = kMaxCluster; ctas > 1; ctas /= 2) {
      cudaLaunchConfig_t cfg = {};
      cfg.gridDim = dim3(static_cast<unsigned>(ctas), 1, 1);
      cfg.blockDim = dim3(kRouteThreads, 1, 1);
      cfg.dynamicSmemBytes = route_smem_bytes(wide ? kMaxExperts : 256);
      cudaLaunchAttribute attr[1];
      attr[0].id = cudaLaunchAttributeClusterDimension;
      attr[0].val.clusterDim.x = static_cast<unsigned>(ctas);
      attr[0].val.clusterDim.y = 1;
      attr[0].val.clusterDim.z = 1;
      cfg.attrs = attr;
      cfg.numAttrs = 1;
      int clusters = 0;
      if (cudaOccupancyMaxActiveClusters(&clusters, route_cluster_kernel, &cfg) == cudaSuccess && clusters > 0) break;
      cudaGetLastError();  // a size the device refuses is an answer, not an error
    }
    if (keep) known[dev][wide].store(ctas, std::memory_order_release);
  }
  *out = ctas;
  return MOE_OK;
}

static int route_cluster(const int64_t* ids, int64_t R, int E, int max_ctas, const RouteOut& out, int32_t* status, cudaStream_t s) {
  // as many CTAs as there are 1024-row shares (the scattered stores of the placement are what one SM is slow at)
  int ctas = 1;
  while (ctas < max_ctas && static_cast<int64_t>(ctas) * kRouteThreads < R) ctas *= 2;
  const int64_t share = static_cast<int64_t>(ctas) * kRouteThreads;
  const int held = static_cast<int>((R + share - 1) / share);
  const size_t smem = route_smem_bytes(E);
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(static_cast<unsigned>(ctas), 1, 1);
  cfg.blockDim = dim3(kRouteThreads, 1, 1);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = s;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = static_cast<unsigned>(ctas);
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  MOE_CUDA(cudaLaunchKernelEx(&cfg, route_cluster_kernel, ids, R, E, held, out, status));
  return MOE_OK;
}

// Layout from an existing exclusive prefix (rows already grouped), in one launch: every CTA computes the padded prefix for
// itself (E values) and fills its share of the maps.  It replaces a memset, a one-CTA scan and a row kernel, and in the
// functional grouped GEMM six index operations besides (16 launches of 2-4 us each for 4111 tokens x 8 slots, two calls).
// `perm` (nullable): flat position of sorted row r.  Maps of padded row p that holds sorted row r, all nullable:
//   row_src r | in_rows perm[r] (r without perm) | out_rows perm[r] if scatter, else r;  padding rows: -1, kSkipRow, -1
struct GroupsOut {
  int32_t* pad_offsets;
  int32_t* row_src;
  int32_t* dst_row;
  int32_t* mtile_expert;
  int32_t* tile_pairs;
  int32_t* num_mtiles;
  int32_t* in_rows;
  int32_t* out_rows;
  int32_t mtiles_bound;
  uint32_t* work_counters;
};

__global__ void __launch_bounds__(kMaxExperts)
layout_from_groups_kernel(const int32_t* __restrict__ group_indices, int64_t R, int E, const int64_t* __restrict__ perm,
                          int scatter, GroupsOut out, int32_t* status) {
  __shared__ int32_t sh_lo[kMaxExperts], sh_cnt[kMaxExperts], sh_pad[kMaxExperts + 1], sh_pair[kMaxExperts + 1];
  __shared__ int32_t sums[2][32], cut[2];
  const int e = threadIdx.x, lane = e & 31, warp = e >> 5;
  grid_release();
  if (out.work_counters != nullptr && blockIdx.x == 0 && e < kWorkCounters) out.work_counters[e] = 0;
  int32_t cnt = 0, lo = 0;
  if (e < E) {
    // a prefix that is not monotone, does not start at 0 or does not end at R describes no layout: such experts
    // get no rows here and the status word says so
    lo = group_indices[e];
    const int32_t hi = group_indices[e + 1];
    const bool bad = hi < lo || lo < 0 || hi > R || (e == 0 && lo != 0) || (e == E - 1 && hi != R);
    if (bad && blockIdx.x == 0 && status != nullptr) atomicCAS(status, 0, DS_BAD_LAYOUT);
    cnt = bad ? 0 : hi - lo;
  }
  int32_t padded = (cnt + MOE_TILE_M - 1) / MOE_TILE_M * MOE_TILE_M;
  int32_t pairs = (padded / MOE_TILE_M + 1) / 2;
  // (capped: the sum over a prefix that is none can exceed 32 bits)
  constexpr int32_t kCap = 1 << 29;
  int32_t in_p = padded, in_q = pairs;
#pragma unroll
  for (int off = 1; off < 32; off <<= 1) {
    const int32_t a = __shfl_up_sync(0xFFFFFFFFu, in_p, off);
    const int32_t b = __shfl_up_sync(0xFFFFFFFFu, in_q, off);
    if (lane >= off) { in_p = min(in_p + a, kCap); in_q += b; }
  }
  if (lane == 31) { sums[0][warp] = in_p; sums[1][warp] = in_q; }
  __syncthreads();
  if (warp < 2) {
    int32_t v = sums[warp][lane];
#pragma unroll
    for (int off = 1; off < 32; off <<= 1) {
      const int32_t a = __shfl_up_sync(0xFFFFFFFFu, v, off);
      if (lane >= off) v = min(v + a, kCap);
    }
    const int32_t before = __shfl_up_sync(0xFFFFFFFFu, v, 1);
    sums[warp][lane] = lane > 0 ? before : 0;
  }
  __syncthreads();
  int32_t p1 = in_p + sums[0][warp], q1 = in_q + sums[1][warp];
  // A prefix that runs back and forth can give its experts more rows than there are, and the maps are sized for R: experts
  // whose padded rows would end past them are refused as well (the status word has been set by the step back).
  const bool over = e < E && p1 > out.mtiles_bound * MOE_TILE_M;
  if (__syncthreads_or(over)) {
    if (e == 0) { cut[0] = 0; cut[1] = 0; }
    __syncthreads();
    if (e < E && !over) { atomicMax(&cut[0], p1); atomicMax(&cut[1], q1); }
    __syncthreads();
    if (over) {
      cnt = padded = pairs = 0;
      p1 = cut[0];
      q1 = cut[1];
    }
  }
  if (e < E) {
    sh_lo[e] = lo;
    sh_cnt[e] = cnt;
    sh_pad[e] = p1 - padded;
    sh_pair[e] = q1 - pairs;
    if (e == E - 1) { sh_pad[E] = p1; sh_pair[E] = q1; }
    if (blockIdx.x == 0) {
      out.pad_offsets[e + 1] = p1;
      if (e == 0) out.pad_offsets[0] = 0;
      if (out.tile_pairs != nullptr) {
        out.tile_pairs[out.mtiles_bound + e] = q1 - pairs;
        if (e == E - 1) out.tile_pairs[out.mtiles_bound + E] = q1;
      }
      if (out.num_mtiles != nullptr && e == E - 1) {
        out.num_mtiles[0] = p1 / MOE_TILE_M;
        out.num_mtiles[1] = q1;
        out.num_mtiles[2] = out.mtiles_bound;
        out.num_mtiles[3] = 0;
      }
    }
  }
  __syncthreads();
  const int tid = blockIdx.x * kMaxExperts + e, threads = gridDim.x * kMaxExperts;
  // last expert whose padded rows begin at or before p (empty experts begin where the next one does)
  const auto owner = [&](int32_t p) {
    int a = 0, b = E;
    while (b - a > 1) {
      const int mid = (a + b) >> 1;
      if (sh_pad[mid] <= p) a = mid; else b = mid;
    }
    return a;
  };
  if (out.row_src != nullptr || out.in_rows != nullptr || out.out_rows != nullptr) {
    const int32_t bound = out.mtiles_bound * MOE_TILE_M;
    for (int32_t p = tid; p < bound; p += threads) {
      const int x = owner(p);
      const int32_t in_seg = p - sh_pad[x];
      const bool ok = p < sh_pad[E] && in_seg < sh_cnt[x];
      const int32_t r = sh_lo[x] + in_seg;
      int32_t f = -1;  // a negative entry of perm: no input row (zeros), no output row, whatever its value
      if (ok) {
        const int64_t j = perm != nullptr ? perm[r] : r;
        if (j >= 0) f = static_cast<int32_t>(j);
      }
      if (out.row_src != nullptr) out.row_src[p] = ok ? r : -1;
      if (out.in_rows != nullptr) out.in_rows[p] = ok ? f : kSkipRow;
      if (out.out_rows != nullptr) out.out_rows[p] = ok ? (scatter ? f : r) : -1;
    }
  }
  if (out.dst_row != nullptr) {
    for (int64_t j = tid; j < R; j += threads) {
      int a = 0, b = E;  // largest e with group_indices[e] <= j
      while (b - a > 1) {
        const int mid = (a + b) >> 1;
        if (sh_lo[mid] <= j) a = mid; else b = mid;
      }
      // rows of a segment that was refused (bad prefix) have no padded row
      const int64_t in_seg = j - sh_lo[a];
      out.dst_row[j] = in_seg >= 0 && in_seg < sh_cnt[a] ? sh_pad[a] + static_cast<int32_t>(in_seg) : -1;
    }
  }
  if (out.mtile_expert != nullptr) {
    const int tiles = sh_pad[E] / MOE_TILE_M;
    for (int m = tid; m < tiles; m += threads) {
      const int x = owner(m * MOE_TILE_M);
      out.mtile_expert[m] = x;
      const int in_expert = m - sh_pad[x] / MOE_TILE_M;
      if (out.tile_pairs != nullptr && (in_expert & 1) == 0)
        out.tile_pairs[sh_pair[x] + in_expert / 2] =
            static_cast<int32_t>(static_cast<uint32_t>(m) | (static_cast<uint32_t>(x) << 20) |
                                 ((m + 1) * MOE_TILE_M < sh_pad[x + 1] ? 0x80000000u : 0u));
    }
  }
}

}  // namespace moe

using namespace moe;

extern "C" int64_t moe_padded_rows_bound(int64_t num_rows, int num_experts) {
  if (num_rows < 0 || num_experts <= 0) return 0;
  // sum over experts of ceil(c_e / 128) * 128 <= R + E * 127, rounded up to a tile
  const int64_t worst = num_rows + static_cast<int64_t>(num_experts) * (MOE_TILE_M - 1);
  const int64_t rp = (worst + MOE_TILE_M - 1) / MOE_TILE_M * MOE_TILE_M;
  return rp > 0 ? rp : MOE_TILE_M;
}

extern "C" int64_t moe_mtiles_bound(int64_t num_rows, int num_experts) {
  return moe_padded_rows_bound(num_rows, num_experts) / MOE_TILE_M;
}

extern "C" size_t moe_routing_workspace_bytes(int64_t num_rows, int num_experts) {
  if (num_rows < 0 || num_experts <= 0) return 0;
  const int64_t chunks = num_chunks(num_rows) > 0 ? num_chunks(num_rows) : 1;
  return 2 * static_cast<size_t>(chunks) * num_experts * sizeof(int32_t);  // chunk histogram + chunk offsets
}

extern "C" int64_t moe_routing_one_launch_rows(int num_experts) {
  int ctas = 1;
  if (num_experts <= 0 || num_experts > kMaxExperts || max_route_cluster(num_experts, &ctas) != MOE_OK) ctas = 1;
  return static_cast<int64_t>(ctas) * kRouteThreads * kHeld;
}

namespace moe {

int routing_metadata(const int64_t* expert_idx, int64_t num_rows, int num_experts, int32_t* group_indices, int64_t* perm,
                     int32_t* pad_offsets, int32_t* row_src, int32_t* dst_row, int32_t* mtile_expert, int32_t* tile_pairs,
                     int32_t* num_mtiles, int32_t* status, void* workspace, size_t workspace_bytes,
                     bool workspace_always, void* stream) {
  MOE_CHECK_ARG(num_rows >= 0, "moe_routing_metadata: num_rows=%lld is negative", (long long)num_rows);
  MOE_CHECK_ARG(num_experts > 0, "moe_routing_metadata: num_experts=%d must be positive", num_experts);
  if (num_experts > kMaxExperts) {
    set_error("moe_routing_metadata: num_experts=%d exceeds the supported maximum %d", num_experts, kMaxExperts);
    return MOE_ERR_UNSUPPORTED;
  }
  MOE_CHECK_ARG(moe_mtiles_bound(num_rows, num_experts) < (1ll << 20),
                "moe_routing_metadata: num_rows=%lld needs more than 2^20 row tiles", (long long)num_rows);
  MOE_CHECK_ARG(group_indices && pad_offsets, "moe_routing_metadata: group_indices and pad_offsets are required");
  MOE_CHECK_ARG(num_rows == 0 || expert_idx != nullptr, "moe_routing_metadata: expert_idx is null");
  MOE_CHECK_ARG((mtile_expert == nullptr) == (num_mtiles == nullptr) && (tile_pairs == nullptr || mtile_expert != nullptr),
                "moe_routing_metadata: mtile_expert, tile_pairs and num_mtiles go together");
  const bool scratch = workspace != nullptr && workspace_bytes >= moe_routing_workspace_bytes(num_rows, num_experts);
  int64_t cluster_rows = kClusterRows;
  int max_ctas = kMaxCluster;
  if (scratch || !workspace_always) {
    const int rc = max_route_cluster(num_experts, &max_ctas);
    if (rc != MOE_OK) return rc;
    cluster_rows = static_cast<int64_t>(max_ctas) * kRouteThreads * kHeld;
  }
  MOE_CHECK_ARG(scratch || (!workspace_always && num_rows <= cluster_rows),
                "moe_routing_metadata: workspace of %zu bytes is smaller than the %zu required", workspace_bytes,
                moe_routing_workspace_bytes(num_rows, num_experts));
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  if (num_rows <= cluster_rows) {
    const RouteOut out{group_indices, perm, pad_offsets, row_src, dst_row, mtile_expert, tile_pairs, num_mtiles,
                       static_cast<int32_t>(moe_mtiles_bound(num_rows, num_experts)),
                       static_cast<int32_t>(moe_padded_rows_bound(num_rows, num_experts))};
    return route_cluster(expert_idx, num_rows, num_experts, max_ctas, out, status, s);
  }
  int32_t* chunk_hist = static_cast<int32_t*>(workspace);
  const int64_t chunks = num_chunks(num_rows);
  int32_t* chunk_off = chunk_hist + chunks * num_experts;
  const int blocks = static_cast<int>((chunks + kWarpsPerBlock - 1) / kWarpsPerBlock);
  const size_t sh = static_cast<size_t>(kWarpsPerBlock) * num_experts * sizeof(int32_t);
  if (row_src != nullptr) {
    MOE_CUDA(cudaMemsetAsync(row_src, 0xFF, moe_padded_rows_bound(num_rows, num_experts) * sizeof(int32_t), s));
  }
  chunk_histogram_kernel<<<blocks, kWarpsPerBlock * 32, sh, s>>>(expert_idx, num_rows, num_experts, chunk_hist, status);
  MOE_CUDA(cudaGetLastError());
  scan_chunks_kernel<<<num_experts, kScanThreads, 0, s>>>(chunk_hist, chunk_off, chunks, num_experts, group_indices);
  MOE_CUDA(cudaGetLastError());
  scan_offsets_kernel<<<1, kMaxExperts, 0, s>>>(num_experts, group_indices, pad_offsets, mtile_expert, tile_pairs, num_mtiles,
                                               static_cast<int>(moe_mtiles_bound(num_rows, num_experts)), perm, num_rows);
  MOE_CUDA(cudaGetLastError());
  if (perm || row_src || dst_row) {
    place_rows_kernel<<<blocks, kWarpsPerBlock * 32, sh, s>>>(expert_idx, num_rows, num_experts, chunk_off,
                                                             group_indices, pad_offsets, perm, row_src, dst_row);
    MOE_CUDA(cudaGetLastError());
  }
  return MOE_OK;
}

}  // namespace moe

extern "C" int moe_routing_metadata(const int64_t* expert_idx, int64_t num_rows, int num_experts,
                                    int32_t* group_indices, int64_t* perm, int32_t* pad_offsets, int32_t* row_src,
                                    int32_t* dst_row, int32_t* mtile_expert, int32_t* tile_pairs,
                                    int32_t* num_mtiles, int32_t* status, void* workspace, size_t workspace_bytes,
                                    void* stream) {
  return routing_metadata(expert_idx, num_rows, num_experts, group_indices, perm, pad_offsets, row_src, dst_row, mtile_expert,
                          tile_pairs, num_mtiles, status, workspace, workspace_bytes, true, stream);
}

static int layout_from_groups(const int32_t* group_indices, int64_t num_rows, int num_experts, const int64_t* perm, int scatter,
                              const GroupsOut& out, int32_t* status, cudaStream_t s) {
  // a CTA per 2048 padded rows: enough of them to spread the maps, few enough that the repeated prefix stays free
  const int64_t ctas = (static_cast<int64_t>(out.mtiles_bound) * MOE_TILE_M + 2047) / 2048;
  const int grid = static_cast<int>(ctas < sm_count() ? ctas : sm_count());
  layout_from_groups_kernel<<<grid, kMaxExperts, 0, s>>>(group_indices, num_rows, num_experts, perm, scatter, out, status);
  MOE_CUDA(cudaGetLastError());
  return MOE_OK;
}

extern "C" int moe_layout_from_groups(const int32_t* group_indices, int64_t num_rows, int num_experts,
                                      int32_t* pad_offsets, int32_t* row_src, int32_t* dst_row, int32_t* mtile_expert,
                                      int32_t* tile_pairs, int32_t* num_mtiles, int32_t* status, void* stream) {
  MOE_CHECK_ARG(group_indices && pad_offsets, "moe_layout_from_groups: group_indices and pad_offsets are required");
  MOE_CHECK_ARG(num_rows >= 0 && num_experts > 0, "moe_layout_from_groups: bad sizes R=%lld E=%d", (long long)num_rows,
                num_experts);
  MOE_CHECK_ARG(moe_mtiles_bound(num_rows, num_experts) < (1ll << 20),
                "moe_layout_from_groups: num_rows=%lld needs more than 2^20 row tiles", (long long)num_rows);
  if (num_experts > kMaxExperts) {
    set_error("moe_layout_from_groups: num_experts=%d exceeds the supported maximum %d", num_experts, kMaxExperts);
    return MOE_ERR_UNSUPPORTED;
  }
  MOE_CHECK_ARG((mtile_expert == nullptr) == (num_mtiles == nullptr) && (tile_pairs == nullptr || mtile_expert != nullptr),
                "moe_layout_from_groups: mtile_expert, tile_pairs and num_mtiles go together");
  return layout_from_groups(group_indices, num_rows, num_experts, nullptr, 0,
                            GroupsOut{pad_offsets, row_src, dst_row, mtile_expert, tile_pairs, num_mtiles, nullptr, nullptr,
                                      static_cast<int32_t>(moe_mtiles_bound(num_rows, num_experts)), nullptr},
                            status, static_cast<cudaStream_t>(stream));
}

extern "C" size_t moe_rows_pass_size(void) { return sizeof(moe_rows_pass); }

extern "C" int moe_rows_gemm(const moe_rows_pass* p, int steps, void* stream) {
  MOE_CHECK_ARG(p != nullptr, "moe_rows_gemm: null pointer argument");
  MOE_CHECK_ARG(p->group_indices && p->pad_offsets && p->out_rows && p->mtile_expert && p->tile_pairs && p->num_mtiles && p->a &&
                    (!p->gather || (p->in_rows && p->padded)) && ((!p->gather && !p->scatter) || p->perm),
                "moe_rows_gemm: null pointer argument");
  MOE_CHECK_ARG(p->num_rows > 0 && p->num_experts > 0 && p->a_rows >= 0 && p->topk > 0, "moe_rows_gemm: bad sizes");
  MOE_CHECK_ARG(p->act >= MOE_ACT_NONE && p->act <= MOE_ACT_GELU_TANH, "moe_rows_gemm: unknown activation %d", p->act);
  const int64_t mtiles = moe_mtiles_bound(p->num_rows, p->num_experts);
  MOE_CHECK_ARG(mtiles < (1ll << 20), "moe_rows_gemm: num_rows=%lld needs more than 2^20 row tiles", (long long)p->num_rows);
  if (p->num_experts > kMaxExperts) {
    set_error("moe_rows_gemm: num_experts=%d exceeds the supported maximum %d", p->num_experts, kMaxExperts);
    return MOE_ERR_UNSUPPORTED;
  }
  const Chain chain;
  const int64_t padded_rows = mtiles * MOE_TILE_M;
  if (steps & MOE_ROWS_LAYOUT)
    MOE_STEP(layout_from_groups(p->group_indices, p->num_rows, p->num_experts, p->gather || p->scatter ? p->perm : nullptr,
                                p->scatter,
                                GroupsOut{p->pad_offsets, nullptr, nullptr, p->mtile_expert, p->tile_pairs, p->num_mtiles,
                                          p->gather ? p->in_rows : nullptr, p->out_rows, static_cast<int32_t>(mtiles),
                                          reinterpret_cast<uint32_t*>(p->counters)},
                                p->status, static_cast<cudaStream_t>(stream)));
  if ((steps & MOE_ROWS_GATHER) && p->gather)
    MOE_STEP(gather_rows(p->a, p->a_rows, p->in_rows, p->num_mtiles, p->padded, padded_rows, p->k_dim, p->topk, p->dtype, stream,
                         true));
  if (steps & MOE_ROWS_GEMM) {
    RowCounts counts{p->pad_offsets, p->group_indices};
    counts.work_counter = reinterpret_cast<uint32_t*>(p->counters);
    counts.routed_rows = p->num_rows;
    // rows that are in expert order already are read where they are; gathered ones from their padded copy
    MOE_STEP(mgrouped_gemm_rows(p->gather ? p->padded : p->a, p->gather ? -1 : p->a_rows, p->w, p->out, p->out_rows,
                                p->mtile_expert, p->tile_pairs, p->num_mtiles, padded_rows, p->k_dim, p->n_dim, p->num_experts,
                                p->act, p->dtype, p->status, stream, counts));
  }
  return MOE_OK;
}
