// Grouped GEMM with transposed tiles: the weights are the 128-lane operand, an expert's rows are the accumulator columns.
//
// gemm_kernel.cuh puts 128 rows on the tensor core's lanes, so a tile costs 128 rows whatever the expert has, and a pair's
// second CTA idles where an expert ends in its first tile.  Here a CTA pair covers 256 weight columns and up to 256 rows of ONE
// expert (a row unit: a pair of row tiles, or one tile), and the extent of the instruction along the rows is chosen per work
// item in steps of 64: per 64-deep step a CTA loads its 16 KB of weights and 4 KB per 32 of its rows.  Nothing is computed
// for rows beyond an expert's last 64-row block, a pair never has an idle half, and the weights in flight do not shrink with
// the rows.  Bit-identical to the other kernels (the same products in the same order).
// Sums of a training pass's four such contractions (32 experts, d 2048, I 1024, K 1024-2048; us, gemm_kernel.cuh -> here, rows
// per expert even / moderately uneven / Zipf): 32 rows 209 / 219 / 214 -> 187 / 198 / 194 (weights streamed at 5.8 TB/s), 128
// rows 248 / 245 / 276 -> 229 / 229 / 247, 320 rows 351 / 354 / 357 -> 326 / 329 / 320, 700 rows 510 / 532 / 534 -> 491 / 504 / 505.
//
// Roles as in gemm_kernel.cuh: warp 0 TMA producer, warp 1 MMA issuer (leader CTA), warps 2-9 epilogue.  Each CTA of the pair
// holds the accumulators of its own 128 weight columns for all rows of the unit: TMEM lane = weight column, TMEM column = row.
// An epilogue warp therefore owns 32 weight columns; it turns 32 x 32 blocks around by exchanging packed pairs between
// neighbouring lanes (one shuffle and one shared-memory word per two elements, free of bank conflicts) and writes them
// as tensor copies of 32 rows x 32 (16 for gated outputs) columns.  The gated backward needs no exchange: the saved (gate, up)
// pair of a weight column is one 32-bit word of the row.
#pragma once

#include "gemm_kernel.cuh"

namespace moe {

struct TMaps {
  CUtensorMap w;     // the weights: box 128 (K-major) or 2 x 64 columns wide, 64 deep
  CUtensorMap c;     // EPI_GLU / EPI_ACT_AUX: un-activated product; EPI_DGLU: saved product
  CUtensorMap d;     // the output
  CUtensorMap r[4];  // the rows: boxes of 32, 64, 96, 128 rows
};

template <int UNIT, int EPI>
struct TPlan {
  static constexpr int kWBytes = 128 * BK * 2;
  static constexpr int kRowBytes = UNIT / 2 * BK * 2;  // a CTA's half of the unit's rows
  static constexpr int kStageBytes = kWBytes + kRowBytes;
  // per epilogue warp: two 32-row x 128-byte tiles of the saved product (gated backward); otherwise 4 KB, cut by the epilogue
  static constexpr int kWarpStaging = EPI == EPI_DGLU ? 8192 : 4096;
  static constexpr int kStagingBytes = kEpilogueWarps * kWarpStaging;
  static constexpr int kBarrierBytes = 1024;
  static constexpr int kBudget = 232448 - 1024 - kBarrierBytes - kStagingBytes;
  static constexpr int kStages = (kBudget / kStageBytes) > 8 ? 8 : (kBudget / kStageBytes);
  static constexpr int kTotal = kStages * kStageBytes + kStagingBytes + kBarrierBytes + 1024;
};

// One 32 x 32 block, lane = column, v[j] = row j, as the 16-bit words of a dense tile of 32 rows x 64 bytes.  Turning and storing
// are apart, so that the shuffles of a block overlap, and the wait for the store that last read the tile comes after the math.
template <typename T>
__device__ __forceinline__ void turn_block(const float (&v)[32], uint32_t (&w)[16], int lane) {
  const uint32_t sel = (lane & 1) ? 0x3276u : 0x5410u;
#pragma unroll
  for (int i = 0; i < 16; ++i) {
    const uint32_t own = Elem<T>::pack2(v[2 * i], v[2 * i + 1]);
    w[i] = __byte_perm(own, __shfl_xor_sync(0xFFFFFFFFu, own, 1), sel);
  }
}
__device__ __forceinline__ void store_block(const uint32_t (&w)[16], uint32_t tile, int lane) {
  const uint32_t addr = tile + (lane & 1) * 64 + (lane >> 1) * 4;
#pragma unroll
  for (int i = 0; i < 16; ++i) asm volatile("st.shared.b32 [%0], %1;" ::"r"(addr + i * 128), "r"(w[i]) : "memory");
}

// The gated activation of such a block (even lanes gate, odd lanes up), 32 rows x 32 bytes: even lanes compute even rows, odd
// lanes odd rows.
template <typename T, bool GEGLU>
__device__ __forceinline__ void turn_glu(const float (&v)[32], uint32_t (&w)[8], int lane) {
  const bool odd = lane & 1;
  float g[16];
#pragma unroll
  for (int i = 0; i < 16; ++i) {
    const float mine = odd ? v[2 * i + 1] : v[2 * i];
    const float got = __shfl_xor_sync(0xFFFFFFFFu, odd ? v[2 * i] : v[2 * i + 1], 1);
    const float gate = odd ? got : mine, up = odd ? mine : got;
    g[i] = (GEGLU ? gelu_f(gate) : silu_f(gate)) * up;
  }
  const uint32_t sel = (lane & 2) ? 0x3276u : 0x5410u;
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    const uint32_t own = Elem<T>::pack2(g[2 * i], g[2 * i + 1]);
    w[i] = __byte_perm(own, __shfl_xor_sync(0xFFFFFFFFu, own, 2), sel);
  }
}
__device__ __forceinline__ void store_glu(const uint32_t (&w)[8], uint32_t tile, int lane) {
  const uint32_t addr = tile + (lane & 3) * 32 + (lane >> 2) * 4;
#pragma unroll
  for (int i = 0; i < 8; ++i) asm volatile("st.shared.b32 [%0], %1;" ::"r"(addr + i * 128), "r"(w[i]) : "memory");
}

// The gated backward of a 32 x 32 block in place: tile holds 32 rows x 32 (gate, up) words with the 128-byte swizzle, lane = word.
template <typename T, bool GEGLU>
__device__ __forceinline__ void dglu_block(const float (&da)[32], uint32_t tile, int lane) {
  // (all loads first: a volatile load does not move over the store of the row before it)
  uint32_t w[32];
#pragma unroll
  for (int r = 0; r < 32; ++r)
    asm volatile("ld.shared.b32 %0, [%1];" : "=r"(w[r]) : "r"(tile + r * 128 + (((lane >> 2) ^ (r & 7)) << 4) + (lane & 3) * 4));
#pragma unroll
  for (int r = 0; r < 32; ++r) {
    const float2 gu = Elem<T>::unpack2(w[r]);
    float act_g, dact_g;
    if (GEGLU) {
      act_g = gelu_f(gu.x);
      dact_g = dgelu_f(gu.x);
    } else {
      const float sg = sigmoidf_fast(gu.x);
      act_g = gu.x * sg;
      dact_g = sg * (1.0f + gu.x * (1.0f - sg));
    }
    w[r] = Elem<T>::pack2(da[r] * gu.y * dact_g, da[r] * act_g);
  }
#pragma unroll
  for (int r = 0; r < 32; ++r)
    asm volatile("st.shared.b32 [%0], %1;" ::"r"(tile + r * 128 + (((lane >> 2) ^ (r & 7)) << 4) + (lane & 3) * 4), "r"(w[r])
                 : "memory");
}

namespace transposed {

template <typename T, int UNIT, bool W_K, int EPI>
__global__ void __launch_bounds__(kThreads, 1)
grouped_gemm_kernel(const __grid_constant__ TMaps maps, const GemmArgs args) {
  using Plan = TPlan<UNIT, EPI>;
  constexpr int kStages = Plan::kStages;
  constexpr int kTilesPerUnit = UNIT / BM;
  constexpr int BN = 256;  // weight columns of the pair
  extern __shared__ uint8_t smem_raw[];
  const uint32_t raw_addr = smem_u32(smem_raw);
  const uint32_t tiles_addr = (raw_addr + 1023u) & ~1023u;
  uint8_t* tiles = smem_raw + (tiles_addr - raw_addr);
  const uint32_t staging_addr = tiles_addr + kStages * Plan::kStageBytes;
  uint64_t* bars = reinterpret_cast<uint64_t*>(tiles + kStages * Plan::kStageBytes + Plan::kStagingBytes);
  const uint32_t full_bar = smem_u32(bars);                      // [kStages]  (used in the leader CTA)
  const uint32_t empty_bar = smem_u32(bars + kStages);           // [kStages]  (one set per CTA)
  const uint32_t tfull_bar = smem_u32(bars + 2 * kStages);       // [2]        (one set per CTA)
  const uint32_t tempty_bar = smem_u32(bars + 2 * kStages + 2);  // [2]        (used in the leader CTA)
  const uint32_t epi_bar = smem_u32(bars + 2 * kStages + 4);     // [kEpilogueWarps][2]  (saved product tiles)
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 2 * kStages + 4 + 2 * kEpilogueWarps);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);
  static_assert((2 * 8 + 4 + 2 * kEpilogueWarps) * 8 + 8 <= kQueueOffset && kQueueOffset + kQueueBarrierBytes + kQueueSlots * 32 <= Plan::kBarrierBytes,
                "barrier area too small");
  const ItemQueue queue(smem_u32(bars) + kQueueOffset);
  const bool queued = args.work_counter != nullptr;

  const int warp = threadIdx.x >> 5;
  const int lane = threadIdx.x & 31;
  const int rank = static_cast<int>(cluster_ctarank());  // 0 = leader of the pair
  const int unit = blockIdx.x >> 1;
  const int num_units = gridDim.x >> 1;

  WaitCtx wctx;
  wctx.abort_flag = abort_flag;
  wctx.peer_abort = mapa_shared(smem_u32(const_cast<int*>(abort_flag)), static_cast<uint32_t>(rank ^ 1));
  wctx.status = args.status;
  wctx.limit = args.wait_limit;

  if (threadIdx.x == 0) {
    for (int s = 0; s < kStages; ++s) {
      mbar_init(full_bar + 8 * s, 2);  // one arrive.expect_tx per CTA
      mbar_init(empty_bar + 8 * s, 1);
    }
    for (int a = 0; a < 2; ++a) {
      mbar_init(tfull_bar + 8 * a, 1);
      mbar_init(tempty_bar + 8 * a, kEpilogueWarps * 2);
    }
    for (int i = 0; i < 2 * kEpilogueWarps; ++i) mbar_init(epi_bar + 8 * i, 1);
    queue.init();
    *abort_flag = 0;
    mbar_fence_init();
    tma_prefetch_desc(&maps.w);
    for (int i = 0; i < UNIT / 64; ++i) tma_prefetch_desc(&maps.r[i]);
    if (EPI == EPI_DGLU || EPI == EPI_ACT_AUX || (EPI == EPI_GLU && args.aux_out != nullptr)) tma_prefetch_desc(&maps.c);
    if (EPI == EPI_DGLU || EPI == EPI_ACT_AUX || args.out_tma) tma_prefetch_desc(&maps.d);
  }
  if (warp == 1) {
    tmem_alloc_pair(smem_u32(tmem_slot), kTmemCols);
    tmem_relinquish_pair();
  }
  prefetch_maps(args);
  tc_fence_before();
  __syncthreads();
  cluster_sync_all();  // the peer's barriers must be initialised before anything arrives on them
  tc_fence_after();
  // Nothing above reads or writes global memory.  Where the row maps and the weights were complete before the kernel before could
  // let this one start, only what that kernel writes has to be waited for: each role waits for itself, the producer after the
  // weights of its first stages.  That fills most of the gap between two contractions: from the wait on, the maps took 1.5 us and
  // the first weights 1 to 3.  Whole passes: 128 tokens, 64 experts, training 523 -> 512 us, 1777 tokens, 12 ungated experts 297 -> 282;
  // 33 tokens, forward 143.6 -> 141.2; equal where the contractions are long.
  if (!args.settled) grid_wait();
  const uint32_t tmem_base = *tmem_slot;

  int mt, nt;
  Window win;
  const int ntiles = total_tiles<false, kTilesPerUnit>(args, mt, nt, win, BN);
  ItemWalk<false, kTilesPerUnit> walk(unit, num_units, ntiles, mt, nt, BN, 0);
  const auto item = [&](int i, bool mark_taken, int code) {
    return queued ? queue.template get<false>(i, args, mark_taken, wctx, code) : walk.get(i, win, args);
  };

  if (warp == 0) {
    // ------------------------------ TMA producer ------------------------------
    int stage = 0;
    uint32_t phase = 0;
    bool ok = true;
    bool freed = false;  // the stage about to be filled was already seen free (probed one stage ahead)
    const uint64_t pol = l2_policy_evict_normal();
    // operand arrival is credited to the leader's barriers, in its own and in the cluster window alike
    const uint32_t full_leader = mapa_shared(full_bar, 0);
    // by one lane: a stage's share of the weights, announcing `bytes`
    const auto load_weights = [&](int s, int kb, const TileCoord& c, uint32_t bytes) {
      const int col0 = c.n0 + rank * 128;
      const uint32_t sw = tiles_addr + s * Plan::kStageBytes;
      const uint32_t fb = full_leader + 8 * s;
      mbar_arrive_expect_tx_cluster(fb, bytes);
      if (W_K) {
        tma_load_3d_pair(sw, &maps.w, kb * BK, col0, c.expert, fb, pol);
      } else if (args.b_blocked) {
        tma_load_4d_pair(sw, &maps.w, 0, kb * BK, col0 >> 6, c.expert, fb, pol);
      } else {
#pragma unroll
        for (int j = 0; j < 2; ++j) tma_load_3d_pair(sw + j * (BK * 128), &maps.w, col0 + 64 * j, kb * BK, c.expert, fb, pol);
      }
    };
    for (int i = 0; ok; ++i) {
      const TileCoord c = item(i, rank == 0, DS_TIMEOUT_PRODUCER);
      if (!c.valid) break;
      const int steps = (c.unit_rows + 63) >> 6;  // of 64 rows, 32 in each CTA
      const CUtensorMap* rows_map = &maps.r[steps - 1];
      const int row0 = c.a_row + rank * steps * 32;
      const uint32_t bytes = Plan::kWBytes + steps * (32 * BK * 2);
      int kb = 0;
      if (i == 0 && args.settled) {
        kb = c.kiters < kStages ? c.kiters : kStages;
        if (elect_one())
          for (int s = 0; s < kb; ++s) load_weights(s, s, c, bytes);
        __syncwarp();
        grid_wait();
        if (elect_one())
          for (int s = 0; s < kb; ++s)
            tma_load_2d_pair(tiles_addr + s * Plan::kStageBytes + Plan::kWBytes, rows_map, s * BK, row0, full_leader + 8 * s, pol);
        __syncwarp();
        if ((stage = kb) == kStages) { stage = 0; phase = 1; }
      }
      for (; kb < c.kiters; ++kb) {
        if (!freed && !__all_sync(0xFFFFFFFFu, mbar_wait(empty_bar + 8 * stage, phase ^ 1, wctx, DS_TIMEOUT_PRODUCER))) {
          ok = false;
          break;
        }
        {
          const int ns = stage + 1 == kStages ? 0 : stage + 1;
          freed = __all_sync(0xFFFFFFFFu, mbar_test_wait(empty_bar + 8 * ns, stage + 1 == kStages ? phase : phase ^ 1));
        }
        if (elect_one()) {
          load_weights(stage, kb, c, bytes);
          tma_load_2d_pair(tiles_addr + stage * Plan::kStageBytes + Plan::kWBytes, rows_map, kb * BK, row0, full_leader + 8 * stage,
                           pol);
        }
        __syncwarp();
        if (++stage == kStages) { stage = 0; phase ^= 1; }
      }
    }
    grid_wait();  // (a producer without an item has not)
    grid_release();  // all operand loads are issued: the next chained kernel may come up beside the last tile
    if (!ok || *abort_flag) {
      // Let copies that were already issued land before the CTA releases its shared memory.
      for (int i = 0; i < 2000; ++i) __nanosleep(1000);
    }
  } else if (warp == 1) {
    // ------------------------------ MMA issuer (leader CTA only) --------------
    if (rank == 0) {
      // the rows' extent of the instruction (bits 17-22, in eights) is filled in per work item
      constexpr uint32_t idesc0 = make_idesc<T, 0, W_K, true, 2>();
      int stage = 0;
      uint32_t phase = 0;
      int acc = 0;
      uint32_t acc_phase = 0;
      bool ok = true;
      bool ready = false;  // the stage about to be consumed was already seen full
      for (int i = 0; ok; ++i) {
        const TileCoord c = item(i, false, DS_TIMEOUT_MMA);
        if (!c.valid) break;
        if (i == 0) grid_wait();  // (the limits of the waits below are not to run out on the kernel before)
        const uint32_t idesc = idesc0 | (static_cast<uint32_t>((c.unit_rows + 63) >> 6) * 8u) << 17;
        if (!__all_sync(0xFFFFFFFFu, mbar_wait(tempty_bar + 8 * acc, acc_phase ^ 1, wctx, DS_TIMEOUT_MMA))) {
          ok = false;
          break;
        }
        tc_fence_after();
        const uint32_t d_tmem = tmem_base + acc * UNIT;
        for (int kb = 0; kb < c.kiters; ++kb) {
          if (!ready && !__all_sync(0xFFFFFFFFu, mbar_wait(full_bar + 8 * stage, phase, wctx, DS_TIMEOUT_MMA))) {
            ok = false;
            break;
          }
          tc_fence_after();
          {
            const int ns = stage + 1 == kStages ? 0 : stage + 1;
            ready = __all_sync(0xFFFFFFFFu, mbar_test_wait(full_bar + 8 * ns, stage + 1 == kStages ? phase ^ 1 : phase));
          }
          const uint32_t sw = tiles_addr + stage * Plan::kStageBytes;
          const uint32_t sr = sw + Plan::kWBytes;
          if (elect_one()) {
#pragma unroll
            for (int k = 0; k < BK / UMMA_K; ++k) {
              const uint64_t dw = W_K ? make_desc(sw + k * (UMMA_K * 2), 16, 1024)
                                      : make_desc(sw + k * (UMMA_K * 128), BK * 128, 1024);
              const uint64_t dr = make_desc(sr + k * (UMMA_K * 2), 16, 1024);
              umma_f16_pair(d_tmem, dw, dr, idesc, (kb | k) != 0 ? 1u : 0u);
            }
            umma_commit_pair_both(empty_bar + 8 * stage);
          }
          __syncwarp();
          if (++stage == kStages) { stage = 0; phase ^= 1; }
        }
        if (!ok) break;
        if (elect_one()) umma_commit_pair_both(tfull_bar + 8 * acc);
        __syncwarp();
        if (++acc == 2) { acc = 0; acc_phase ^= 1; }
      }
      if (!ok || *abort_flag) {
        for (int i = 0; i < 2000; ++i) __nanosleep(1000);
      }
    } else if (queued) {
      queue.template serve<false, kTilesPerUnit>(unit, num_units, ntiles, mt, nt, BN, win, args, wctx);
    }
  } else {
    // ------------------------------ epilogue ----------------------------------
    // Warp w reads TMEM lane quadrant (w % 4), i.e. 32 weight columns; the two warps of a quadrant take the 32-row chunks in turn.
    const int quad = warp & 3;
    const int half = (warp - 2) >> 2;
    int acc = 0;
    uint32_t acc_phase = 0;
    T* out = reinterpret_cast<T*>(args.out);
    const int N = args.n_dim;
    const uint32_t tempty_leader = mapa_shared(tempty_bar, 0);
    const uint32_t stage_base = staging_addr + (warp - 2) * Plan::kWarpStaging;
    const uint32_t my_epi_bar = epi_bar + (warp - 2) * 16;
    uint32_t q = 0;      // running count of saved-product tiles this warp has received; two tiles are used in turn
    uint32_t turn = 0;   // staging tile of plain and gated results, two in turn
    const bool side_input = EPI == EPI_DGLU || (EPI == EPI_ACT_AUX && args.aux_in != nullptr);
    constexpr uint32_t kSideTile = EPI == EPI_DGLU ? 4096 : 2048;
    for (int i = 0;; ++i) {
      const TileCoord c = item(i, false, DS_TIMEOUT_EPILOGUE);
      if (!c.valid) break;
      if (i == 0) grid_wait();
      const int col0 = c.n0 + rank * 128 + quad * 32;  // this warp's first weight column
      const int chunks = col0 < N ? ((c.unit_rows + 63) >> 6) * 2 : 0;
      if (side_input && half < chunks) {
        // the saved product does not depend on the accumulator: request the first chunk's tile before waiting for the MMAs
        if (lane == 0) {
          bulk_wait_read_all();
          const uint32_t bar = my_epi_bar + 8 * (q & 1);
          mbar_arrive_expect_tx(bar, kSideTile);
          tma_load_2d_plain(stage_base + (q & 1) * kSideTile, &maps.c, EPI == EPI_DGLU ? 2 * col0 : col0, c.m0 + half * 32, bar);
        }
        __syncwarp();
      }
      if (!__all_sync(0xFFFFFFFFu, mbar_wait(tfull_bar + 8 * acc, acc_phase, wctx, DS_TIMEOUT_EPILOGUE))) break;
      tc_fence_after();
      const uint32_t taddr = tmem_base + (static_cast<uint32_t>(quad * 32) << 16) + acc * UNIT;
      bool failed = false;
#pragma unroll 1
      for (int chunk = half; chunk < chunks; chunk += 2) {
        const int row0 = c.m0 + chunk * 32;
        const uint32_t side = stage_base + (q & 1) * kSideTile;
        if (side_input) {
          if (chunk + 2 < chunks && lane == 0) {
            bulk_wait_read_all();  // the store that last read the other tile is done with it
            const uint32_t nbar = my_epi_bar + 8 * ((q + 1) & 1);
            mbar_arrive_expect_tx(nbar, kSideTile);
            tma_load_2d_plain(stage_base + ((q + 1) & 1) * kSideTile, &maps.c, EPI == EPI_DGLU ? 2 * col0 : col0, row0 + 64, nbar);
          }
          __syncwarp();
          if (!__all_sync(0xFFFFFFFFu, mbar_wait(my_epi_bar + 8 * (q & 1), (q >> 1) & 1, wctx, DS_TIMEOUT_EPILOGUE))) {
            failed = true;
            break;
          }
        }
        float v[32];
        {
          uint32_t raw[32];
          tmem_ld_32x32(taddr + chunk * 32, raw);
          tmem_ld_wait();
#pragma unroll
          for (int i = 0; i < 32; ++i) v[i] = __uint_as_float(raw[i]);
        }
        if (EPI == EPI_ACT) {
          apply_act(v, args.act);
          const uint32_t tile = stage_base + (turn & 1) * 2048;
          ++turn;
          uint32_t w[16];
          if (args.out_tma) {
            turn_block<T>(v, w, lane);
            if (lane == 0) bulk_wait_read_one();  // the store before the last has read this tile
            __syncwarp();
            store_block(w, tile, lane);
            fence_proxy_async_smem();
            __syncwarp();
            if (lane == 0) {
              tma_store_2d(&maps.d, col0, row0, tile);
              bulk_commit();
            }
          } else {
            // row map, or scaled and added into token-order rows: lane l looks up row l of the chunk
            const bool accumulate = args.combine_row_src != nullptr;
            int dst = -1;
            if (accumulate) {
              const int j = args.combine_row_src[row0 + lane];
              float scale = 1.0f;
              if (j >= 0) {
                dst = j / args.combine_topk;
                if (args.combine_scores != nullptr) scale = Elem<T>::to_float(reinterpret_cast<const T*>(args.combine_scores)[j]);
              }
#pragma unroll
              for (int i = 0; i < 32; ++i) v[i] *= __shfl_sync(0xFFFFFFFFu, scale, i);
            } else {
              dst = args.push_row[row0 + lane];
            }
            turn_block<T>(v, w, lane);
            store_block(w, tile, lane);
            __syncwarp();
            const int piece = lane & 3;
            const bool in = col0 + piece * 8 < N;
#pragma unroll
            for (int j = 0; j < 4; ++j) {
              const int r = j * 8 + (lane >> 2);
              const int to = __shfl_sync(0xFFFFFFFFu, dst, r);
              uint4 u;
              asm volatile("ld.shared.v4.b32 {%0, %1, %2, %3}, [%4];"
                           : "=r"(u.x), "=r"(u.y), "=r"(u.z), "=r"(u.w)
                           : "r"(tile + r * 64 + piece * 16));
              if (to >= 0 && in) {
                T* p = out + static_cast<long long>(to) * N + col0 + piece * 8;
                if (accumulate) red_add_v8<T>(p, u);
                else *reinterpret_cast<uint4*>(p) = u;
              }
            }
            __syncwarp();
          }
        } else if (EPI == EPI_GLU) {
          // tiles: with the un-activated product 2 KB of it and 1 KB of the result, else two of 1 KB in turn
          const bool aux = args.aux_out != nullptr;
          const uint32_t tile = stage_base + (aux ? 2048 : (turn & 1) * 1024);
          ++turn;
          uint32_t w[16], g[8];
          if (aux) turn_block<T>(v, w, lane);
          if (args.act == MOE_ACT_GEGLU) turn_glu<T, true>(v, g, lane);
          else turn_glu<T, false>(v, g, lane);
          if (args.out_tma) {
            if (lane == 0) {
              if (aux) bulk_wait_read_all();
              else bulk_wait_read_one();
            }
            __syncwarp();
          }
          if (aux) store_block(w, stage_base, lane);
          store_glu(g, tile, lane);
          if (args.out_tma) {
            fence_proxy_async_smem();
            __syncwarp();
            if (lane == 0) {
              if (aux) tma_store_2d(&maps.c, col0, row0, stage_base);
              tma_store_2d(&maps.d, col0 >> 1, row0, tile);
              bulk_commit();
            }
          } else {
            const int dst = args.push_row[row0 + lane];
            __syncwarp();
            const int piece = lane & 1;
            const bool in = (col0 >> 1) + piece * 8 < (N >> 1);
#pragma unroll
            for (int j = 0; j < 2; ++j) {
              const int r = j * 16 + (lane >> 1);
              const int to = __shfl_sync(0xFFFFFFFFu, dst, r);
              uint4 u;
              asm volatile("ld.shared.v4.b32 {%0, %1, %2, %3}, [%4];"
                           : "=r"(u.x), "=r"(u.y), "=r"(u.z), "=r"(u.w)
                           : "r"(tile + r * 32 + piece * 16));
              if (to >= 0 && in)
                *reinterpret_cast<uint4*>(out + static_cast<long long>(to) * (N >> 1) + (col0 >> 1) + piece * 8) = u;
            }
            __syncwarp();
          }
        } else if (EPI == EPI_DGLU) {
          if (args.act == MOE_ACT_GEGLU) dglu_block<T, true>(v, side, lane);
          else dglu_block<T, false>(v, side, lane);
          fence_proxy_async_smem();
          __syncwarp();
          if (lane == 0) {
            tma_store_2d(&maps.d, 2 * col0, row0, side);
            bulk_commit();
          }
          ++q;
        } else if (side_input) {  // EPI_ACT_AUX, backward: the row block of the saved product is replaced in place
          float x[32];
#pragma unroll
          for (int r = 0; r < 32; ++r) {
            uint16_t u;
            asm volatile("ld.shared.u16 %0, [%1];" : "=h"(u) : "r"(side + r * 64 + lane * 2));
            x[r] = Elem<T>::unpack2(u).x;
          }
          mul_dact(v, x, args.act);
          uint32_t w[16];
          turn_block<T>(v, w, lane);
          __syncwarp();
          store_block(w, side, lane);
          fence_proxy_async_smem();
          __syncwarp();
          if (lane == 0) {
            tma_store_2d(&maps.d, col0, row0, side);
            bulk_commit();
          }
          ++q;
        } else {  // EPI_ACT_AUX, forward: un-activated and activated product from one tile each
          uint32_t w[16], g[16];
          turn_block<T>(v, w, lane);
          apply_act(v, args.act);
          turn_block<T>(v, g, lane);
          if (lane == 0) bulk_wait_read_all();
          __syncwarp();
          store_block(w, stage_base, lane);
          store_block(g, stage_base + 2048, lane);
          fence_proxy_async_smem();
          __syncwarp();
          if (lane == 0) {
            tma_store_2d(&maps.c, col0, row0, stage_base);
            tma_store_2d(&maps.d, col0, row0, stage_base + 2048);
            bulk_commit();
          }
        }
      }
      if (failed) break;
      // this warp has read its part of the accumulator: one arrival per warp on the leader's barrier
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive_cluster(tempty_leader + 8 * acc);
      if (++acc == 2) { acc = 0; acc_phase ^= 1; }
    }
    if (lane == 0) bulk_wait_all();  // this warp's bulk stores are complete
  }

  grid_wait();  // this kernel is not complete before the one before it, whatever it had to do
  tc_fence_before();
  __syncthreads();
  cluster_sync_all();  // neither CTA may exit while its peer can still touch its memory or barriers
  if (warp == 1) {
    __syncwarp();
    tc_fence_after();
    tmem_dealloc_pair(tmem_base, kTmemCols);
  }
}

}  // namespace transposed

// Launches one variant with as many persistent CTA pairs as fit the current device.
template <typename T, int UNIT, bool W_K, int EPI>
int launch_t(const TMaps& maps, const GemmArgs& args, const LaunchParams& lp);

#ifdef MOE_GEMM_DEFINE_LAUNCH
template <typename T, int UNIT, bool W_K, int EPI>
int launch_t(const TMaps& maps, const GemmArgs& args, const LaunchParams& lp) {
  auto kernel = transposed::grouped_gemm_kernel<T, UNIT, W_K, EPI>;
  static_assert(TPlan<UNIT, EPI>::kStages >= 4, "too few operand stages");
  static std::atomic<int> grids[64];
  PersistentLaunch l;
  const int rc = configure<2>(l, kernel, TPlan<UNIT, EPI>::kTotal, grids, lp);
  if (rc != MOE_OK) return rc;
  MOE_CUDA(cudaLaunchKernelEx(&l.cfg, kernel, maps, args));
  return MOE_OK;
}
#endif  // MOE_GEMM_DEFINE_LAUNCH

}  // namespace moe
