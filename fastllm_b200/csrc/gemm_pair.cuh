// Large-M 16-bit GEMM body on CTA pairs: 256 tokens x 256 out-features, the pair's two SMs on one product (cta_group::2).
// Included after gemm_largem.cuh (epilogue, hook).
//
// Bound of the one-CTA body: a 128 x 256 tile brings 48 KB into shared memory for every 64 of k, more than the L2 hands an SM in the 512 cycles
// that the tensor core needs for them.  A pair's CTA holds its own 128 tokens and half of the 256 weight rows, which the tensor cores of both
// read: 32 KB for the same work, and the ring is six stages deep.
// One launch, us (TFLOP/s), one CTA a tile -> pairs: 8190 x 4096 x 14336 775 (1241) -> 667 (1443), 8190 x 4096 x 4096 205 (1342) -> 177 (1551),
// 1000 x 28672 x 4096 263 (892) -> 234 (1002).  Back to back the power limit takes over: 8190 x 28672 x 4096 1285 -> 1309 TFLOP/s.
#pragma once
#include "gemm_largem.cuh"

namespace fb {

struct PairCfg {
  static constexpr int BN = 256;
  static constexpr int A_BYTES = 128 * 128;              // 128 token rows x 64 of k
  static constexpr int B_BYTES = 128 * 128;              // this CTA's half of the 256 weight rows
  static constexpr int STAGE_BYTES = A_BYTES + B_BYTES;
  static constexpr int STAGES = 6;
  static constexpr int BODY_BYTES = STAGES * STAGE_BYTES;
  static constexpr int SMEM_BYTES = BODY_BYTES + 256 + 1024;
  static constexpr int TMEM_COLS = 2 * BN;               // two accumulators: epilogue of tile i overlaps the MMAs of tile i + 1
};

// Warp roles as in gemm_largem_device.  Both CTAs load their own operands on the first CTA's `full` barriers; its warp 1 issues the products and
// commits them to `empty` and `acc_full` of both; the epilogue warps of both hand an accumulator back to the first CTA.
template <bool BF16, class Hook, bool EXTRA = false>
__device__ __forceinline__ void gemm_pair_device(const CUtensorMap& tmX, const CUtensorMap& tmW, const GemmParams& p, int tiles_m, int tiles_n, const Hook& hook,
                                                 const GemmExtra& ex = GemmExtra()) {
  using Cfg = PairCfg;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint64_t* full_bar = reinterpret_cast<uint64_t*>(smem + Cfg::BODY_BYTES);      // the first CTA's are used
  uint64_t* empty_bar = full_bar + Cfg::STAGES;
  uint64_t* acc_full = empty_bar + Cfg::STAGES;        // [2] accumulator ready for the epilogue
  uint64_t* acc_empty = acc_full + 2;                  // [2] accumulator drained (4 epilogue warps of each CTA; the first CTA's are used)
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(acc_empty + 2);

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int rank = (int)cluster_ctarank(), pair = (int)(blockIdx.x >> 1), pairs = (int)(gridDim.x >> 1);
  const int kb_cnt = p.kb_total;
  const int tiles = tiles_m * tiles_n;
  bool dead = false;

  if (threadIdx.x == 0) {
    for (int s = 0; s < Cfg::STAGES; ++s) { mbar_init(&full_bar[s], 1); mbar_init(&empty_bar[s], 1); }
    for (int b = 0; b < 2; ++b) { mbar_init(&acc_full[b], 1); mbar_init(&acc_empty[b], 8); }
    mbar_init_fence();
    tma_prefetch_desc(&tmW);
    tma_prefetch_desc(&tmX);
  }
  if (warp == 1) { tmem_alloc_pair(tmem_slot, Cfg::TMEM_COLS); tmem_relinquish_pair(); }
  tc_fence_before_sync();
  __syncthreads();
  cluster_sync_all();                                  // the other CTA's barriers exist, too
  tc_fence_after_sync();
  const uint32_t tmem_base = *tmem_slot;

  if (warp == 0) {
    if (elect_one()) {
      int it = 0;                                      // k-block counter across all of this pair's tiles
      for (int t = pair; t < tiles && !dead; t += pairs) {
        int m_tile, n_tile;
        hook.tile_coords(t, tiles_m, tiles_n, m_tile, n_tile);
        const int x0 = p.batch_w_rows > 0 ? n_tile * Cfg::BN / p.batch_w_rows * p.batch_x_cols : 0;      // block-diagonal weights
        for (int i = 0; i < kb_cnt; ++i, ++it) {
          const int s = it % Cfg::STAGES;
          if (!mbar_wait(&empty_bar[s], ((uint32_t)(it / Cfg::STAGES) & 1u) ^ 1u, dead, KID_GEMM_LARGEM, 5)) break;
          uint8_t* a = smem + s * Cfg::STAGE_BYTES;
          const uint32_t bar = mapa_u32(smem_u32(&full_bar[s]), 0);
          if (rank == 0) mbar_expect_tx(&full_bar[s], 2 * Cfg::STAGE_BYTES);
          tma_load_2d_pair(a, &tmX, bar, x0 + i * 64, m_tile * 256 + rank * 128);
          tma_load_2d_pair(a + Cfg::A_BYTES, &tmW, bar, i * 64, n_tile * Cfg::BN + rank * 128);
        }
      }
      // the last products' commits have reached this CTA before it may leave
      for (int k = it > Cfg::STAGES ? it - Cfg::STAGES : 0; k < it; ++k)
        if (!mbar_wait(&empty_bar[k % Cfg::STAGES], (uint32_t)(k / Cfg::STAGES) & 1u, dead, KID_GEMM_LARGEM, 6)) break;
    }
    __syncwarp();
  } else if (warp == 1) {
    if (rank == 0 && elect_one()) {
      int it = 0, u = 0;                               // u: tiles done by this pair
      for (int t = pair; t < tiles && !dead; t += pairs, ++u) {
        const int buf = u & 1;
        const uint32_t use = (uint32_t)(u >> 1) & 1u;      // how often this buffer has been used, parity
        if (!mbar_wait_cluster(&acc_empty[buf], use ^ 1u, dead, KID_GEMM_LARGEM, 8)) break;     // first use passes at once
        tc_fence_after_sync();
        const uint32_t acc = tmem_base + (uint32_t)(buf * Cfg::BN);
        for (int i = 0; i < kb_cnt; ++i, ++it) {
          const int s = it % Cfg::STAGES;
          if (!mbar_wait_cluster(&full_bar[s], (uint32_t)(it / Cfg::STAGES) & 1u, dead, KID_GEMM_LARGEM, 7)) break;
          tc_fence_after_sync();
          const uint32_t a_addr = smem_u32(smem + s * Cfg::STAGE_BYTES);
          const uint64_t da = make_smem_desc(a_addr, 16, 1024, SWZ_128B);
          const uint64_t db = make_smem_desc(a_addr + Cfg::A_BYTES, 16, 1024, SWZ_128B);
#pragma unroll
          for (int k = 0; k < 4; ++k) umma_f16_pair(acc, da + 2 * k, db + 2 * k, p.idesc, (i | k) != 0 ? 1u : 0u);
          umma_commit_pair(&empty_bar[s]);
        }
        if (dead) break;
        umma_commit_pair(&acc_full[buf]);
      }
    }
    __syncwarp();
  } else {
    const int q = warp & 3;
    int u = 0;
    for (int t = pair; t < tiles; t += pairs, ++u) {
      int m_tile, n_tile;
      hook.tile_coords(t, tiles_m, tiles_n, m_tile, n_tile);
      const int buf = u & 1;
      const uint32_t use = (uint32_t)(u >> 1) & 1u;
      if (!mbar_wait_cluster(&acc_full[buf], use, dead, KID_GEMM_LARGEM, 9)) break;
      tc_fence_after_sync();
      largem_epilogue<Cfg::BN, BF16, EXTRA>(p, tmem_base + (uint32_t)(buf * Cfg::BN), 2 * m_tile + rank, n_tile, q, lane, ex);
      tc_fence_before_sync();                          // this warp's TMEM reads are done before the buffer is handed back
      __syncwarp();
      if (lane == 0) mbar_arrive_cluster(mapa_u32(smem_u32(&acc_empty[buf]), 0));
    }
  }
  __syncwarp();
  tc_fence_before_sync();
  __syncthreads();
  cluster_sync_all();                                  // neither CTA's barriers or operands are in use any more
  if (warp == 1) tmem_dealloc_pair(tmem_base, Cfg::TMEM_COLS);
  __syncwarp();
  cluster_sync_all();
}

}  // namespace fb
