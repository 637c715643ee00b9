// 16-bit GEMM body for a few hundred token rows (sm_100a): swap-AB on CTA pairs, one pass over the weights.  Included after gemm_pair.cuh.
//
// Bound: a prompt of a few hundred tokens needs each weight once (HBM) and a few hundred products per weight (tensor core), both about as long; what
// the other kernels lose is tiles.  The small-M kernel pads 129 rows to 256 and loads 48 KB for every 64 of k, the large-M kernels leave a last round of
// tiles nearly empty (333 rows x 28672 features: 336 tiles of 128 x 256 on 148 SMs).  Here a pair's tile is 256 weight rows x all tokens (up to 512
// columns of TMEM, rounded up to 32): a weight tile is loaded once, 16 KB + 64 B per token and SM for every 64 of k.  Where the last round of tiles would leave
// half of the pairs idle it is split over k among them; the splits' fp32 tiles meet in a workspace in the L2, and every split adds up, in the order of the
// splits, and stores its share of the tokens.  (Equal shares of all k blocks, two partial tiles a pair, were slower than whole splits: 4096 x 14336 at 333
// rows 50 against 41 us, the partial tiles' writes.)  Measured figures stand at the rule that chooses this kernel (fb_gemm_mid_pick).
#pragma once
#include "gemm_pair.cuh"

namespace fb {

constexpr int KID_GEMM_MID = 4;

struct MidPlan {
  int nt1, nt2;              // token columns of the two products of a k step (multiples of 32; nt2 may be 0)
  int tok_tiles, row_tiles;  // tiles of nt1 + nt2 tokens, of 256 weight rows
  int full, rest, splits;    // tiles computed whole (round robin over the pairs); the remaining ones, each by `splits` pairs
  int stages;
  uint32_t idesc1, idesc2;
  float* part;               // [rest][splits][2 CTAs][nt][128] partial tiles
  unsigned long long* flags; // [rest][2 CTAs][splits: reader][splits: writer]
  unsigned long long tag;    // what a writer leaves in its flags: another value in every launch; the reader puts 0 back
};

struct MidCfg {
  static constexpr int A_BYTES = 128 * 128;              // 128 weight rows x 64 of k
  static constexpr int GROUPS = 4;                       // epilogue groups of four warps
  static constexpr int CHUNK = 16;                       // tokens that a group takes at a time
  static constexpr int STAGING = CHUNK * 128 * 4;
  static constexpr int MAX_STAGES = 8;
  static constexpr int PIPE_BYTES = 196608;              // 4 stages of 512 tokens, 5 of 352, 8 of 128
  static constexpr int SMEM_BYTES = PIPE_BYTES + GROUPS * STAGING + 512 + 1024;
  static constexpr int THREADS = 64 + GROUPS * 128;
  static constexpr int TMEM_COLS = 512;
};
static_assert(MidCfg::SMEM_BYTES <= 232448, "shared memory of a CTA");

__device__ __forceinline__ void bar_named(int id, int threads) { asm volatile("bar.sync %0, %1;\n" ::"r"(id), "r"(threads) : "memory"); }
__device__ __forceinline__ void st_release_u64(unsigned long long* p, unsigned long long v) {
  asm volatile("st.release.gpu.global.u64 [%0], %1;\n" ::"l"(p), "l"(v) : "memory");
}
__device__ __forceinline__ unsigned long long ld_acquire_u64(const unsigned long long* p) {
  unsigned long long v;
  asm volatile("ld.acquire.gpu.global.u64 %0, [%1];\n" : "=l"(v) : "l"(p) : "memory");
  return v;
}

// Warp 0 loads, warp 1 of the pair's first CTA issues the products, warps 2.. are four epilogue groups of four warps that take turns at 16 tokens.
// Up to 256 tokens there are two accumulators (the epilogue of a tile runs under the products of the next), one beyond.
template <bool BF16>
__device__ __forceinline__ void gemm_mid_device(const CUtensorMap& tmW, const CUtensorMap& tmX1, const CUtensorMap& tmX2, const GemmParams& p, const MidPlan& pl) {
  using Cfg = MidCfg;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  const int nt = pl.nt1 + pl.nt2, nst = pl.stages;
  const int b1_bytes = pl.nt1 * 64, stage_bytes = Cfg::A_BYTES + nt * 64;        // half of the tokens in each CTA, 128 bytes a row
  float* staging = reinterpret_cast<float*>(smem + nst * stage_bytes);           // [groups][16][128]
  uint64_t* full_bar = reinterpret_cast<uint64_t*>(staging + Cfg::GROUPS * Cfg::STAGING / 4);      // the first CTA's are used
  uint64_t* empty_bar = full_bar + Cfg::MAX_STAGES;
  uint64_t* acc_full = empty_bar + Cfg::MAX_STAGES;    // [2]
  uint64_t* acc_empty = acc_full + 2;                  // [2] drained (16 epilogue warps of each CTA; the first CTA's are used)
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(acc_empty + 2);

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int rank = (int)cluster_ctarank(), pair = (int)(blockIdx.x >> 1), pairs = (int)(gridDim.x >> 1);
  const bool two = nt <= 256;                          // two accumulators
  const int whole = pl.full > pair ? (pl.full - pair + pairs - 1) / pairs : 0;      // tiles of this pair, then at most one split of another
  const int r = pl.rest ? pair % pl.rest : 0, split = pl.rest ? pair / pl.rest : 0;
  const bool splits_one = pair < pl.rest * pl.splits;
  const int works = whole + (splits_one ? 1 : 0);
  auto work = [&](int w, int& tile, int& kb0, int& kb1) {
    if (w < whole) { tile = pair + w * pairs; kb0 = 0; kb1 = p.kb_total; return; }
    tile = pl.full + r;
    kb0 = (int)((long long)split * p.kb_total / pl.splits);
    kb1 = (int)((long long)(split + 1) * p.kb_total / pl.splits);
  };
  bool dead = false;
  pdl_launch_dependents();

  if (threadIdx.x == 0) {
    for (int s = 0; s < nst; ++s) { mbar_init(&full_bar[s], 1); mbar_init(&empty_bar[s], 1); }
    for (int b = 0; b < 2; ++b) { mbar_init(&acc_full[b], 1); mbar_init(&acc_empty[b], 8 * Cfg::GROUPS); }
    mbar_init_fence();
    tma_prefetch_desc(&tmW);
    tma_prefetch_desc(&tmX1);
    if (pl.nt2) tma_prefetch_desc(&tmX2);
  }
  if (warp == 1) { tmem_alloc_pair(tmem_slot, Cfg::TMEM_COLS); tmem_relinquish_pair(); }
  tc_fence_before_sync();
  __syncthreads();
  cluster_sync_all();                                  // the other CTA's barriers exist, too
  tc_fence_after_sync();
  const uint32_t tmem_base = *tmem_slot;

  if (warp == 0) {
    if (elect_one()) {
      int it = 0;                                      // k-block counter across all of this pair's work
      const uint64_t pol_w = l2_policy_evict_first(), pol_x = l2_policy_evict_last();
      for (int w = 0; w < works && !dead; ++w) {
        int tile, kb0, kb1;
        work(w, tile, kb0, kb1);
        const int row = (tile / pl.tok_tiles) * 256 + rank * 128, tok = (tile % pl.tok_tiles) * nt;
        // weights do not depend on the kernel before this one: the first ring of them is requested before the dependency wait
        const int pre = w == 0 ? min(nst, kb1 - kb0) : 0;
        for (int i = 0; i < pre; ++i) {
          if (rank == 0) mbar_expect_tx(&full_bar[i], 2 * stage_bytes);
          tma_load_2d_pair_hint(smem + i * stage_bytes, &tmW, mapa_u32(smem_u32(&full_bar[i]), 0), (kb0 + i) * 64, row, pol_w);
        }
        if (w == 0) pdl_wait();
        for (int i = kb0; i < kb1; ++i, ++it) {
          const int s = it % nst;
          uint8_t* a = smem + s * stage_bytes;
          const uint32_t bar = mapa_u32(smem_u32(&full_bar[s]), 0);
          if (it >= pre) {
            if (!mbar_wait(&empty_bar[s], ((uint32_t)(it / nst) & 1u) ^ 1u, dead, KID_GEMM_MID, 1)) break;
            if (rank == 0) mbar_expect_tx(&full_bar[s], 2 * stage_bytes);
            tma_load_2d_pair_hint(a, &tmW, bar, i * 64, row, pol_w);
          }
          tma_load_2d_pair_hint(a + Cfg::A_BYTES, &tmX1, bar, i * 64, tok + rank * (pl.nt1 / 2), pol_x);
          if (pl.nt2) tma_load_2d_pair_hint(a + Cfg::A_BYTES + b1_bytes, &tmX2, bar, i * 64, tok + pl.nt1 + rank * (pl.nt2 / 2), pol_x);
        }
      }
      // the last products' commits have reached this CTA before it may leave
      for (int k = it > nst ? it - nst : 0; k < it; ++k)
        if (!mbar_wait(&empty_bar[k % nst], (uint32_t)(k / nst) & 1u, dead, KID_GEMM_MID, 2)) break;
    }
    __syncwarp();
  } else if (warp == 1) {
    if (rank == 0 && elect_one()) {
      int it = 0;
      for (int w = 0; w < works && !dead; ++w) {
        int tile, kb0, kb1;
        work(w, tile, kb0, kb1);
        const int buf = two ? w & 1 : 0;
        const uint32_t use = (uint32_t)(two ? w >> 1 : w) & 1u;
        if (!mbar_wait_cluster(&acc_empty[buf], use ^ 1u, dead, KID_GEMM_MID, 3)) break;      // first use passes at once
        tc_fence_after_sync();
        const uint32_t acc = tmem_base + (uint32_t)(buf * 256);
        for (int i = kb0; i < kb1; ++i, ++it) {
          const int s = it % nst;
          if (!mbar_wait_cluster(&full_bar[s], (uint32_t)(it / nst) & 1u, dead, KID_GEMM_MID, 4)) break;
          tc_fence_after_sync();
          const uint32_t a_addr = smem_u32(smem + s * stage_bytes);
          const uint64_t da = make_smem_desc(a_addr, 16, 1024, SWZ_128B);
          const uint64_t db1 = make_smem_desc(a_addr + Cfg::A_BYTES, 16, 1024, SWZ_128B);
          const uint64_t db2 = make_smem_desc(a_addr + Cfg::A_BYTES + b1_bytes, 16, 1024, SWZ_128B);
#pragma unroll
          for (int k = 0; k < 4; ++k) {
            umma_f16_pair(acc, da + 2 * k, db1 + 2 * k, pl.idesc1, (i != kb0 || k) ? 1u : 0u);
            if (pl.nt2) umma_f16_pair(acc + (uint32_t)pl.nt1, da + 2 * k, db2 + 2 * k, pl.idesc2, (i != kb0 || k) ? 1u : 0u);
          }
          umma_commit_pair(&empty_bar[s]);
        }
        if (dead) break;
        umma_commit_pair(&acc_full[buf]);
      }
    }
    __syncwarp();
  } else {
    const int q = warp & 3, group = (warp - 2) >> 2, gtid = threadIdx.x - 64 - group * 128, etid = threadIdx.x - 64;
    constexpr int ALL = Cfg::GROUPS * 128;
    const int n_local = q * 32 + lane;
    const bool swiglu = (p.flags & GEMM_SWIGLU) != 0;
    const int vec = swiglu ? 16 : 32;                  // float4 results of a token in this CTA's 128 weight rows
    float* P = staging + group * (Cfg::STAGING / 4);
    const size_t tile_floats = (size_t)nt * 128;
    pdl_wait();
    for (int w = 0; w < works; ++w) {
      int tile, kb0, kb1;
      work(w, tile, kb0, kb1);
      const bool whole_tile = w < whole;
      const int buf = two ? w & 1 : 0;
      const uint32_t use = (uint32_t)(two ? w >> 1 : w) & 1u;
      const int n_tile = (tile / pl.tok_tiles) * 2 + rank, tok = (tile % pl.tok_tiles) * nt;
      const int valid = min(nt, p.M - tok);
      const uint32_t acc = tmem_base + (uint32_t)(buf * 256) + ((uint32_t)(q * 32) << 16);
      mbar_wait_cluster(&acc_full[buf], use, dead, KID_GEMM_MID, 5);      // (on expiry: reported; the barriers below are met all the same)
      tc_fence_after_sync();
      float* mine = whole_tile ? nullptr : pl.part + ((size_t)(r * pl.splits + split) * 2 + rank) * tile_floats;
      for (int c = group * Cfg::CHUNK; c < valid; c += Cfg::GROUPS * Cfg::CHUNK) {
        uint32_t t[Cfg::CHUNK];
        __syncwarp();
        tmem_ld_32x32b_x16(acc + (uint32_t)c, t);
        tmem_ld_wait();
        if (!whole_tile) {
#pragma unroll
          for (int j = 0; j < Cfg::CHUNK; ++j)
            if (c + j < valid) mine[(size_t)(c + j) * 128 + n_local] = __uint_as_float(t[j]);
          continue;
        }
        bar_named(1 + group, 128);                     // the group has stored the tokens staged before
#pragma unroll
        for (int j = 0; j < Cfg::CHUNK; ++j) P[j * 128 + n_local] = __uint_as_float(t[j]);
        bar_named(1 + group, 128);
        const int items = min(Cfg::CHUNK, valid - c) * vec;
        for (int e = gtid; e < items; e += 128) {
          const int j = e / vec, n = (e - j * vec) * 4;
          const float4 v = *reinterpret_cast<const float4*>(P + j * 128 + n);
          float4 u = make_float4(0.f, 0.f, 0.f, 0.f);
          if (swiglu) u = *reinterpret_cast<const float4*>(P + j * 128 + 64 + n);
          smallm_finish<BF16>(p, tok + c + j, n_tile, n, v, u);
        }
      }
      tc_fence_before_sync();                          // this warp's TMEM reads are done before the accumulator is handed back
      __syncwarp();
      if (lane == 0) mbar_arrive_cluster(mapa_u32(smem_u32(&acc_empty[buf]), 0));
    }
    // a split tile: every split adds up, in the order of the splits, and stores its share of the tokens
    if (splits_one) {
      const int n = pl.splits;
      unsigned long long* flags = pl.flags + (size_t)(r * 2 + rank) * n * n;
      __threadfence();
      bar_named(1 + Cfg::GROUPS, ALL);
      if (etid < n) {
        st_release_u64(flags + etid * n + split, pl.tag);
        unsigned long long* f = flags + split * n + etid;
        const uint64_t t0 = globaltimer_ns();
        while (!dead && ld_acquire_u64(f) != pl.tag) {
          if (globaltimer_ns() - t0 > FB_WAIT_LIMIT_NS) { report_error(ERR_WAIT_TIMEOUT, KID_GEMM_MID, 6); dead = true; }
        }
        *f = 0ull;                                     // one writer, one reader: the next launch finds no tag
      }
      bar_named(1 + Cfg::GROUPS, ALL);
      const int tile = pl.full + r, n_tile = (tile / pl.tok_tiles) * 2 + rank, tok = (tile % pl.tok_tiles) * nt;
      const int valid = max(0, min(nt, p.M - tok));
      const int t0 = split * valid / n, t1 = (split + 1) * valid / n;
      const float* src0 = pl.part + ((size_t)r * n * 2 + rank) * tile_floats;
      const int items = (t1 - t0) * vec;
      for (int e0 = etid; e0 < items; e0 += 2 * ALL) {
        float4 v[2], u[2];
        int at[2];
#pragma unroll
        for (int k = 0; k < 2; ++k) {
          const int e = min(e0 + k * ALL, items - 1), j = e / vec;
          at[k] = (t0 + j) * 128 + (e - j * vec) * 4;
          v[k] = __ldcg(reinterpret_cast<const float4*>(src0 + at[k]));
          u[k] = swiglu ? __ldcg(reinterpret_cast<const float4*>(src0 + at[k] + 64)) : make_float4(0.f, 0.f, 0.f, 0.f);
        }
#pragma unroll 3
        for (int s = 1; s < n; ++s) {
          const float* src = src0 + (size_t)s * 2 * tile_floats;
#pragma unroll
          for (int k = 0; k < 2; ++k) {
            const float4 a = __ldcg(reinterpret_cast<const float4*>(src + at[k]));
            v[k].x += a.x; v[k].y += a.y; v[k].z += a.z; v[k].w += a.w;
            if (swiglu) {
              const float4 b = __ldcg(reinterpret_cast<const float4*>(src + at[k] + 64));
              u[k].x += b.x; u[k].y += b.y; u[k].z += b.z; u[k].w += b.w;
            }
          }
        }
#pragma unroll
        for (int k = 0; k < 2; ++k)
          if (e0 + k * ALL < items) smallm_finish<BF16>(p, tok + (at[k] >> 7), n_tile, at[k] & 127, v[k], u[k]);
      }
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
