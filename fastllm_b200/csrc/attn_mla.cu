// Absorbed multi-head latent attention (MLA) decode for sm_100a over a paged latent cache.
//
// Cache entry per token: up to 512 compressed-KV dims, optionally followed by 64 rotary key dims (16 bit); page length 128.
// Query per head: q_nope already multiplied by W_UK, followed by the rotated q_pe where the model has one.
//     S^T[128 tokens x N heads] = Lat_page[128 x dq] * Q^T              column tiles of 64, K-major, SW128 (DeepSeek: 9)
//     O^T[dv dims    x N heads] = Lat_page[:, :dv]^T * P^T              row blocks of 128 dims, A read MN-major (DeepSeek: 4)
// With a sliding window the plan lists the pages the window touches and the softmax masks the keys before it.  Values behind a request's
// end are cleared in shared memory before the second product (P = 0 alone would pass NaN and infinity on).
// The latent page is both K and V: it is loaded ONCE into 16 KB tiles (one CTA per SM, 144 KB of page + 36 KB of queries).  Its halves of 64 tokens
// are two chains of load, scores, softmax (two warps each) and second product, with barriers, maxima and accumulators of their own: one half's loads are
// on their way while the other computes.  A work item is a run of consecutive pages of one request and one group of <= 32 heads; a half keeps (max, sum)
// per head across the run, four warps rescale its accumulator when a maximum moves, and the halves are added up in the item's epilogue, so
// the un-normalised partial output is written once per item.  A combine kernel merges the items of a request.
// Bound: a half's chain (load 3 us of about 5; 72 KB of each SM are under way on the mean).  16 heads, 512 + 64, with the combine, us, one chain a page and
// pages in thirds of a CTA's share before: 32 requests of 2560 tokens 51 -> 41, of 1280 35 -> 29, of 5120 73 -> 72, 148 of 640 52 -> 44, 148 of 1280 73 -> 71.
//
// Reference: MergeMLAPaged / FastllmCudaMLAPaged -> FlashInfer BatchMLAPagedAttention<512, 64>, one request per call
// (src/devices/cuda/attention/fastllm-attention.cu:3619-3727); the absorb GEMMs stay outside (src/models/deepseekv2.cpp:283-697).
#include "ptx.cuh"
#include "launch.h"
#include "tmap.h"

FB_DEFINE_ERROR_API(attn_mla)

namespace fb {

constexpr int KID_MLA = 12;
constexpr int ML_PAGE = 128;
constexpr int ML_MAX_TILES = 9;                   // 64-column tiles of the latent page (the last one may be partly filled)
constexpr int ML_MAX_LORA = 512;
constexpr int ML_N = 32;                          // MMA N: heads per item (padded)
constexpr int ML_TILE_BYTES = ML_PAGE * 64 * 2;   // 16 KB
constexpr int ML_QTILE_BYTES = ML_N * 64 * 2;     // 4 KB
constexpr int ML_P_BYTES = ML_N * ML_PAGE * 2;    // 8 KB
constexpr int ml_smem(int tiles) { return tiles * (ML_TILE_BYTES + ML_QTILE_BYTES) + ML_P_BYTES + 2048 /*barriers, reductions*/ + 1024 /*align*/; }
constexpr int ML_HALF_BYTES = ML_TILE_BYTES / 2;   // 64 tokens
// tensor memory: S of the page halves [0,32), [32,64); O of half h from 64 + h o_cols, 32 columns a block of 128 dims
__host__ __device__ constexpr int ml_tmem(int o_cols) { return 64 + 2 * o_cols <= 256 ? 256 : 512; }
constexpr int ML_THREADS = 352;                   // loads, scores, two warps a half's softmax, four that rescale accumulators, second products

struct MlaParams {
  const int* work;          // [n_work][4] = (request, first page, page count, head group)
  const int* n_work;
  const int* page_table; int max_pages;
  const int* seq_lens;
  float* part_o;            // [n_work_cap][ML_N][512]
  float* part_ml;           // [n_work_cap][ML_N][2]
  int H, B, max_items;
  int tiles, vtiles;        // 64-column tiles of a latent row, of its value part
  int o_stride;             // floats per head in part_o: the value width rounded up to 128
  int o_cols;               // columns of a half's O
  int window;               // keys a query sees (0: all)
  float scale_log2;
  uint32_t idesc_s, idesc_o;
};

// ---- plan: one item per (request, run of pages, head group); also the per-request item ranges for the combine ----
// item_range: [B][2] = (first item, item count) of the request's head group 0; groups follow each other per run.
__global__ void mla_plan_kernel(const int* __restrict__ seq_lens, int B, int n_groups, int ctas, int window, int* __restrict__ work,
                                int* __restrict__ n_work, int* __restrict__ item_range, int max_items) {
  __shared__ int offs[1025];
  __shared__ int s_ppi, s_items[4];
  pdl_launch_dependents();
  pdl_wait();
  const int t = threadIdx.x;
  int np = 0, page0 = 0;                 // pages the request's query sees: [page0, page0 + np)
  if (t < B) {
    const int seq = seq_lens[t];
    if (window > 0 && seq > window) page0 = (seq - window) / ML_PAGE;
    np = (seq + ML_PAGE - 1) / ML_PAGE - page0;
  }
  offs[t + 1] = np;
  if (t < 4) s_items[t] = 0;
  if (t == 0) offs[0] = 0;
  __syncthreads();
  for (int d = 1; d < blockDim.x; d <<= 1) {
    int v = 0;
    if (t >= d) v = offs[t + 1 - d];
    __syncthreads();
    if (t >= d) offs[t + 1] += v;
    __syncthreads();
  }
  // Pages an item: one, where that leaves no CTA a second item; else rounds of the CTAs over the items times an item's pages and what it costs beside them
  // (half a page), least of four lengths, two items a CTA to one (32 requests of 20 pages, 148 CTAs: 5 pages in one round, not 3 in two).
  const int total = offs[blockDim.x] * n_groups, fine = (total + 2 * ctas - 1) / (2 * ctas), whole = (total + ctas - 1) / ctas;
  if (whole <= 1) {
    if (t == 0) s_ppi = 1;
  } else {
    auto pages = [&](int c) { return c < 2 ? fine + c : whole + (c - 2) * (1 + whole / 8); };
#pragma unroll
    for (int c = 0; c < 4; ++c) {
      const int n = __reduce_add_sync(0xffffffffu, (np + pages(c) - 1) / pages(c));
      if ((t & 31) == 0 && n > 0) atomicAdd(&s_items[c], n);
    }
    __syncthreads();
    if (t == 0) {
      int best = 1, cost = 0x7fffffff;
      for (int c = 0; c < 4; ++c) {
        const int k = (s_items[c] * n_groups + ctas - 1) / ctas * (2 * pages(c) + 1);
        if (k < cost) { cost = k; best = pages(c); }
      }
      s_ppi = best;
    }
  }
  __syncthreads();
  const int ppi = s_ppi;
  // runs per request, exclusive scan over requests (reuse offs)
  const int runs = t < B ? (np + ppi - 1) / ppi : 0;
  __syncthreads();
  offs[t + 1] = runs;
  if (t == 0) offs[0] = 0;
  __syncthreads();
  for (int d = 1; d < blockDim.x; d <<= 1) {
    int v = 0;
    if (t >= d) v = offs[t + 1 - d];
    __syncthreads();
    if (t >= d) offs[t + 1] += v;
    __syncthreads();
  }
  if (t < B) {
    const int first = offs[t] * n_groups;
    item_range[2 * t] = first;
    item_range[2 * t + 1] = runs;
    for (int r = 0; r < runs; ++r)
      for (int g = 0; g < n_groups; ++g) {
        const int it = first + r * n_groups + g;
        if (it < max_items) {
          work[4 * it] = t;
          work[4 * it + 1] = page0 + r * ppi;
          work[4 * it + 2] = (np - r * ppi) < ppi ? (np - r * ppi) : ppi;
          work[4 * it + 3] = g;
        }
      }
  }
  if (t == 0) { const int total = offs[blockDim.x] * n_groups; *n_work = total < max_items ? total : max_items; }
}

// Reads and validates one work item; every warp role uses this, so a rejected item is rejected by all of them alike.
__device__ __forceinline__ bool mla_item(const MlaParams& p, int w, int& b, int& p0, int& cnt, int& hg) {
  b = p.work[4 * w]; p0 = p.work[4 * w + 1]; cnt = p.work[4 * w + 2]; hg = p.work[4 * w + 3];
  if ((unsigned)b >= (unsigned)p.B || p0 < 0 || cnt < 0 || p0 + cnt > p.max_pages || hg < 0 || hg * ML_N >= p.H) {
    b = 0; p0 = 0; cnt = 0; hg = 0;
    return false;
  }
  return true;
}

// N numbers of each lane (N a power of two, at most 32) to the maximum or the sum of each over the warp: a lane gives half of its numbers away at every
// step, so that N - 1 + log2(32 / N) exchanges do.  Returns that of number ml_reduced<N>(lane).
template <int N, bool MAX>
__device__ __forceinline__ float ml_reduce(float (&v)[N], int lane) {
  auto join = [](float a, float b) { return MAX ? fmaxf(a, b) : a + b; };
  int n = N;
#pragma unroll
  for (int mask = 16; mask > 0; mask >>= 1) {
    if (n > 1) {
      n >>= 1;
      const bool up = (lane & mask) != 0;
#pragma unroll
      for (int i = 0; i < N / 2; ++i) {
        if (i >= n) break;
        const float give = up ? v[i] : v[i + n], keep = up ? v[i + n] : v[i];
        v[i] = join(keep, __shfl_xor_sync(0xffffffffu, give, mask));
      }
    } else {
      v[0] = join(v[0], __shfl_xor_sync(0xffffffffu, v[0], mask));
    }
  }
  return v[0];
}
template <int N>
__device__ __forceinline__ int ml_reduced(int lane) { return lane >> (N == 32 ? 0 : 1); }

template <bool BF16, int GP>
__global__ void __launch_bounds__(ML_THREADS, 1)
mla_decode_kernel(const __grid_constant__ CUtensorMap tmLat, const __grid_constant__ CUtensorMap tmQ, const MlaParams p) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  const int ML_TILES = p.tiles;
  uint8_t* lat = smem;                                         // tiles [128 tokens x 64 cols]
  uint8_t* qs = lat + ML_TILES * ML_TILE_BYTES;                // tiles [32 heads x 64 cols]
  uint8_t* p_smem = qs + ML_TILES * ML_QTILE_BYTES;
  uint64_t* bars = reinterpret_cast<uint64_t*>(p_smem + ML_P_BYTES);
  uint64_t* full = bars;                         // [9][2] half of a tile landed
  uint64_t* empty = full + 2 * ML_MAX_TILES;     // [9][2] consumed by its last MMA
  uint64_t* s_full = empty + 2 * ML_MAX_TILES;   // [2]
  uint64_t* p_ready = s_full + 2;                // [2]
  uint64_t* o_full = p_ready + 2;                // [2]
  uint64_t* o_fit = o_full + 2;                  // [2] O is in units of the step's maxima
  uint64_t* q_full = o_fit + 2;
  uint64_t* q_empty = q_full + 1;
  uint64_t* o_read = q_full + 2;                 // epilogue has read O of the finished item
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(q_full + 4);
  float* red_max = reinterpret_cast<float*>(tmem_slot + 4);    // [4 warps][32]
  float* red_sum = red_max + 128;                                // [4 warps][32]
  float* facs = red_sum + 128;                                   // [2 halves][32] factors of a rescaling; after an item: weights of the halves
  int* grown = reinterpret_cast<int*>(facs + 64);                // [2]

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  bool dead = false;
  const int o_cols = p.o_cols;
  if (warp == 0) {                               // a barrier a lane and turn
    constexpr int BARS = 4 * ML_MAX_TILES + 11;
    for (int i = lane; i < BARS; i += 32) {
      const int k = i - 4 * ML_MAX_TILES;        // s_full, p_ready, o_full, o_fit (two each), q_full, q_empty, o_read
      mbar_init(&bars[i], k == 2 || k == 3 ? 64 : k == 6 || k == 7 || k == 10 ? 128 : 1);
    }
    mbar_init_fence();
    if (lane == 0) { tma_prefetch_desc(&tmLat); tma_prefetch_desc(&tmQ); }
  }
  if (warp == 1) { tmem_alloc(tmem_slot, ml_tmem(o_cols)); tmem_relinquish(); }
  tc_fence_before_sync();
  __syncthreads();
  tc_fence_after_sync();
  const uint32_t tmem_s = *tmem_slot;
  const uint32_t tmem_o = tmem_s + 64;
  pdl_launch_dependents();                       // (this CTA has its tensor memory: a later kernel's cannot take it first)
  pdl_wait();
  int n_items = *p.n_work;
  if (n_items < 0) n_items = 0;
  if (n_items > p.max_items) n_items = p.max_items;

  if (warp == 0) {
    if (elect_one()) {
      int pi = 0, ii = 0;                  // CTA-local page and item counters (barrier phases)
      for (int w = blockIdx.x; w < n_items; w += gridDim.x, ++ii) {
        int b, p0, cnt, hg;
        if (!mla_item(p, w, b, p0, cnt, hg)) report_error(ERR_BAD_ARG, KID_MLA, 20);
        if (!mbar_wait(q_empty, ((uint32_t)ii & 1u) ^ 1u, dead, KID_MLA, 1)) break;
        mbar_expect_tx(q_full, ML_TILES * ML_QTILE_BYTES);
        for (int j = 0; j < ML_TILES; ++j) tma_load_2d(qs + j * ML_QTILE_BYTES, &tmQ, q_full, j * 64, b * p.H + hg * ML_N);
        for (int i = 0; i < cnt; ++i, ++pi) {
          const int page = p.page_table[(size_t)b * p.max_pages + p0 + i];
          for (int jh = 0; jh < 2 * ML_TILES && !dead; ++jh) {
            const int h = jh >= ML_TILES ? 1 : 0, j = jh - h * ML_TILES;
            if (!mbar_wait(&empty[2 * j + h], ((uint32_t)pi & 1u) ^ 1u, dead, KID_MLA, 2)) break;
            mbar_expect_tx(&full[2 * j + h], ML_HALF_BYTES);
            tma_load_2d(lat + j * ML_TILE_BYTES + h * ML_HALF_BYTES, &tmLat, &full[2 * j + h], j * 64, page * ML_PAGE + h * 64);
          }
          if (dead) break;
        }
        if (dead) break;
      }
    }
    __syncwarp();
  } else if (warp == 1) {
    if (elect_one()) {
      int pi = 0, ii = 0;
      for (int w = blockIdx.x; w < n_items; w += gridDim.x, ++ii) {
        int b, p0, cnt, hg;
        mla_item(p, w, b, p0, cnt, hg);
        if (!mbar_wait(q_full, (uint32_t)ii & 1u, dead, KID_MLA, 3)) break;
        if (cnt == 0) umma_commit(q_empty);                  // rejected item: hand the query buffer straight back
        // S^T of half u & 1 of page u / 2: the product takes all 128 rows of the tiles, those of the other half (whatever is there, or on its way)
        // give rows of S that nothing reads
        for (int u = 0; u < 2 * cnt && !dead; ++u) {
          const int h = u & 1, pg = pi + (u >> 1);
          const uint32_t ph = (uint32_t)pg & 1u;
          if (pg > 0 && !mbar_wait(&p_ready[h], ph ^ 1u, dead, KID_MLA, 15)) break;      // this half's last scores have been read
          for (int j = 0; j < ML_TILES; ++j) {
            if (!mbar_wait(&full[2 * j + h], ph, dead, KID_MLA, 4)) break;
            tc_fence_after_sync();
            const uint32_t a0 = smem_u32(lat + j * ML_TILE_BYTES), b0 = smem_u32(qs + j * ML_QTILE_BYTES);
#pragma unroll
            for (int k = 0; k < 4; ++k)
              umma_f16(tmem_s + h * ML_N, make_smem_desc(a0 + k * 32, 16, 1024, SWZ_128B), make_smem_desc(b0 + k * 32, 16, 1024, SWZ_128B),
                       p.idesc_s, (j | k) != 0 ? 1u : 0u);
          }
          if (dead) break;
          umma_commit(&s_full[h]);
          for (int j = p.vtiles; j < ML_TILES; ++j) umma_commit(&empty[2 * j + h]);     // rotary tiles are not part of V
          if (u == 2 * cnt - 1) umma_commit(q_empty);        // queries are free once the item's last S product is done
        }
        pi += cnt;
        if (dead) break;
      }
    }
    __syncwarp();
  } else if (warp == 10) {
    // (a warp of its own: a half's second products do not stand behind the loads that the other half's scores wait for)
    if (elect_one()) {
      int pi = 0, ii = 0;
      for (int w = blockIdx.x; w < n_items && !dead; w += gridDim.x, ++ii) {
        int b, p0, cnt, hg;
        mla_item(p, w, b, p0, cnt, hg);
        for (int u = 0; u < 2 * cnt; ++u) {
          const int h = u & 1;
          const uint32_t ph = (uint32_t)(pi + (u >> 1)) & 1u;
          if (!mbar_wait(&p_ready[h], ph, dead, KID_MLA, 5) || !mbar_wait(&o_fit[h], ph, dead, KID_MLA, 11)) break;
          if (u < 2 && ii > 0 && !mbar_wait(o_read, ((uint32_t)ii & 1u) ^ 1u, dead, KID_MLA, 6)) break;
          tc_fence_after_sync();
          // ---- O^T[blk] (+)= V_blk^T * P^T, V_blk = latent columns [128 blk, +128) = tiles 2 blk, 2 blk + 1 ----
          // (a last half block reads past its one tile; those rows of O^T are never stored)
          for (int blk = 0; 2 * blk < p.vtiles; ++blk) {
            const uint32_t vb = smem_u32(lat + 2 * blk * ML_TILE_BYTES + h * ML_HALF_BYTES);
#pragma unroll
            for (int k = 0; k < 4; ++k)
              umma_f16(tmem_o + h * o_cols + blk * ML_N, make_smem_desc(vb + k * 2048, ML_TILE_BYTES, 1024, SWZ_128B),
                       make_smem_desc(smem_u32(p_smem) + (4 * h + k) * 1024, 512, 128, SWZ_NONE), p.idesc_o, ((u >> 1) | k) != 0 ? 1u : 0u);
            umma_commit(&empty[4 * blk + h]);
            if (2 * blk + 1 < p.vtiles) umma_commit(&empty[4 * blk + 2 + h]);
          }
          umma_commit(&o_full[h]);
        }
        pi += cnt;
      }
    }
    __syncwarp();
  } else if (warp >= 6) {
    // O of a half whose maxima have grown, into their new units (its rows are dims, which the half's own two warps hold only a part of)
    const uint32_t lane_off = (uint32_t)((warp & 3) * 32) << 16;
    int pi = 0;
    for (int w = blockIdx.x; w < n_items; w += gridDim.x) {
      int b, p0, cnt, hg;
      mla_item(p, w, b, p0, cnt, hg);
      for (int u = 0; u < 2 * cnt; ++u) {
        const int half = u & 1;
        const uint32_t ph = (uint32_t)(pi + (u >> 1)) & 1u;
        mbar_wait(&p_ready[half], ph, dead, KID_MLA, 12);
        if (u >= 2 && grown[half] != 0) {
          mbar_wait(&o_full[half], ph ^ 1u, dead, KID_MLA, 13);
          __syncwarp();
          tc_fence_after_sync();
#pragma unroll 1
          for (int blk = 0; 2 * blk < p.vtiles; ++blk) {
            uint32_t o[32];
            tmem_ld_32x32b_x32(tmem_o + half * o_cols + blk * ML_N + lane_off, o);
            tmem_ld_wait();
#pragma unroll
            for (int h = 0; h < GP; ++h) o[h] = __float_as_uint(__uint_as_float(o[h]) * facs[half * 32 + h]);
            tmem_st_32x32b_x32(tmem_o + half * o_cols + blk * ML_N + lane_off, o);
          }
          tmem_st_wait();
          tc_fence_before_sync();
        }
        mbar_arrive(&o_fit[half]);
      }
      pi += cnt;
    }
  } else {
    const int q = warp & 3, half = q >> 1;         // of the page
    const int t = q * 32 + lane;                   // token within the page (softmax) / dim within a 128-block (epilogue)
    if (GP < ML_N) {                               // heads that are not there never get a weight
      uint8_t* pb = p_smem + (t >> 3) * (ML_N / 8) * 128 + (t & 7) * 2;
#pragma unroll
      for (int h = GP; h < ML_N; ++h) *reinterpret_cast<uint16_t*>(pb + (h >> 3) * 128 + (h & 7) * 16) = 0;
    }
    const uint32_t lane_off = (uint32_t)(q * 32) << 16;
    int pi = 0, ii = 0;
    for (int w = blockIdx.x; w < n_items; w += gridDim.x, ++ii) {
      int b, p0, cnt, hg;
      mla_item(p, w, b, p0, cnt, hg);
      const int seq = p.seq_lens[b];
      const int first_key = (p.window > 0 && seq > p.window) ? seq - p.window : 0;
      const int nh = min(GP, p.H - hg * ML_N);     // real heads in this group
      float m_run[GP], l_part[GP];
#pragma unroll
      for (int h = 0; h < GP; ++h) { m_run[h] = -INFINITY; l_part[h] = 0.f; }
      for (int i = 0; i < cnt; ++i, ++pi) {
        const uint32_t ph = (uint32_t)pi & 1u;
        const int key = (p0 + i) * ML_PAGE + t;
        const bool valid = key < seq && key >= first_key;
        mbar_wait(&s_full[half], ph, dead, KID_MLA, 7);
        __syncwarp();
        tc_fence_after_sync();
        uint32_t r[32];
        tmem_ld_32x32b_x32(tmem_s + half * ML_N + lane_off, r);
        tmem_ld_wait();
        float sv[GP];
#pragma unroll
        for (int h = 0; h < GP; ++h) sv[h] = (valid && h < nh) ? __uint_as_float(r[h]) * p.scale_log2 : -INFINITY;
        // a head's maximum over the 64 keys
        {
          float v[GP];
#pragma unroll
          for (int h = 0; h < GP; ++h) v[h] = sv[h];
          red_max[q * 32 + ml_reduced<GP>(lane)] = ml_reduce<GP, true>(v, lane);      // (GP 16: two lanes, the same number)
        }
        asm volatile("bar.sync %0, 64;\n" ::"r"(2 + half) : "memory");
        float fac[GP];
        bool moved = false;
#pragma unroll
        for (int h = 0; h < GP; ++h) {
          const float4 a = *reinterpret_cast<const float4*>(red_max + half * 64 + (h & ~3)), c = *reinterpret_cast<const float4*>(red_max + half * 64 + 32 + (h & ~3));
          const float mn = fmaxf(m_run[h], (h & 3) == 0 ? fmaxf(a.x, c.x) : (h & 3) == 1 ? fmaxf(a.y, c.y) : (h & 3) == 2 ? fmaxf(a.z, c.z) : fmaxf(a.w, c.w));
          fac[h] = 1.f;
          if (m_run[h] == -INFINITY) m_run[h] = mn;           // (nothing in O yet but zeros)
          else if (mn > m_run[h]) { fac[h] = exp2f(m_run[h] - mn); moved = true; m_run[h] = mn; }
        }
        if (i > 0) {
          // the product of this half's last step must be complete before P is overwritten
          mbar_wait(&o_full[half], ph ^ 1u, dead, KID_MLA, 8);
          tc_fence_after_sync();
        }
        if (q == 2 * half && lane == 0) {
          grown[half] = moved ? 1 : 0;                        // same decision in every thread: the maxima are the half's
          if (moved) {
#pragma unroll
            for (int h = 0; h < GP; ++h) facs[half * 32 + h] = fac[h];
          }
        }
        // P^T[n][t], K-major core matrices: ((t/8) * (N/8) + n/8) * 128 + (n%8) * 16 + (t%8) * 2 bytes
        uint8_t* pb = p_smem + (t >> 3) * (ML_N / 8) * 128 + (t & 7) * 2;
#pragma unroll
        for (int h = 0; h < GP; ++h) {
          float pv = 0.f;
          if (h < nh && valid) pv = exp2f(sv[h] - m_run[h]);
          const uint16_t bits = BF16 ? __bfloat16_as_ushort(__float2bfloat16_rn(pv)) : __half_as_ushort(__float2half_rn(pv));
          *reinterpret_cast<uint16_t*>(pb + (h >> 3) * 128 + (h & 7) * 16) = bits;
          const float seen = BF16 ? __bfloat162float(__ushort_as_bfloat16(bits)) : __half2float(__ushort_as_half(bits));
          l_part[h] = l_part[h] * fac[h] + seen;
        }
        if (key >= seq) {
          // slots behind the request's end have no weight, but what an earlier owner left there may be no number: their values count as zeros.
          // (The half's scores are made, so every tile has landed, and none is refilled before its product below.)
#pragma unroll 1
          for (int j = 0; j < p.vtiles; ++j) {
            mbar_wait(&full[2 * j + half], ph, dead, KID_MLA, 10);
            uint4* vrow = reinterpret_cast<uint4*>(lat + j * ML_TILE_BYTES + t * 128);
#pragma unroll
            for (int e = 0; e < 8; ++e) vrow[(e + t) & 7] = make_uint4(0u, 0u, 0u, 0u);      // (a warp's rows share banks)
          }
        }
        fence_proxy_async_smem();
        tc_fence_before_sync();
        mbar_arrive(&p_ready[half]);
      }
      // ---- item epilogue: the halves' sums in the units of the larger maximum ----
      if (cnt > 0) {
        mbar_wait(&o_full[0], (uint32_t)(pi - 1) & 1u, dead, KID_MLA, 9);
        mbar_wait(&o_full[1], (uint32_t)(pi - 1) & 1u, dead, KID_MLA, 14);
        __syncwarp();
        tc_fence_after_sync();
        red_sum[q * 32 + ml_reduced<GP>(lane)] = ml_reduce<GP, false>(l_part, lane);
#pragma unroll
        for (int h = 0; h < GP; ++h)
          if (lane == 0) red_max[q * 32 + h] = m_run[h];
      }
      asm volatile("bar.sync 1, 128;\n" ::: "memory");
      if (cnt > 0 && t < nh) {
        const float m0 = red_max[t], m1 = red_max[64 + t], m = fmaxf(m0, m1);
        const float f0 = m0 == -INFINITY ? 0.f : exp2f(m0 - m), f1 = m1 == -INFINITY ? 0.f : exp2f(m1 - m);
        facs[t] = f0;
        facs[32 + t] = f1;
        p.part_ml[((size_t)w * ML_N + t) * 2] = m;
        p.part_ml[((size_t)w * ML_N + t) * 2 + 1] = (red_sum[t] + red_sum[32 + t]) * f0 + (red_sum[64 + t] + red_sum[96 + t]) * f1;
      }
      asm volatile("bar.sync 1, 128;\n" ::: "memory");
      if (cnt > 0) {
        float* po = p.part_o + (size_t)w * ML_N * p.o_stride;
#pragma unroll 1
        for (int blk = 0; 2 * blk < p.vtiles; ++blk) {
          uint32_t o[32], o1[32];
          tmem_ld_32x32b_x32(tmem_o + blk * ML_N + lane_off, o);
          tmem_ld_32x32b_x32(tmem_o + o_cols + blk * ML_N + lane_off, o1);
          tmem_ld_wait();
#pragma unroll
          for (int h = 0; h < GP; ++h)
            if (h < nh) po[(size_t)h * p.o_stride + blk * 128 + t] = __uint_as_float(o[h]) * facs[h] + __uint_as_float(o1[h]) * facs[32 + h];
        }
        tc_fence_before_sync();
      }
      mbar_arrive(o_read);
      asm volatile("bar.sync 1, 128;\n" ::: "memory");        // the factors have been read
    }
  }
  tc_fence_before_sync();
  __syncthreads();
  if (warp == 1) tmem_dealloc(tmem_s, ml_tmem(o_cols));
}

// one CTA per (request, head): merges the request's items of that head's group; 128 threads x 4 dims per pass
template <bool BF16>
__global__ void mla_combine_kernel(const float* __restrict__ part_o, const float* __restrict__ part_ml, const int* __restrict__ item_range,
                                   uint16_t* __restrict__ out, int H, int n_groups, int dv, int o_stride, const float* __restrict__ head_gate) {
  pdl_launch_dependents();
  pdl_wait();
  const int b = blockIdx.x, h = blockIdx.y, t = threadIdx.x;
  const int g = h / ML_N, hl = h - g * ML_N;
  const int first = item_range[2 * b], runs = item_range[2 * b + 1];
  float M = -INFINITY;
  for (int r = 0; r < runs; ++r) M = fmaxf(M, part_ml[((size_t)(first + r * n_groups + g) * ML_N + hl) * 2]);
  for (int d = t * 4; d < dv; d += 512) {
    float L = 0.f;
    float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
    for (int r = 0; r < runs; ++r) {
      const size_t it = (size_t)(first + r * n_groups + g);
      const float wgt = exp2f(part_ml[(it * ML_N + hl) * 2] - M);
      L += part_ml[(it * ML_N + hl) * 2 + 1] * wgt;
      const float4 o = *reinterpret_cast<const float4*>(&part_o[(it * ML_N + hl) * o_stride + d]);
      acc.x += o.x * wgt; acc.y += o.y * wgt; acc.z += o.z * wgt; acc.w += o.w * wgt;
    }
    float inv = L > 0.f ? 1.0f / L : 0.f;
    if (head_gate != nullptr) inv *= 1.0f / (1.0f + __expf(-head_gate[(size_t)b * H + h]));
    uint2 pk;
    pk.x = pack_16<BF16>(acc.x * inv, acc.y * inv);
    pk.y = pack_16<BF16>(acc.z * inv, acc.w * inv);
    *reinterpret_cast<uint2*>(&out[((size_t)b * H + h) * dv + d]) = pk;
  }
}

}  // namespace fb

using namespace fb;

// q: [B, H, dq] (q_lat | rotary part), lat_pool: [num_slots, dq], out: [B, H, dv]; all 16-bit (dtype 0 = fp16, 1 = bf16).  dv <= dq
// columns of a latent row are its values; dq, dv multiples of 8, dv of 64 when rotary columns follow.  window > 0: the query (the
// request's last token) sees the last `window` tokens only.  head_gate (null: none): fp32 logits [B, H] of a sigmoid gate per head.  Scratch: work [4 * max_items] ints, n_work [1], item_range [2 * B],
// part_o [max_items * 32 * roundup(dv, 128)] floats, part_ml [max_items * 32 * 2] floats, with max_items >= fb_mla_max_items(B, H).
extern "C" int fb_mla_max_items(int B, int H) {
  static int sm_count = 0;
  if (sm_count == 0) {
    int dev = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sm_count, cudaDevAttrMultiProcessorCount, dev);
  }
  // pages per item = ceil(total * groups / target), so the items are at most target + one short run per (request, group)
  return 2 * sm_count + B * ((H + ML_N - 1) / ML_N);
}

extern "C" int fb_mla_decode(const void* q, const void* lat_pool, void* out, const int* page_table, const int* seq_lens, int* work,
                             int* n_work, int* item_range, float* part_o, float* part_ml, int B, int H, int dq, int dv,
                             long long num_slots, int max_pages, int max_items, int window, float scale, const float* head_gate, int dtype, void* stream_) {
  if (B <= 0) return 0;
  if (B > 1024 || H <= 0 || max_pages <= 0) return -1;
  if (dq <= 0 || dv <= 0 || dv > dq || dq % 8 != 0 || dv % 8 != 0 || dv > ML_MAX_LORA || dq > ML_MAX_TILES * 64 || (dv < dq && dv % 64 != 0) || window < 0)
    return -1;
  if (max_items < fb_mla_max_items(B, H)) return -1;
  cudaStream_t stream = reinterpret_cast<cudaStream_t>(stream_);
  const int n_groups = (H + ML_N - 1) / ML_N;
  static int sm_count = 0;
  if (sm_count == 0) {
    int dev = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sm_count, cudaDevAttrMultiProcessorCount, dev);
  }
  CUtensorMap tmLat, tmQ;
  if (!make_tmap_2d(&tmLat, lat_pool, (uint64_t)num_slots, dq, dq, ML_PAGE / 2, 64, 2, 3)) return -2;
  if (!make_tmap_2d(&tmQ, q, (uint64_t)B * H, dq, dq, ML_N, 64, 2, 3)) return -2;
  int threads = 32;
  while (threads < B) threads <<= 1;
  launch_k(mla_plan_kernel, dim3(1), dim3(threads), 0, stream, 0, seq_lens, B, n_groups, sm_count, window, work, n_work, item_range, max_items);
  MlaParams p;
  p.work = work; p.n_work = n_work; p.page_table = page_table; p.max_pages = max_pages; p.seq_lens = seq_lens;
  p.part_o = part_o; p.part_ml = part_ml; p.H = H; p.B = B; p.max_items = max_items;
  p.tiles = (dq + 63) / 64; p.vtiles = (dv + 63) / 64; p.o_stride = (dv + 127) / 128 * 128; p.o_cols = (dv + 127) / 128 * ML_N; p.window = window;
  p.scale_log2 = scale * 1.4426950408889634f;
  const uint32_t f = dtype == 1 ? 1u : 0u;
  p.idesc_s = make_idesc(f, f, 0, 0, 128, ML_N);
  p.idesc_o = make_idesc(f, f, 1, 0, 128, ML_N);
  const int gp = (H <= 16) ? 16 : 32;
  const int smem = ml_smem(p.tiles < 2 ? 2 : p.tiles);          // the half block of a one-tile row reads 16 KB past it
#define FB_MLA_LAUNCH(BF, GPV)                                                                                          \
  {                                                                                                                     \
    static DeviceOnce cfg;                                                                                            \
    if (cfg.need()) { cudaFuncSetAttribute(mla_decode_kernel<BF, GPV>, cudaFuncAttributeMaxDynamicSharedMemorySize, ml_smem(ML_MAX_TILES)); } \
    launch_k<PDL_ATTN>(mla_decode_kernel<BF, GPV>, dim3(sm_count), dim3(ML_THREADS), smem, stream, 0, tmLat, tmQ, p);           \
    launch_k<PDL_COMBINE>(mla_combine_kernel<BF>, dim3(B, H), dim3(128), 0, stream, 0, part_o, part_ml, item_range, (uint16_t*)out, H, n_groups, dv, p.o_stride, head_gate); \
  }
  if (dtype == 1) { if (gp == 16) FB_MLA_LAUNCH(true, 16) else FB_MLA_LAUNCH(true, 32) }
  else { if (gp == 16) FB_MLA_LAUNCH(false, 16) else FB_MLA_LAUNCH(false, 32) }
#undef FB_MLA_LAUNCH
  return (int)cudaGetLastError();
}
