// Mixture-of-experts execution for sm_100a: routing plan, token gather, grouped expert GEMMs, weighted combine.
//
//   moe_plan     one CTA: per-local-expert token counts, segment offsets padded to 16 rows, and for every (token, k)
//                pair its row in the expert-sorted buffer (-1 if the expert lives on another rank).  Deterministic:
//                rows inside a segment follow (token, k) order.
//   moe_gather   copies each routed token row into its sorted position
//   grouped GEMM swap-AB tcgen05 products of all experts in one persistent launch (moe_stream_kernel): a tile list over the
//                experts that got rows, weights from the stacked matrix, activations from the sorted buffer.  gate/up uses
//                the SwiGLU epilogue.
//   moe_combine  out[t] = sum_k w[t,k] * y_sorted[pos[t,k]]   in fixed k order (deterministic), plus a shared expert's row, gated
//
// Role of the reference's MergeMOE / FusedMOE (src/devices/cuda/cudadevice.cpp:8279-8562) and of its routed-row
// kernels ("Grouped...Indexed", src/devices/cuda/moe/fastllm-moe-fp8.cu; route count/offset/scatter in
// fastllm-moe-vllm-marlin.cu:405-528), which run the expert FFNs as CUDA-core GEMVs or Marlin mma.sync.
#include "gemm_smallm.cuh"
#include "launch.h"
#include "tmap.h"

FB_DEFINE_ERROR_API(moe)

namespace fb {

constexpr int KID_MOE_GROUPED = 40;

// counts / offsets / pos of the experts in [first, first + n_local); rows of a segment follow (token, k) order.
// One CTA, warp votes: pairs are taken in chunks of 32; a chunk's lanes learn by `match.any` how many earlier lanes
// go to the same expert, one lane per (chunk, expert) records the chunk's count, a scan over the chunks per expert turns the
// counts into bases, and rank = base of the chunk + earlier lanes of the chunk.  Needs chunks * n_local <= 8192 (16-bit counts in
// shared memory).
__global__ void __launch_bounds__(1024)
moe_plan_warp_kernel(const int* __restrict__ idx, int pairs, int first, int n_local, int* __restrict__ counts,
                     int* __restrict__ offsets, int* __restrict__ pos, int* __restrict__ total_rows, int pad) {
  __shared__ int s_idx[4096];
  __shared__ uint16_t s_w[8192];
  __shared__ int s_cnt[1024];
  __shared__ int s_off[1024];
  pdl_launch_dependents();
  pdl_wait();
  const int chunks = (pairs + 31) >> 5;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, nwarps = blockDim.x >> 5;
  const uint32_t lt_mask = (1u << lane) - 1u;
  for (int i = threadIdx.x; i < pairs; i += blockDim.x) {
    const int e = idx[i] - first;
    s_idx[i] = (e >= 0 && e < n_local) ? e : -1;
  }
  for (int i = threadIdx.x; i < chunks * n_local; i += blockDim.x) s_w[i] = 0;
  __syncthreads();
  for (int c = warp; c < chunks; c += nwarps) {
    const int i = (c << 5) + lane;
    const int e = i < pairs ? s_idx[i] : -1;
    const uint32_t same = __match_any_sync(0xffffffffu, e);
    if (e >= 0 && (same & lt_mask) == 0) s_w[c * n_local + e] = (uint16_t)__popc(same);
  }
  __syncthreads();
  for (int e = threadIdx.x; e < n_local; e += blockDim.x) {
    int run = 0;
    for (int c = 0; c < chunks; ++c) {
      const int v = s_w[c * n_local + e];
      s_w[c * n_local + e] = (uint16_t)run;
      run += v;
    }
    s_cnt[e] = run;
  }
  __syncthreads();
  if (threadIdx.x < 32) {
    int carry = 0;
    for (int base = 0; base < n_local; base += 32) {
      const int e = base + threadIdx.x;
      const int c = e < n_local ? (s_cnt[e] + pad - 1) / pad * pad : 0;
      int incl = c;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const int v = __shfl_up_sync(0xffffffffu, incl, o);
        if ((int)threadIdx.x >= o) incl += v;
      }
      if (e < n_local) s_off[e] = carry + incl - c;
      carry += __shfl_sync(0xffffffffu, incl, 31);
    }
    if (threadIdx.x == 0) *total_rows = carry;
  }
  __syncthreads();
  for (int e = threadIdx.x; e < n_local; e += blockDim.x) { counts[e] = s_cnt[e]; offsets[e] = s_off[e]; }
  for (int c = warp; c < chunks; c += nwarps) {
    const int i = (c << 5) + lane;
    const int e = i < pairs ? s_idx[i] : -1;
    const uint32_t same = __match_any_sync(0xffffffffu, e);
    if (i < pairs) pos[i] = e < 0 ? -1 : s_off[e] + (int)s_w[c * n_local + e] + __popc(same & lt_mask);
  }
}

// Larger problems, the same order: a CTA per 1024 pairs.  It counts the experts of all pairs itself, those before its own apart (the ids are a few
// hundred KB in L2; no scratch, no second launch, nothing to wait for), then ranks its own pairs like the kernel above, a chunk of 32 a warp.
// 32760 pairs, 128 experts: 8 us (71 us when one CTA walked all pairs twice).  Shared memory: [2][n_local] counters, [32][n_local] 16-bit ones.
__global__ void __launch_bounds__(1024)
moe_plan_blocks_kernel(const int* __restrict__ idx, int pairs, int first, int n_local, int* __restrict__ counts, int* __restrict__ offsets,
                       int* __restrict__ pos, int* __restrict__ total_rows, int pad) {
  extern __shared__ int s_dyn[];
  int* before = s_dyn;                                         // pairs ahead of this CTA's, then their expert's row for its first one
  int* rest = before + n_local;
  uint16_t* s_w = reinterpret_cast<uint16_t*>(rest + n_local);
  pdl_launch_dependents();
  pdl_wait();
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, start = blockIdx.x * 1024;
  const uint32_t lt_mask = (1u << lane) - 1u;
  for (int e = tid; e < 2 * n_local; e += 1024) s_dyn[e] = 0;
  for (int i = tid; i < 16 * n_local; i += 1024) reinterpret_cast<uint32_t*>(s_w)[i] = 0u;
  __syncthreads();
  int own = -1;
#pragma unroll 4
  for (int i = tid; i < pairs; i += 1024) {
    const int e = idx[i] - first;
    const bool ok = e >= 0 && e < n_local;
    if (ok) atomicAdd(i < start ? before + e : rest + e, 1);
    if (i - tid == start) own = ok ? e : -1;
  }
  const uint32_t same = __match_any_sync(0xffffffffu, own);
  const int rank = __popc(same & lt_mask);
  if (own >= 0 && rank == 0) s_w[warp * n_local + own] = (uint16_t)__popc(same);
  __syncthreads();
  for (int e = tid; e < n_local; e += 1024) {
    int run = 0;
    for (int w = 0; w < 32; ++w) {
      const int v = s_w[w * n_local + e];
      s_w[w * n_local + e] = (uint16_t)run;
      run += v;
    }
  }
  if (warp == 31) {
    int carry = 0;
    for (int base = 0; base < n_local; base += 32) {
      const int e = base + lane, b = e < n_local ? before[e] : 0, n = e < n_local ? b + rest[e] : 0, c = (n + pad - 1) / pad * pad;
      int incl = c;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const int v = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= o) incl += v;
      }
      if (e < n_local) {
        before[e] = carry + incl - c + b;
        if (blockIdx.x == 0) { counts[e] = n; offsets[e] = carry + incl - c; }
      }
      carry += __shfl_sync(0xffffffffu, incl, 31);
    }
    if (lane == 0 && blockIdx.x == 0) *total_rows = carry;
  }
  __syncthreads();
  if (start + tid < pairs) pos[start + tid] = own < 0 ? -1 : before[own] + (int)s_w[warp * n_local + own] + rank;
}

// A token's row to its places in the sorted buffer, read once and written topk times: bound by the writes.  Width 2048, us (a CTA a place, 128 threads,
// before): 4095 tokens x 8 places 40 -> 23, 4001 x 10 45 -> 30, 4000 x 6 28 -> 19.  Few tokens do not fill the chip by themselves: a CTA a place.
template <int U>
__global__ void __launch_bounds__(256) moe_gather_kernel(const uint16_t* __restrict__ x, const int* __restrict__ pos, uint16_t* __restrict__ xs, int topk, int H) {
  pdl_launch_dependents();
  pdl_wait();
  const int t = blockIdx.x, step = gridDim.y;
  const uint4* src = reinterpret_cast<const uint4*>(x + (size_t)t * H);
  for (int i = threadIdx.x; i < H / 8; i += 256) {
    const uint4 v = src[i];
    for (int k = blockIdx.y; k < topk; k += U * step) {
#pragma unroll
      for (int u = 0; u < U; ++u) {
        const int r = k + u * step < topk ? pos[t * topk + k + u * step] : -1;
        if (r >= 0) reinterpret_cast<uint4*>(xs + (size_t)r * H)[i] = v;
      }
    }
  }
}

// The rows of U places are asked for together; the sums keep the order of the places.  Bound by the rows' reads: 4095 tokens x 8 places of 2048, 32 -> 29 us.
template <bool BF16>
__global__ void __launch_bounds__(256) moe_combine_kernel(const uint16_t* __restrict__ ys, const int* __restrict__ pos, const float* __restrict__ w,
                                                          const uint16_t* __restrict__ add, const float* __restrict__ add_gate, int ld_gate,
                                                          uint16_t* __restrict__ out, int topk, int H) {
  constexpr int U = 4;
  const int t = blockIdx.x;
  pdl_launch_dependents();
  pdl_wait();
  const float ga = add_gate != nullptr ? 1.0f / (1.0f + __expf(-add_gate[(size_t)t * ld_gate])) : 1.0f;
  for (int c = threadIdx.x; c < H / 8; c += 256) {
    float acc[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
    auto add_row = [&](const uint4& v, float f) {
      const float2 a = unpack_16<BF16>(v.x), b = unpack_16<BF16>(v.y), cc = unpack_16<BF16>(v.z), d = unpack_16<BF16>(v.w);
      acc[0] += f * a.x; acc[1] += f * a.y; acc[2] += f * b.x; acc[3] += f * b.y;
      acc[4] += f * cc.x; acc[5] += f * cc.y; acc[6] += f * d.x; acc[7] += f * d.y;
    };
    uint4 own = make_uint4(0u, 0u, 0u, 0u);
    if (add != nullptr) own = *reinterpret_cast<const uint4*>(add + (size_t)t * H + c * 8);
    for (int k0 = 0; k0 < topk; k0 += U) {
      uint4 v[U];
      float wk[U];
      bool ok[U];
#pragma unroll
      for (int u = 0; u < U; ++u) {
        const int r = k0 + u < topk ? pos[t * topk + k0 + u] : -1;
        ok[u] = r >= 0;
        if (ok[u]) { v[u] = *reinterpret_cast<const uint4*>(ys + (size_t)r * H + c * 8); wk[u] = w[t * topk + k0 + u]; }
      }
#pragma unroll
      for (int u = 0; u < U; ++u)
        if (ok[u]) add_row(v[u], wk[u]);
    }
    if (add != nullptr) add_row(own, ga);
    uint4 o;
    o.x = pack_16<BF16>(acc[0], acc[1]); o.y = pack_16<BF16>(acc[2], acc[3]);
    o.z = pack_16<BF16>(acc[4], acc[5]); o.w = pack_16<BF16>(acc[6], acc[7]);
    *reinterpret_cast<uint4*>(out + (size_t)t * H + c * 8) = o;
  }
}

// Plans of all table-routed layers of a model in one launch, one CTA per layer: the experts of a token are the entries of its
// id's row of the layer's table, so the whole forward pass's routing is known once the token ids are.
//   meta  [L][4] = (table address, top, experts, table rows);  counts / offsets [L][e_stride], total [L], pos [L][T * k_stride]
// Rows inside an expert's segment come in no particular order (every row's product is computed by itself).
__global__ void __launch_bounds__(1024)
moe_plan_table_kernel(const long long* __restrict__ meta, const int* __restrict__ ids, int T, int* __restrict__ counts,
                      int* __restrict__ offsets, int* __restrict__ pos, int* __restrict__ total_rows, int e_stride, int k_stride, int pad) {
  __shared__ int s_cnt[1024];
  __shared__ int s_off[1024];
  pdl_launch_dependents();
  pdl_wait();
  const int l = blockIdx.x;
  const int* table = reinterpret_cast<const int*>(meta[4 * l]);
  const int top = (int)meta[4 * l + 1], E = (int)meta[4 * l + 2], rows = (int)meta[4 * l + 3];
  counts += (size_t)l * e_stride; offsets += (size_t)l * e_stride; pos += (size_t)l * T * k_stride;
  const int pairs = T * top;
  auto expert = [&](int i) {
    int id = ids[i / top];
    id = id < 0 ? 0 : (id >= rows ? rows - 1 : id);
    const int e = table[(size_t)id * top + i % top];
    return e < 0 || e >= E ? -1 : e;
  };
  for (int e = threadIdx.x; e < E; e += blockDim.x) s_cnt[e] = 0;
  __syncthreads();
  for (int i = threadIdx.x; i < pairs; i += blockDim.x) {
    const int e = expert(i);
    if (e >= 0) atomicAdd(&s_cnt[e], 1);
  }
  __syncthreads();
  if (threadIdx.x < 32) {
    int carry = 0;
    for (int base = 0; base < E; base += 32) {
      const int e = base + threadIdx.x;
      const int c = e < E ? (s_cnt[e] + pad - 1) / pad * pad : 0;
      int incl = c;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const int v = __shfl_up_sync(0xffffffffu, incl, o);
        if ((int)threadIdx.x >= o) incl += v;
      }
      if (e < E) { counts[e] = s_cnt[e]; offsets[e] = s_off[e] = carry + incl - c; }
      carry += __shfl_sync(0xffffffffu, incl, 31);
    }
    if (threadIdx.x == 0) total_rows[l] = carry;
  }
  __syncthreads();
  for (int i = threadIdx.x; i < pairs; i += blockDim.x) {
    const int e = expert(i);
    pos[i] = e < 0 ? -1 : atomicAdd(&s_off[e], 1);
  }
}

// Grouped dense GEMM: one CTA per SM walks (expert, row chunk, 128 weight rows) tiles, swap-AB as in the decode GEMM (weight rows x tokens).
//
// Bound: the weight stream while an expert gets few rows (every touched expert is read once), the tensor core from a few hundred rows on.
// The tile list is made on the device from the routed counts; the ring of operand stages runs on across tiles, so the short k of
// an expert's projections (512 to 2048: 8 to 32 stages) does not pay a pipeline fill, a TMEM set-up and a drain per tile, and two
// accumulators let the epilogue of a tile run under the products of the next.  Chunks of one expert are neighbours in the list: the
// second reads the weights from L2.  The product is as wide as the chunk has rows (multiples of 16), whatever the tile is laid out for.
// Per layer of width 2048 (gate/up + down; us; one CTA per tile before): 128 experts x 768 at 4095 x 8 rows 948 -> 326, 512 x 512 at 4001 x 10
// rows 1597 -> 592, at 32 x 10 rows 657 -> 263, 128 x 768 at 32 x 8 rows 237 -> 179.
struct MoeStreamInfo {
  const int* counts;       // [n_local] routed rows per expert
  const int* offsets;      // [n_local] first row of the expert's segment in the sorted buffer
  int n_local, n_tiles;    // tiles of a chunk: 128 weight rows, 256 for a pair
  int w_tiles;             // 128-row weight tiles per expert
};

constexpr int MS_MAX_EXPERTS = 1024;
constexpr int MS_EXTRA_FLAGS = GEMM_EXTRA_FLAGS | GEMM_BIAS | GEMM_RELU2;       // done by the EXTRA kernels alone
// Tiles laid out for this many rows or more are done by CTA pairs: 128 experts, 4095 x 8 rows 238 + 133 -> 206 + 120 us; with tiles of 128 rows
// (512 experts, 4001 x 10 rows) pairs take 378 + 233 us, one CTA a tile 380 + 212.
constexpr int MS_PAIR_FROM = 256;
template <int MPAD, bool PAIR>
struct MoeStreamCfg {
  static constexpr int A_BYTES = 128 * 128;
  static constexpr int X_ROWS = PAIR ? MPAD / 2 : MPAD;             // token rows that one CTA holds
  static constexpr int BOX = X_ROWS < 64 ? X_ROWS : 64;             // token rows per load
  static constexpr int STAGE_BYTES = A_BYTES + X_ROWS * 128;
  static constexpr int X_BYTES = 2 * (MPAD < 32 ? MPAD : 32) * 64 * 4;      // sums that gate and up warps exchange, two buffers of 32 tokens
  static constexpr int TAIL_BYTES = X_BYTES + 3 * MS_MAX_EXPERTS * 4 + 32 + 512;
  static constexpr int MAX_STAGES = (226 * 1024 - TAIL_BYTES) / STAGE_BYTES;
  static constexpr int STAGES = MAX_STAGES > 12 ? 12 : MAX_STAGES;
  static constexpr int SMEM_BYTES = STAGES * STAGE_BYTES + TAIL_BYTES + 1024;
  static constexpr int TMEM_COLS = 2 * MPAD < 32 ? 32 : 2 * MPAD;
};

struct MoeTile { int e, n_tile, row0, rows; };
// tile t of the list; first[e] = chunks of the experts before e, counts[e] = rows
template <int MPAD>
__device__ __forceinline__ MoeTile moe_tile(const MoeStreamInfo& gi, const int* first, const int* counts, int t) {
  int lo = 0, hi = gi.n_local - 1;                     // the last expert whose first tile is at or before t
  while (lo < hi) {
    const int mid = (lo + hi + 1) >> 1;
    if (first[mid] * gi.n_tiles <= t) lo = mid; else hi = mid - 1;
  }
  MoeTile r;
  const int ch = first[lo + 1] - first[lo], at = t - first[lo] * gi.n_tiles, cnt = counts[lo];
  const int per = ((cnt + ch - 1) / ch + 15) & ~15;    // rows of a chunk: equal shares, at most MPAD
  const int chunk = at % ch;
  r.e = lo;
  r.n_tile = at / ch;
  r.row0 = chunk * per;
  r.rows = min(per, cnt - r.row0);
  return r;
}

// One output column of the first cnt of N tokens, ld apart.  One epilogue warp sits on each sub-core, so its instructions are a chain: with an
// address from scratch and two conditions per element (21 instructions) the epilogue took longer than the tile's products.
template <int N, bool BF16>
__device__ __forceinline__ void store_column(uint16_t* out, int ld, const float (&v)[N], int cnt) {
  if (cnt >= N) {
#pragma unroll
    for (int j = 0; j < N; ++j, out += ld) *out = (uint16_t)(pack_16<BF16>(v[j], 0.f) & 0xFFFFu);
  } else {
#pragma unroll
    for (int j = 0; j < N; ++j, out += ld) {
      if (j >= cnt) break;
      *out = (uint16_t)(pack_16<BF16>(v[j], 0.f) & 0xFFFFu);
    }
  }
}

template <int MPAD, bool BF16, bool EXTRA, bool PAIR>
__global__ void __launch_bounds__(192, 1)
moe_stream_kernel(const __grid_constant__ CUtensorMap tmW, const __grid_constant__ CUtensorMap tmX, const GemmParams p, const MoeStreamInfo gi) {
  using Cfg = MoeStreamCfg<MPAD, PAIR>;
  extern __shared__ uint8_t smem_raw[];
  __shared__ int wsum[6];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  float* X = reinterpret_cast<float*>(smem + Cfg::STAGES * Cfg::STAGE_BYTES);
  int* first = reinterpret_cast<int*>(reinterpret_cast<uint8_t*>(X) + Cfg::X_BYTES);              // [n_local + 1]
  int* counts = first + MS_MAX_EXPERTS + 8;            // copies of the plan's tables: a tile is looked up by three roles
  int* offsets = counts + MS_MAX_EXPERTS;
  uint64_t* full_bar = reinterpret_cast<uint64_t*>(offsets + MS_MAX_EXPERTS);
  uint64_t* empty_bar = full_bar + Cfg::STAGES;
  uint64_t* acc_full = empty_bar + Cfg::STAGES;        // [2]
  uint64_t* acc_empty = acc_full + 2;                  // [2]
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(acc_empty + 2);
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int rank = PAIR ? (int)cluster_ctarank() : 0;
  const int unit = PAIR ? (int)(blockIdx.x >> 1) : (int)blockIdx.x, units = PAIR ? (int)(gridDim.x >> 1) : (int)gridDim.x;
  bool dead = false;
  pdl_launch_dependents();
  if (tid == 0) {
    for (int s = 0; s < Cfg::STAGES; ++s) { mbar_init(&full_bar[s], 1); mbar_init(&empty_bar[s], 1); }
    for (int b = 0; b < 2; ++b) { mbar_init(&acc_full[b], 1); mbar_init(&acc_empty[b], PAIR ? 8 : 4); }
    mbar_init_fence();
    tma_prefetch_desc(&tmW);
    tma_prefetch_desc(&tmX);
  }
  if (warp == 1) {
    if (PAIR) { tmem_alloc_pair(tmem_slot, Cfg::TMEM_COLS); tmem_relinquish_pair(); }
    else { tmem_alloc(tmem_slot, Cfg::TMEM_COLS); tmem_relinquish(); }
  }
  pdl_wait();                                          // counts and offsets come from the plan kernel
  {
    const int each = (gi.n_local + 191) / 192, e0 = tid * each;
    int sum = 0;
    for (int i = 0; i < each; ++i) {
      if (e0 + i >= gi.n_local) break;
      const int c = gi.counts[e0 + i];
      counts[e0 + i] = c;
      offsets[e0 + i] = gi.offsets[e0 + i];
      sum += (c + MPAD - 1) / MPAD;
    }
    int incl = sum;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) { const int v = __shfl_up_sync(0xffffffffu, incl, o); if (lane >= o) incl += v; }
    if (lane == 31) wsum[warp] = incl;
    __syncthreads();
    int run = incl - sum;
    for (int w = 0; w < warp; ++w) run += wsum[w];
    for (int i = 0; i < each; ++i) {
      if (e0 + i >= gi.n_local) break;
      first[e0 + i] = run;
      run += (counts[e0 + i] + MPAD - 1) / MPAD;
      if (e0 + i == gi.n_local - 1) first[gi.n_local] = run;
    }
  }
  tc_fence_before_sync();
  __syncthreads();
  if (PAIR) cluster_sync_all();                        // the other CTA's barriers exist, too
  tc_fence_after_sync();
  const uint32_t tmem_base = *tmem_slot;
  const int total = first[gi.n_local] * gi.n_tiles, kb_cnt = p.kb_total;

  if (warp == 0) {
    if (elect_one()) {
      const uint64_t pol_w = l2_policy_evict_first();
      const uint64_t pol_x = l2_policy_evict_last();
      int it = 0;
      for (int t = unit; t < total && !dead; t += units) {
        const MoeTile m = moe_tile<MPAD>(gi, first, counts, t);
        if (m.rows <= 0) continue;
        const int share = PAIR ? ((m.rows + 31) & ~31) >> 1 : m.rows;              // token rows of this CTA
        const int w_row = (m.e * gi.w_tiles + (PAIR ? 2 * m.n_tile + rank : m.n_tile)) * 128, x_row = offsets[m.e] + m.row0 + rank * share;
        const int boxes = (share + Cfg::BOX - 1) / Cfg::BOX;
        for (int i = 0; i < kb_cnt; ++i, ++it) {
          const int s = it % Cfg::STAGES;
          if (!mbar_wait(&empty_bar[s], ((uint32_t)(it / Cfg::STAGES) & 1u) ^ 1u, dead, KID_MOE_GROUPED, 1)) break;
          uint8_t* a = smem + s * Cfg::STAGE_BYTES;
          if (PAIR) {
            const uint32_t bar = mapa_u32(smem_u32(&full_bar[s]), 0);
            if (rank == 0) mbar_expect_tx(&full_bar[s], 2 * (Cfg::A_BYTES + boxes * Cfg::BOX * 128));
            tma_load_2d_pair(a, &tmW, bar, i * 64, w_row);
            for (int b = 0; b < boxes; ++b) tma_load_2d_pair(a + Cfg::A_BYTES + b * Cfg::BOX * 128, &tmX, bar, i * 64, x_row + b * Cfg::BOX);
            continue;
          }
          mbar_expect_tx(&full_bar[s], Cfg::A_BYTES + boxes * Cfg::BOX * 128);
          if (MPAD <= 64) tma_load_2d_hint(a, &tmW, &full_bar[s], i * 64, w_row, pol_w);
          else tma_load_2d(a, &tmW, &full_bar[s], i * 64, w_row);                 // (the expert's next chunk reads them again)
          for (int b = 0; b < boxes; ++b) tma_load_2d_hint(a + Cfg::A_BYTES + b * Cfg::BOX * 128, &tmX, &full_bar[s], i * 64, x_row + b * Cfg::BOX, pol_x);
        }
      }
      // a pair: the last products' commits have reached this CTA before it may leave
      for (int k = !PAIR ? it : it > Cfg::STAGES ? it - Cfg::STAGES : 0; k < it; ++k)
        if (!mbar_wait(&empty_bar[k % Cfg::STAGES], (uint32_t)(k / Cfg::STAGES) & 1u, dead, KID_MOE_GROUPED, 5)) break;
    }
    __syncwarp();
  } else if (warp == 1) {
    if (rank == 0 && elect_one()) {
      int it = 0, u = 0;
      for (int t = unit; t < total && !dead; t += units) {
        const MoeTile m = moe_tile<MPAD>(gi, first, counts, t);
        if (m.rows <= 0) continue;
        const int buf = u & 1;
        const uint32_t use = ((uint32_t)(u >> 1) & 1u) ^ 1u;
        if (!(PAIR ? mbar_wait_cluster(&acc_empty[buf], use, dead, KID_MOE_GROUPED, 4) : mbar_wait(&acc_empty[buf], use, dead, KID_MOE_GROUPED, 4))) break;
        tc_fence_after_sync();
        // N = rows in multiples of 16 (a pair: of 16 a CTA)
        const uint32_t acc = tmem_base + (uint32_t)(buf * MPAD), idesc = p.idesc | ((PAIR ? (uint32_t)((m.rows + 31) >> 5) << 1 : (uint32_t)((m.rows + 15) >> 4)) << 18);
        for (int i = 0; i < kb_cnt; ++i, ++it) {
          const int s = it % Cfg::STAGES;
          const uint32_t ph = (uint32_t)(it / Cfg::STAGES) & 1u;
          if (!(PAIR ? mbar_wait_cluster(&full_bar[s], ph, dead, KID_MOE_GROUPED, 2) : mbar_wait(&full_bar[s], ph, dead, KID_MOE_GROUPED, 2))) break;
          tc_fence_after_sync();
          const uint32_t a_addr = smem_u32(smem + s * Cfg::STAGE_BYTES);
          const uint64_t da = make_smem_desc(a_addr, 16, 1024, SWZ_128B), db = make_smem_desc(a_addr + Cfg::A_BYTES, 16, 1024, SWZ_128B);
#pragma unroll
          for (int k = 0; k < 4; ++k) {
            if (PAIR) umma_f16_pair(acc, da + 2 * k, db + 2 * k, idesc, (i | k) != 0 ? 1u : 0u);
            else umma_f16(acc, da + 2 * k, db + 2 * k, idesc, (i | k) != 0 ? 1u : 0u);
          }
          if (PAIR) umma_commit_pair(&empty_bar[s]); else umma_commit(&empty_bar[s]);
        }
        if (dead) break;
        if (PAIR) umma_commit_pair(&acc_full[buf]); else umma_commit(&acc_full[buf]);
        ++u;
      }
    }
    __syncwarp();
  } else {
    // a thread whose wait ran out still walks the tiles: it meets the named barriers below
    const int q = warp & 3, n_local = q * 32 + lane;
    const bool swiglu = (p.flags & GEMM_SWIGLU) != 0;
    uint16_t* outp = reinterpret_cast<uint16_t*>(p.out);
    int u = 0, ci = 0;                                 // tiles and 32-token pieces done
    for (int t = unit; t < total; t += units) {
      MoeTile m = moe_tile<MPAD>(gi, first, counts, t);
      if (m.rows <= 0) continue;
      if (PAIR) m.n_tile = 2 * m.n_tile + rank;        // this CTA's weight rows
      const int buf = u & 1;
      if (PAIR) mbar_wait_cluster(&acc_full[buf], (uint32_t)(u >> 1) & 1u, dead, KID_MOE_GROUPED, 3);
      else mbar_wait(&acc_full[buf], (uint32_t)(u >> 1) & 1u, dead, KID_MOE_GROUPED, 3);
      ++u;
      __syncwarp();
      tc_fence_after_sync();
      const uint32_t acc = tmem_base + (uint32_t)(buf * MPAD) + ((uint32_t)(q * 32) << 16);
      uint16_t* orow = outp + (size_t)(offsets[m.e] + m.row0) * p.ld_out;
      constexpr int CH = MPAD < 32 ? MPAD : 32;
      for (int c0 = 0; c0 < m.rows; c0 += CH, ++ci) {
        uint32_t r[32];
        __syncwarp();
        if (CH == 32) tmem_ld_32x32b_x32(acc + c0, r); else tmem_ld_32x32b_x16(acc + c0, r);
        tmem_ld_wait();
        const int cnt = min(CH, m.rows - c0);
        if (swiglu) {
          // rows 0..63 of a tile are gate rows, 64..127 the up rows of the same columns.  The gate's warps do the first half of the tokens and take the
          // up sums from shared memory, the up warps do the second half and take the gate sums; two buffers, so one barrier a piece is enough
          constexpr int HALF = CH / 2;
          const int col = n_local & 63, first_tok = q < 2 ? 0 : HALF;
          float* xb = X + (ci & 1) * CH * 64 + col;
          float v[HALF], o[HALF];
          if (q < 2) {
#pragma unroll
            for (int j = 0; j < HALF; ++j) { v[j] = __uint_as_float(r[j]); xb[(HALF + j) * 64] = __uint_as_float(r[HALF + j]); }
          } else {
#pragma unroll
            for (int j = 0; j < HALF; ++j) { v[j] = __uint_as_float(r[HALF + j]); xb[j * 64] = __uint_as_float(r[j]); }
          }
          asm volatile("bar.sync 1, 128;\n" ::: "memory");
#pragma unroll
          for (int j = 0; j < HALF; ++j) o[j] = xb[(first_tok + j) * 64];
          const bool clamp = (p.flags & GEMM_GLU_CLAMP) != 0;
          const int n = m.n_tile * 64 + col;
          float bg = 0.f, bu = 0.f;
          if (EXTRA && (p.flags & GEMM_BIAS) && n < (p.N >> 1)) {
            const uint16_t* b = reinterpret_cast<const uint16_t*>(p.bias) + (size_t)m.e * p.N + m.n_tile * 128 + col;
            bg = unpack_16<BF16>(b[0]).x;
            bu = unpack_16<BF16>(b[64]).x;
          }
#pragma unroll
          for (int j = 0; j < HALF; ++j) {
            float g = q < 2 ? v[j] : o[j], up = q < 2 ? o[j] : v[j];
            if (EXTRA) { g += bg; up += bu; }
            v[j] = clamp ? glu_clamp_f(g, up, p.act_limit, p.act_alpha) : EXTRA && (p.flags & GEMM_GEGLU) ? gelu_tanh_f(g) * up : silu_f(g) * up;
            if (EXTRA && (p.flags & GEMM_RELU2)) v[j] = relu2_f(v[j]);
          }
          if (!dead && n < (p.N >> 1)) store_column<HALF, BF16>(orow + (size_t)(c0 + first_tok) * p.ld_out + n, p.ld_out, v, cnt - first_tok);
        } else {
          const int n = m.n_tile * 128 + n_local;
          float v[CH];
#pragma unroll
          for (int j = 0; j < CH; ++j) v[j] = __uint_as_float(r[j]);
          if (EXTRA) {
            const float bias = (p.flags & GEMM_BIAS) && n < p.N ? unpack_16<BF16>(reinterpret_cast<const uint16_t*>(p.bias)[(size_t)m.e * p.N + n]).x : 0.f;
#pragma unroll
            for (int j = 0; j < CH; ++j) {
              v[j] += bias;
              if (p.flags & GEMM_RELU2) v[j] = relu2_f(v[j]);
              if (p.flags & GEMM_GELU) v[j] = gelu_erf_f(v[j]);
              if (p.flags & GEMM_GELU_TANH) v[j] = gelu_tanh_f(v[j]);
            }
          }
          if (!dead && n < p.N) store_column<CH, BF16>(orow + (size_t)c0 * p.ld_out + n, p.ld_out, v, cnt);
        }
      }
      tc_fence_before_sync();
      __syncwarp();
      if (lane == 0) {
        if (PAIR) mbar_arrive_cluster(mapa_u32(smem_u32(&acc_empty[buf]), 0)); else mbar_arrive(&acc_empty[buf]);
      }
    }
  }
  __syncwarp();
  tc_fence_before_sync();
  __syncthreads();
  if (PAIR) cluster_sync_all();                        // neither CTA's barriers or operands are in use any more
  if (warp == 1) {
    if (PAIR) tmem_dealloc_pair(tmem_base, Cfg::TMEM_COLS); else tmem_dealloc(tmem_base, Cfg::TMEM_COLS);
  }
  __syncwarp();
  if (PAIR) cluster_sync_all();
}

template <int MPAD, bool BF16, bool PAIR>
static cudaError_t launch_stream(const CUtensorMap& tmW, const CUtensorMap& tmX, const GemmParams& p, const MoeStreamInfo& gi, int grid, cudaStream_t stream) {
  using Cfg = MoeStreamCfg<MPAD, PAIR>;
  auto plain = moe_stream_kernel<MPAD, BF16, false, PAIR>;
  auto extra = moe_stream_kernel<MPAD, BF16, true, PAIR>;
  static DeviceOnce configured;
  if (configured.need()) {
    cudaError_t e = cudaFuncSetAttribute(plain, cudaFuncAttributeMaxDynamicSharedMemorySize, Cfg::SMEM_BYTES);
    if (e == cudaSuccess) e = cudaFuncSetAttribute(extra, cudaFuncAttributeMaxDynamicSharedMemorySize, Cfg::SMEM_BYTES);
    if (e != cudaSuccess) return e;
  }
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(grid);
  cfg.blockDim = dim3(192);
  cfg.dynamicSmemBytes = Cfg::SMEM_BYTES;
  cfg.stream = stream;
  cudaLaunchAttribute attr[2];
  if (PAIR) {
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = 2;
    attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
  }
  cfg.attrs = attr; cfg.numAttrs = add_pdl_attr(attr, PAIR ? 1 : 0);
  return cudaLaunchKernelEx(&cfg, (p.flags & MS_EXTRA_FLAGS) ? extra : plain, tmW, tmX, p, gi);
}

// The same for few tiles: a cluster splits a tile's k among its CTAs and adds the parts up through distributed shared memory, in rank order; a CTA
// group per (expert, chunk, 128 weight rows).  With 32 tiles (one expert of 4096 outputs) the persistent launch leaves four fifths of the SMs idle.
// One expert, 4096 x 14336: 52 -> 31 us at 1 to 32 rows, 70 -> 35 at 128; 4096 x 7168, gated: 31 -> 22.
struct MoeSplitInfo {
  const int* counts;       // [n_local] routed rows per expert
  const int* offsets;      // [n_local] first row of the expert's segment in the sorted buffer
  int n_local, rows_per_chunk, n_rows_w;      // experts, MPAD, weight rows per expert in the stacked matrix
};

template <int MPAD, bool BF16, class Epi>
__global__ void __launch_bounds__(192, 1)
moe_split_kernel(const __grid_constant__ CUtensorMap tmW, const __grid_constant__ CUtensorMap tmX, const GemmParams base, const MoeSplitInfo gi) {
  pdl_launch_dependents();
  pdl_wait();                                        // counts and offsets come from the plan kernel
  int e = 0, chunk = 0;
  if (!moe_find_item(gi.counts, gi.n_local, gi.rows_per_chunk, (int)blockIdx.z, e, chunk)) return;      // uniform over the cluster
  GemmParams p = base;
  const int row0 = chunk * gi.rows_per_chunk, seg = gi.offsets[e] + row0;
  p.M = min(gi.counts[e] - row0, gi.rows_per_chunk);
  p.x_row0 = seg;
  p.w_row0 = e * gi.n_rows_w;
  p.out = reinterpret_cast<uint16_t*>(base.out) + (size_t)seg * base.ld_out;
  if (base.bias != nullptr) p.bias = reinterpret_cast<const uint16_t*>(base.bias) + (size_t)e * base.N;
  uint32_t tmem_base;
  gemm_smallm_device<MPAD, BF16, 1, Epi>(tmW, tmX, p, tmem_base, KID_MOE_GROUPED, Epi());
  if ((threadIdx.x >> 5) == 1) tmem_dealloc(tmem_base, SmallMCfg<MPAD, 1>::TMEM_COLS);
}

template <int MPAD, bool BF16>
static cudaError_t launch_split(const CUtensorMap& tmW, const CUtensorMap& tmX, const GemmParams& p, const MoeSplitInfo& gi, int nsplit, int n_tiles, int chunks,
                                cudaStream_t stream) {
  using Cfg = SmallMCfg<MPAD, 1>;
  auto plain = moe_split_kernel<MPAD, BF16, StoreEpilogue<BF16>>;
  auto extra = moe_split_kernel<MPAD, BF16, ExtraEpilogue<BF16>>;
  static DeviceOnce configured;
  if (configured.need()) {
    cudaError_t e = cudaFuncSetAttribute(plain, cudaFuncAttributeMaxDynamicSharedMemorySize, Cfg::SMEM_BYTES);
    if (e == cudaSuccess) e = cudaFuncSetAttribute(extra, cudaFuncAttributeMaxDynamicSharedMemorySize, Cfg::SMEM_BYTES);
    if (e != cudaSuccess) return e;
  }
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(nsplit, n_tiles, chunks);
  cfg.blockDim = dim3(192);
  cfg.dynamicSmemBytes = Cfg::SMEM_BYTES;
  cfg.stream = stream;
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = nsplit;
  attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
  cfg.attrs = attr; cfg.numAttrs = add_pdl_attr(attr, 1);
  return cudaLaunchKernelEx(&cfg, (p.flags & GEMM_EXTRA_FLAGS) ? extra : plain, tmW, tmX, p, gi);
}

}  // namespace fb

using namespace fb;

extern "C" int fb_moe_plan(const int* idx, int T, int topk, int first, int n_local, int* counts, int* offsets, int* pos,
                           int* total_rows, int pad, void* stream) {
  if (n_local <= 0 || n_local > 1024 || T <= 0) return -1;
  auto s = reinterpret_cast<cudaStream_t>(stream);
  const int pairs = T * topk;
  if (pairs <= 4096 && ((pairs + 31) / 32) * n_local <= 8192) {
    launch_k(moe_plan_warp_kernel, dim3(1), dim3(1024), 0, s, 0, idx, pairs, first, n_local, counts, offsets, pos, total_rows, pad);
    return (int)cudaGetLastError();
  }
  static DeviceOnce cfg;
  if (cfg.need()) cudaFuncSetAttribute(moe_plan_blocks_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, 72 * 1024);
  launch_k(moe_plan_blocks_kernel, dim3((pairs + 1023) / 1024), dim3(1024), (size_t)72 * n_local, s, 0, idx, pairs, first, n_local, counts, offsets, pos, total_rows, pad);
  return (int)cudaGetLastError();
}

extern "C" int fb_moe_plan_table(const long long* meta, int L, const int* ids, int T, int* counts, int* offsets, int* pos, int* total_rows,
                                 int e_stride, int k_stride, int pad, void* stream) {
  if (L <= 0 || T <= 0) return 0;
  if (e_stride <= 0 || e_stride > 1024 || k_stride <= 0) return -1;
  launch_k(moe_plan_table_kernel, dim3(L), dim3(1024), 0, reinterpret_cast<cudaStream_t>(stream), 0, meta, ids, T, counts, offsets, pos,
           total_rows, e_stride, k_stride, pad);
  return (int)cudaGetLastError();
}

extern "C" int fb_moe_gather(const void* x, const int* pos, void* xs, int T, int topk, int H, void* stream) {
  if (T <= 0) return 0;
  if (H % 8 != 0) return -1;
  const bool few = T < 256;                        // not a CTA for every SM by tokens alone
  launch_k(few ? moe_gather_kernel<1> : moe_gather_kernel<4>, dim3(T, few ? topk : 1), dim3(256), 0, reinterpret_cast<cudaStream_t>(stream), 0, (const uint16_t*)x, pos,
           (uint16_t*)xs, topk, H);
  return (int)cudaGetLastError();
}

// add (optional) [T, H]: a shared expert's rows; add_gate (optional): one fp32 logit per token (ld_gate apart), add counts times its sigmoid.
extern "C" int fb_moe_combine_gated(const void* ys, const int* pos, const float* w, const void* add, const float* add_gate, int ld_gate, void* out, int T, int topk,
                                    int H, int dtype, void* stream) {
  if (T <= 0) return 0;
  if (H % 8 != 0) return -1;
  auto s = reinterpret_cast<cudaStream_t>(stream);
  if (dtype == 1)
    launch_k(moe_combine_kernel<true>, dim3(T), dim3(256), 0, s, 0, (const uint16_t*)ys, pos, w, (const uint16_t*)add, add_gate, ld_gate, (uint16_t*)out, topk, H);
  else
    launch_k(moe_combine_kernel<false>, dim3(T), dim3(256), 0, s, 0, (const uint16_t*)ys, pos, w, (const uint16_t*)add, add_gate, ld_gate, (uint16_t*)out, topk, H);
  return (int)cudaGetLastError();
}

extern "C" int fb_moe_combine(const void* ys, const int* pos, const float* w, const void* add, void* out, int T, int topk, int H,
                              int dtype, void* stream) {
  return fb_moe_combine_gated(ys, pos, w, add, nullptr, 0, out, T, topk, H, dtype, stream);
}

extern "C" int fb_moe_grouped_gemm_act(const void* Xs, const void* W, void* out, const void* bias, const int* counts, const int* offsets,
                                       int rows_cap, int E_local, int N, int K, int ld_out, int max_rows_per_expert, int dtype, int flags,
                                       int total_rows, float act_limit, float act_alpha, void* stream_);

// Grouped Y_e = X_e W_e^T over the sorted buffer.  Xs: [rows_cap, K] sorted rows; W: stacked [E_local * N, K] with every
// expert's rows padded to a multiple of 128; out: [rows_cap, N or N/2]; bias (with GEMM_BIAS): 16-bit [E_local, N], added before the activation.
// max_rows_per_expert: low 16 bits the most rows an expert can get (T for decode: every token could pick the same one), above them the rows of a
// typical busy expert, for which the tiles are laid out (0: the most).
extern "C" int fb_moe_grouped_gemm(const void* Xs, const void* W, void* out, const void* bias, const int* counts, const int* offsets,
                                   int rows_cap, int E_local, int N, int K, int ld_out, int max_rows_per_expert, int dtype, int flags,
                                   int total_rows, void* stream_) {
  return fb_moe_grouped_gemm_act(Xs, W, out, bias, counts, offsets, rows_cap, E_local, N, K, ld_out, max_rows_per_expert, dtype, flags, total_rows, 0.f,
                                 1.f, stream_);
}

// act_limit / act_alpha: constants of the GEMM_GLU_CLAMP activation.
extern "C" int fb_moe_grouped_gemm_act(const void* Xs, const void* W, void* out, const void* bias, const int* counts, const int* offsets,
                                       int rows_cap, int E_local, int N, int K, int ld_out, int max_rows_per_expert, int dtype, int flags,
                                       int total_rows, float act_limit, float act_alpha, void* stream_) {
  cudaStream_t stream = reinterpret_cast<cudaStream_t>(stream_);
  if (E_local <= 0 || rows_cap <= 0) return 0;
  if (K % 8 != 0 || N % 8 != 0 || ((flags & GEMM_SWIGLU) && N % 128 != 0) || (dtype != 0 && dtype != 1) || E_local > MS_MAX_EXPERTS ||
      ((flags & GEMM_BIAS) && bias == nullptr) || (flags & ~(MS_EXTRA_FLAGS | GEMM_SWIGLU | GEMM_GLU_CLAMP)))
    return -1;
  const int n_tiles = (N + 127) / 128;
  const bool bf16 = dtype == 1;
  const int hint = max_rows_per_expert >> 16, most = max_rows_per_expert & 0xFFFF, want = hint > 0 && hint < most ? hint : most;
  int mpad = 16;
  while (mpad < want && mpad < 256) mpad <<= 1;
  GemmParams p = {};
  p.out = out; p.bias = bias; p.N = N; p.K = K; p.ld_out = ld_out; p.kb_total = (K + 63) / 64; p.flags = flags;
  p.act_limit = act_limit; p.act_alpha = act_alpha;
  const bool pair = mpad >= MS_PAIR_FROM;
  p.idesc = make_idesc(bf16 ? 1 : 0, bf16 ? 1 : 0, 0, 0, pair ? 256 : 128, 0);
  MoeStreamInfo gi;
  gi.counts = counts; gi.offsets = offsets; gi.n_local = E_local; gi.n_tiles = pair ? (n_tiles + 1) / 2 : n_tiles; gi.w_tiles = n_tiles;
  CUtensorMap tmW, tmX;
  if (!make_tmap_2d(&tmW, W, (uint64_t)E_local * n_tiles * 128, K, K, 128, 64, 2, 3)) return -2;
  if (!make_tmap_2d(&tmX, Xs, rows_cap, K, K, mpad < 64 ? mpad : 64, 64, 2, 3)) return -2;
  static int sms = 0;
  if (sms == 0) {
    int dev = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  }
  // no more CTAs than tiles can exist: every routed row touches an expert, every expert's last chunk may be short
  long long bound = (long long)E_local * ((most + mpad - 1) / mpad);
  if (total_rows > 0 && bound > (long long)total_rows) bound = total_rows;
  // Few tiles: four or two CTAs a tile, where that many fit and k is long enough to pay for adding the parts up.  Both sides in us, one CTA a tile ->
  // split: 4 ways, 2048 of k, 12 tiles 14.4 -> 13.3 (128 rows 19.5 -> 16.4); 1408 of k, 16 tiles, 128 rows 14.3 -> 18.4 stays whole; 2 ways, 7168 of k, 64
  // tiles 31.7 -> 29.8 (128 rows 46 -> 33); 2048 of k, 56 tiles, 128 rows 18.5 -> 22.5 stays whole.
  const long long most_tiles = bound * n_tiles;
  const int nsplit = 4 * most_tiles <= sms && p.kb_total >= 32 ? 4 : 2 * most_tiles <= sms && p.kb_total >= 64 ? 2 : 1;
  if (nsplit > 1 && mpad <= 128) {
    p.kb_per_split = (p.kb_total + nsplit - 1) / nsplit;
    p.idesc = make_idesc(bf16 ? 1 : 0, bf16 ? 1 : 0, 0, 0, 128, mpad);
    p.scatter_rows = 1;
    if (!make_tmap_2d(&tmX, Xs, rows_cap, K, K, mpad, 64, 2, 3)) return -2;
    MoeSplitInfo si;
    si.counts = counts; si.offsets = offsets; si.n_local = E_local; si.rows_per_chunk = mpad; si.n_rows_w = n_tiles * 128;
#define FB_MS(MP) \
  return (int)(bf16 ? launch_split<MP, true>(tmW, tmX, p, si, nsplit, n_tiles, (int)bound, stream) : launch_split<MP, false>(tmW, tmX, p, si, nsplit, n_tiles, (int)bound, stream));
    switch (mpad) {
      case 16: FB_MS(16)
      case 32: FB_MS(32)
      case 64: FB_MS(64)
      default: FB_MS(128)
    }
#undef FB_MS
  }
  const int units = pair ? sms / 2 : sms;
  const int grid = (int)(bound * gi.n_tiles < units ? bound * gi.n_tiles : units) * (pair ? 2 : 1);
#define FB_MG(MP) \
  return (int)(bf16 ? launch_stream<MP, true, (MP >= MS_PAIR_FROM)>(tmW, tmX, p, gi, grid, stream) : launch_stream<MP, false, (MP >= MS_PAIR_FROM)>(tmW, tmX, p, gi, grid, stream));
  switch (mpad) {
    case 16: FB_MG(16)
    case 32: FB_MG(32)
    case 64: FB_MG(64)
    case 128: FB_MG(128)
    default: FB_MG(256)
  }
#undef FB_MG
}
