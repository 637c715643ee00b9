// Causal paged prefill attention for head widths other than 128 (multiples of 8 up to 256) on sm_100a (tcgen05 + TMEM).
//
// One CTA owns one query head and 128 consecutive new tokens of one request and walks the pages in steps of 64 keys:
//     S[128 q x 64 k] = Q * K^T        O[128 q x V] += P * V
// Two score buffers: the tensor core makes the scores of step i + 1 while the softmax warps, two threads a query row, 32 keys each, work on step i.  Keys and
// values have rings of their own (two steps each; a key step is free as soon as its scores exist).  At 256 x 256 the queries take 64 KB,
// the rings 128 KB, P 32 KB, and O 256 of the 512 TMEM columns, so that one CTA fills an SM; K and V of a group's heads meet in the L2.  (Narrower
// heads leave shared memory for a second CTA, but all columns are taken whatever V is: it waits for them.)
// Probabilities enter the second product as two 16-bit terms (rounded value, rounded remainder): 16 bits of them in bf16.  In fp16 the terms are
// scaled by 2^13, which the sum shares, so that what they leave out is 2^-38 of the largest weight.  O is rescaled only when a row's maximum has grown
// by more than 2^8 (fp16: 2^2), which changes no rounding of P and keeps fp16 terms finite (up to 2^15).
// The weights of a step are made in registers under the second product of the step before; only their way into shared memory waits for it.
// Bound: the chain of a step through the softmax threads (scores, maximum, weights, P), two warps on each sub-core.
// 4001 tokens x 16 heads x 256: 194 us; 216 with one thread a row, 258 when the weights waited for the product, too (PyTorch, gathered fp32 keys and
// values and fp32 scores in memory: 7.0 ms).
#include "ptx.cuh"
#include "launch.h"
#include "tmap.h"

FB_DEFINE_ERROR_API(attn_wide)

namespace fb {

constexpr int KID_ATTN_WIDE = 19;
constexpr int AX_Q = 128;                         // query rows of a CTA
constexpr int AX_KV = 64;                         // keys a step
constexpr int AX_QT = AX_Q * 128;                 // bytes of a [128 x 64] tile
constexpr int AX_KT = AX_KV * 128;                // bytes of a [64 x 64] tile
constexpr int AX_PT = AX_Q * AX_KV * 2;
constexpr int AX_THREADS = 320;                   // loads, products, two threads a query row

struct AttnWideParams {
  const int* blocks;                              // [n][2] = (request, first new token)
  const int* cu_q; const int* kv_lens;
  const int* page_table; int max_pages, num_pages;
  uint16_t* out; long long ld_out;
  const uint16_t* gate; long long ld_gate;        // null: none; else o * sigmoid(gate), laid out like out
  int V, dt, vt, ks, group;
  float scale_log2;
  uint32_t idesc_s, idesc_o;
};

template <bool BF16>
__global__ void __launch_bounds__(AX_THREADS, 1)
attn_wide_kernel(const __grid_constant__ CUtensorMap tmQ, const __grid_constant__ CUtensorMap tmK, const __grid_constant__ CUtensorMap tmV, const AttnWideParams p) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  const int dt = p.dt, vt = p.vt;
  uint8_t* q_smem = smem;                                   // [dt] tiles of 16 KB
  uint8_t* k_smem = q_smem + dt * AX_QT;                    // [2][dt] tiles of 8 KB
  uint8_t* v_smem = k_smem + 2 * dt * AX_KT;                // [2][vt]
  uint8_t* p_smem = v_smem + 2 * vt * AX_KT;                // two terms
  uint64_t* bars = reinterpret_cast<uint64_t*>(p_smem + 2 * AX_PT);
  uint64_t* full_k = bars;            // [2]
  uint64_t* full_v = bars + 2;
  uint64_t* empty_k = bars + 4;
  uint64_t* empty_v = bars + 6;
  uint64_t* s_full = bars + 8;        // [2]
  uint64_t* q_full = bars + 10;
  uint64_t* p_ready = bars + 11;
  uint64_t* o_full = bars + 12;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 13);

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int head = blockIdx.x, kv_head = head / p.group;
  const int req = p.blocks[2 * blockIdx.y], q0 = p.blocks[2 * blockIdx.y + 1];
  const int row0 = p.cu_q[req] + q0, q_len = p.cu_q[req + 1] - p.cu_q[req];
  const int rows = min(AX_Q, q_len - q0), pos0 = p.kv_lens[req] - q_len + q0;
  const int n_steps = rows > 0 && pos0 >= 0 ? (pos0 + rows + AX_KV - 1) / AX_KV : 0;
  bool dead = false;

  if (threadIdx.x == 0) {
    for (int s = 0; s < 2; ++s) { mbar_init(&full_k[s], 1); mbar_init(&full_v[s], 1); mbar_init(&empty_k[s], 1); mbar_init(&empty_v[s], 1); mbar_init(&s_full[s], 1); }
    mbar_init(q_full, 1); mbar_init(p_ready, 256); mbar_init(o_full, 1);
    mbar_init_fence();
    tma_prefetch_desc(&tmQ); tma_prefetch_desc(&tmK); tma_prefetch_desc(&tmV);
  }
  if (warp == 1) { tmem_alloc(tmem_slot, 512); tmem_relinquish(); }
  tc_fence_before_sync();
  __syncthreads();
  tc_fence_after_sync();
  const uint32_t tmem0 = *tmem_slot, tmem_o = tmem0 + 2 * AX_KV;      // S of even and odd steps, then O

  if (warp == 0) {
    if (n_steps > 0 && elect_one()) {
      mbar_expect_tx(q_full, dt * AX_QT);
      for (int j = 0; j < dt; ++j) tma_load_3d(q_smem + j * AX_QT, &tmQ, q_full, j * 64, head, row0);
      for (int it = 0; it < n_steps; ++it) {
        const int s = it & 1, key = it * AX_KV;
        const uint32_t ph = (uint32_t)(it >> 1) & 1u;
        int page = (key >> 7) < p.max_pages ? p.page_table[(size_t)req * p.max_pages + (key >> 7)] : 0;
        if ((unsigned)page >= (unsigned)p.num_pages) { report_error(ERR_BAD_ARG, KID_ATTN_WIDE, 20); page = 0; }
        const int row = page * 128 + (key & 127);
        if (!mbar_wait(&empty_k[s], ph ^ 1u, dead, KID_ATTN_WIDE, 1)) break;
        mbar_expect_tx(&full_k[s], dt * AX_KT);
        for (int j = 0; j < dt; ++j) tma_load_3d(k_smem + (s * dt + j) * AX_KT, &tmK, &full_k[s], j * 64, kv_head, row);
        if (!mbar_wait(&empty_v[s], ph ^ 1u, dead, KID_ATTN_WIDE, 2)) break;
        mbar_expect_tx(&full_v[s], vt * AX_KT);
        for (int j = 0; j < vt; ++j) tma_load_3d(v_smem + (s * vt + j) * AX_KT, &tmV, &full_v[s], j * 64, kv_head, row);
      }
    }
    __syncwarp();
  } else if (warp == 1) {
    if (n_steps > 0 && elect_one()) {
      const uint32_t qb = smem_u32(q_smem), pb = smem_u32(p_smem);
      auto issue_s = [&](int it) {
        const int s = it & 1;
        if (!mbar_wait(&full_k[s], (uint32_t)(it >> 1) & 1u, dead, KID_ATTN_WIDE, 3)) return false;
        tc_fence_after_sync();
        const uint32_t kb = smem_u32(k_smem + s * dt * AX_KT);
        for (int k = 0; k < p.ks; ++k)
          umma_f16(tmem0 + (uint32_t)(s * AX_KV), make_smem_desc(qb + (k >> 2) * AX_QT + (k & 3) * 32, 16, 1024, SWZ_128B),
                   make_smem_desc(kb + (k >> 2) * AX_KT + (k & 3) * 32, 16, 1024, SWZ_128B), p.idesc_s, k != 0 ? 1u : 0u);
        umma_commit(&s_full[s]);
        umma_commit(&empty_k[s]);
        return true;
      };
      bool ok = mbar_wait(q_full, 0, dead, KID_ATTN_WIDE, 4) && issue_s(0);
      for (int it = 0; ok && it < n_steps; ++it) {
        // (the scores of step it - 1, in the buffer that this one takes, were read before its P was announced)
        if (it + 1 < n_steps && !issue_s(it + 1)) break;
        const int s = it & 1;
        if (!mbar_wait(p_ready, (uint32_t)it & 1u, dead, KID_ATTN_WIDE, 5)) break;
        if (!mbar_wait(&full_v[s], (uint32_t)(it >> 1) & 1u, dead, KID_ATTN_WIDE, 6)) break;
        tc_fence_after_sync();
        const uint32_t vb = smem_u32(v_smem + s * vt * AX_KT);
#pragma unroll
        for (int k = 0; k < 8; ++k)                           // 16 keys a product, both terms of P
          umma_f16(tmem_o, make_smem_desc(pb + (k >> 2) * AX_PT + (k & 3) * 32, 16, 1024, SWZ_128B),
                   make_smem_desc(vb + (k & 3) * 2048, AX_KT, 1024, SWZ_128B), p.idesc_o, (it | k) != 0 ? 1u : 0u);
        umma_commit(o_full);
        umma_commit(&empty_v[s]);
      }
    }
    __syncwarp();
  } else {
    const int q = warp & 3, half = (warp - 2) >> 2, r = q * 32 + lane, pos = pos0 + r, b0 = half * (AX_KV / 2);      // keys b0 .. b0 + 31 of a step
    const uint32_t lane_off = (uint32_t)(q * 32) << 16;
    uint8_t* prow = p_smem + r * 128;
    float* rowx = reinterpret_cast<float*>(bars + 16);       // [2][128]
    auto other = [&](float v) {                              // the number of the row's other thread
      rowx[half * AX_Q + r] = v;
      asm volatile("bar.sync %0, 64;\n" ::"r"(1 + q) : "memory");
      v = rowx[(half ^ 1) * AX_Q + r];
      asm volatile("bar.sync %0, 64;\n" ::"r"(1 + q) : "memory");
      return v;
    };
    float m_run = -INFINITY, l_run = 0.f;
    for (int n = 0; n < n_steps; ++n) {
      mbar_wait(&s_full[n & 1], (uint32_t)(n >> 1) & 1u, dead, KID_ATTN_WIDE, 7);
      __syncwarp();
      tc_fence_after_sync();
      uint32_t sr[32];
      tmem_ld_32x32b_x32(tmem0 + (uint32_t)((n & 1) * AX_KV) + lane_off + b0, sr);
      tmem_ld_wait();
      const int kv0 = n * AX_KV;
      if (kv0 + AX_KV - 1 > pos0) {                           // a row of the block does not see the whole step
#pragma unroll
        for (int j = 0; j < 32; ++j)
          if (kv0 + b0 + j > pos) sr[j] = 0xff800000u;
      }
      float mx[4] = {m_run, m_run, m_run, m_run};
#pragma unroll
      for (int j = 0; j < 32; ++j) mx[j & 3] = fmaxf(mx[j & 3], __uint_as_float(sr[j]));
      float m_new = fmaxf(fmaxf(mx[0], mx[1]), fmaxf(mx[2], mx[3]));
      m_new = fmaxf(m_new, other(m_new));
      // (the first key is in step 0: from there on the maximum is finite)
      float alpha = 1.f;
      if ((m_new - m_run) * p.scale_log2 > (BF16 ? 8.f : 2.f)) { alpha = exp2f((m_run - m_new) * p.scale_log2); m_run = m_new; }
      const float m_use = m_run * p.scale_log2 - (BF16 ? 0.f : 13.f);
      // P under the product of the step before: two scores give way to the first and the second terms of their weights
      float la[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
      for (int j = 0; j < 16; ++j) {
        const float p0 = exp2f(fmaf(__uint_as_float(sr[2 * j]), p.scale_log2, -m_use));
        const float p1 = exp2f(fmaf(__uint_as_float(sr[2 * j + 1]), p.scale_log2, -m_use));
        sr[2 * j] = pack_16<BF16>(p0, p1);
        const float2 f = unpack_16<BF16>(sr[2 * j]);
        sr[2 * j + 1] = pack_16<BF16>(p0 - f.x, p1 - f.y);
        la[j & 3] += p0 + p1;
      }
      if (n > 0) {
        mbar_wait(o_full, (uint32_t)(n - 1) & 1u, dead, KID_ATTN_WIDE, 8);      // P may be overwritten, O rescaled
        __syncwarp();
        tc_fence_after_sync();
        if (__any_sync(0xffffffffu, alpha != 1.f)) {
#pragma unroll 1
          for (int c0 = half * 32; c0 < vt * 64; c0 += 64) {
            uint32_t o[32];
            tmem_ld_32x32b_x32(tmem_o + lane_off + c0, o);
            tmem_ld_wait();
#pragma unroll
            for (int j = 0; j < 32; ++j) o[j] = __float_as_uint(__uint_as_float(o[j]) * alpha);
            tmem_st_32x32b_x32(tmem_o + lane_off + c0, o);
          }
          tmem_st_wait();
        }
      }
#pragma unroll
      for (int g = 0; g < 4; ++g) {
        const int at = ((4 * half + g) ^ (r & 7)) << 4;
        *reinterpret_cast<uint4*>(prow + at) = make_uint4(sr[8 * g], sr[8 * g + 2], sr[8 * g + 4], sr[8 * g + 6]);
        *reinterpret_cast<uint4*>(prow + AX_PT + at) = make_uint4(sr[8 * g + 1], sr[8 * g + 3], sr[8 * g + 5], sr[8 * g + 7]);
      }
      l_run = fmaf(l_run, alpha, (la[0] + la[1]) + (la[2] + la[3]));
      if (n == n_steps - 1 && pos0 + rows < kv0 + AX_KV) {
        // keys behind the block's last row have no weight, but what stands there may be no number: their values count as zeros.  (The
        // product of step n - 2, which had this buffer before, was issued ahead of this step's scores: the wait is for this step's values.)
        mbar_wait(&full_v[n & 1], (uint32_t)(n >> 1) & 1u, dead, KID_ATTN_WIDE, 10);
        if (half == 0 && (r & 63) >= pos0 + rows - kv0) {
          uint4* vrow = reinterpret_cast<uint4*>(v_smem + (n & 1) * vt * AX_KT + (r & 63) * 128);
          for (int j = r >> 6; j < vt; j += 2)
#pragma unroll
            for (int e = 0; e < 8; ++e) vrow[j * (AX_KT / 16) + ((e + r) & 7)] = make_uint4(0u, 0u, 0u, 0u);      // (a warp's rows share banks)
        }
      }
      fence_proxy_async_smem();
      tc_fence_before_sync();
      mbar_arrive(p_ready);
    }
    if (n_steps > 0) {
      mbar_wait(o_full, (uint32_t)(n_steps - 1) & 1u, dead, KID_ATTN_WIDE, 9);
      __syncwarp();
      tc_fence_after_sync();
      const float l_sum = l_run + other(l_run);
      const float inv = l_sum > 0.f ? 1.f / l_sum : 0.f;
      const bool live = r < rows;
      uint16_t* orow = p.out + (size_t)(row0 + r) * p.ld_out + (size_t)head * p.V;
      const uint16_t* grow = p.gate != nullptr ? p.gate + (size_t)(row0 + r) * p.ld_gate + (size_t)head * p.V : nullptr;
#pragma unroll 1
      for (int c0 = half * 32; c0 < p.V; c0 += 64) {
        uint32_t o[32];
        __syncwarp();
        tmem_ld_32x32b_x32(tmem_o + lane_off + c0, o);
        tmem_ld_wait();
        if (!live) continue;
#pragma unroll
        for (int g = 0; g < 4; ++g) {
          if (c0 + 8 * g >= p.V) break;
          float v[8];
#pragma unroll
          for (int j = 0; j < 8; ++j) v[j] = __uint_as_float(o[8 * g + j]) * inv;
          if (grow != nullptr) {
            const uint4 gv = *reinterpret_cast<const uint4*>(grow + c0 + 8 * g);
            const uint32_t gu[4] = {gv.x, gv.y, gv.z, gv.w};
#pragma unroll
            for (int j = 0; j < 4; ++j) {
              const float2 f = unpack_16<BF16>(gu[j]);
              v[2 * j] = v[2 * j] / (1.f + __expf(-f.x));
              v[2 * j + 1] = v[2 * j + 1] / (1.f + __expf(-f.y));
            }
          }
          *reinterpret_cast<uint4*>(orow + c0 + 8 * g) = make_uint4(pack_16<BF16>(v[0], v[1]), pack_16<BF16>(v[2], v[3]), pack_16<BF16>(v[4], v[5]), pack_16<BF16>(v[6], v[7]));
        }
      }
    }
  }
  tc_fence_before_sync();
  __syncthreads();
  if (warp == 1) tmem_dealloc(tmem0, 512);
}

}  // namespace fb

using namespace fb;

// q [T, >= H * D] (row stride ld_q), k_pool [num_slots, G, D], v_pool [num_slots, G, V], 128 slots a page; blocks [n_blocks][2] = (request,
// first of up to 128 new tokens); cu_q, kv_lens, page_table as the packed batch has them; out / gate (optional) [T, H * V].
extern "C" int fb_attn_wide(const void* q, long long ld_q, int T, const void* k_pool, const void* v_pool, long long num_slots, const int* page_table, int max_pages,
                            const int* cu_q, const int* kv_lens, void* out, long long ld_out, const void* gate, long long ld_gate, const int* blocks, int n_blocks,
                            int H, int G, int D, int V, float scale, int dtype, void* stream_) {
  if (n_blocks <= 0) return 0;
  if (D <= 0 || V <= 0 || D > 256 || V > 256 || D % 8 != 0 || V % 8 != 0 || T <= 0 || num_slots < 128 || H <= 0 || G <= 0 || H % G != 0 || n_blocks > 65535 ||
      max_pages <= 0 || ld_out % 8 != 0 || ld_gate % 8 != 0 || (dtype != 0 && dtype != 1))
    return -1;
  CUtensorMap tmQ, tmK, tmV;
  if (!make_tmap_3d(&tmQ, q, D, H, T, D, ld_q, 64, AX_Q)) return -2;
  if (!make_tmap_3d(&tmK, k_pool, D, G, num_slots, D, (long long)G * D, 64, AX_KV)) return -2;
  if (!make_tmap_3d(&tmV, v_pool, V, G, num_slots, V, (long long)G * V, 64, AX_KV)) return -2;
  AttnWideParams p = {};
  p.blocks = blocks; p.cu_q = cu_q; p.kv_lens = kv_lens; p.page_table = page_table; p.max_pages = max_pages; p.num_pages = (int)(num_slots / 128);
  p.out = (uint16_t*)out; p.ld_out = ld_out; p.gate = (const uint16_t*)gate; p.ld_gate = ld_gate;
  p.V = V; p.dt = (D + 63) / 64; p.vt = (V + 63) / 64; p.ks = (D + 15) / 16; p.group = H / G;
  p.scale_log2 = scale * 1.4426950408889634f;
  const uint32_t fm = dtype == 1 ? 1u : 0u;
  p.idesc_s = make_idesc(fm, fm, 0, 0, 128, AX_KV);
  p.idesc_o = make_idesc(fm, fm, 0, 1, 128, p.vt * 64);
  const int smem = p.dt * AX_QT + 2 * (p.dt + p.vt) * AX_KT + 2 * AX_PT + 128 + 2 * AX_Q * 4 + 1024;
  static DeviceOnce cfg;
  if (cfg.need()) {
    cudaError_t e = cudaFuncSetAttribute(attn_wide_kernel<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, 227 * 1024);
    if (e == cudaSuccess) e = cudaFuncSetAttribute(attn_wide_kernel<false>, cudaFuncAttributeMaxDynamicSharedMemorySize, 227 * 1024);
    if (e != cudaSuccess) return (int)e;
  }
  cudaStream_t s = reinterpret_cast<cudaStream_t>(stream_);
  if (dtype == 1) attn_wide_kernel<true><<<dim3(H, n_blocks), AX_THREADS, smem, s>>>(tmQ, tmK, tmV, p);
  else attn_wide_kernel<false><<<dim3(H, n_blocks), AX_THREADS, smem, s>>>(tmQ, tmK, tmV, p);
  return (int)cudaGetLastError();
}
