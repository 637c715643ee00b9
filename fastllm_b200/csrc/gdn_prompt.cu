// Gated DeltaNet prompts for sm_100a: the causal convolution over packed sequences and the chunked gated delta rule with the gated RMSNorm
// behind it.  Per value head, with q, k normalised to unit length (q also scaled by 128^-1/2), decay g_t <= 0 and write strength beta_t:
//     S_t = e^(g_t) S_(t-1) + k_t (beta_t (v_t - (e^(g_t) S_(t-1))^T k_t))^T,     o_t = S_t^T q_t.
//
// 64 tokens a chunk, G the running sum of g inside it, S the state it starts from:
//     V' = T (beta v - beta e^G (K S)),   T = (I + A)^-1,   A_ts = beta_t e^(G_t - G_s) (k_t . k_s) for s < t
//     S <- e^(G_last) S + sum_t e^(G_last - G_t) k_t V'_t^T,     o_t = e^(G_t) q_t S + sum_(s <= t) e^(G_t - G_s) (q_t . k_s) V'_s
//  * gdn_chunk_inverse_kernel  gates, norms and T of every (chunk, head), in parallel: K K^T on the tensor core, the unit lower-triangular
//                              inverse by forward substitution, a column per thread in registers.
//  * gdn_chunk_scan_kernel     the chain over the chunks.  Columns of the state never meet: four warps carry 16 of them through all chunks.
//                              S^T stays in registers as accumulator fragments, which are operand fragments of the next product as they
//                              are (the k index of both operands is permuted alike); the chunk's keys and T are fetched a chunk ahead.
//  * gdn_chunk_out_kernel      outputs of every (chunk, head), in parallel, with the norm over the head and the gate in the epilogue.
// Products have fp32 accumulators.  Queries, keys and values are 16-bit numbers and exact (their norms are factors of rows, applied in
// fp32); an fp32 operand of the chain over bf16 keys enters as three bf16 terms, all 24 bits, elsewhere as two tf32 terms (22 bits; fp16 V' three).
// Decays, norms, gates, T and the state are fp32.  The tensor core cuts its sums off instead of rounding them, which adds up where a state forgets
// slowly: in the chain every product of 8 or 16 terms is summed by itself, smallest terms first, and added in fp32.  Error of the states against
// 64 bits over 28 calls of 30 tokens and more: 0.11 to 1.12 of that of fp32 operators, 0.67 in the mean (two tf32 terms and running sums: 2.1 times where
// little is forgotten).
//
// 4001 tokens x 32 heads, bf16: 0.44 ms a layer (convolution 56 us, T 61, chain 198, outputs 126); PyTorch operators took about 1500 launches and 12 ms.
#include "ptx.cuh"
#include "launch.h"

FB_DEFINE_ERROR_API(gdn_prompt)

namespace fb {

constexpr int GP_T = 64;                         // tokens a chunk
constexpr int GP_D = 128;                        // width of keys and of values
constexpr int GP_LDK = GP_D + 8;                 // 16-bit rows of keys / queries: 272 bytes, conflict-free ldmatrix
constexpr int GP_LDT = GP_T + 8;                 // fp32 rows read as pairs: conflict-free
constexpr int GP_VECS = 9;                       // vectors of 64 a (chunk, head), see below
// write strengths; beta e^G / |k|; e^(G_last - G) / |k|; e^G / |q|; the running log2-decay and what its rounding left; 1 / |k|; 128^-1/2 / |q|; e^G_last
enum { GV_BETA, GV_CB, GV_CD, GV_EQ, GV_G, GV_GLO, GV_RK, GV_RQ, GV_LAST };

struct GdnPromptParams {
  const uint16_t* y; long long ld_y;             // [T, 2 Hk 128 + Hv 128] queries | keys | values behind the convolution
  const uint16_t* a; const uint16_t* b; long long ld_ab;       // [T, Hv] decay and write-strength logits
  const uint16_t* z; long long ld_z;             // [T, Hv 128] output gate
  const float* A_log; const float* dt_bias;      // [Hv]
  const uint16_t* norm_w;                        // [128]
  float* state;                                  // [slots, Hv, 128, 128]
  uint16_t* out;                                 // [T, Hv 128]
  const int* chunks;                             // [n_chunks][3] = (first row, rows, state slot in a request's first chunk, else -1)
  const int* reqs;                               // [n_reqs][4] = (first chunk, chunks, state slot, rows)
  float* inv;                                    // [units][64][64]; unit = chunk * Hn + head - h0
  float* vecs;                                   // [units][GP_VECS][64]
  float4* vnew;                                  // [units][8 blocks of 16 v][8 tiles of 8 t][32 lanes], as the accumulators hold them: (v, t), (v, t + 1),
  float4* s0;                                    // (v + 8, t), (v + 8, t + 1) of v = lane / 4, t = 2 (lane % 4); [units][8][16 tiles of 8 d][32]
  int Hk, Hv, h0, Hn;
  float eps;
};

template <bool BF16> __device__ __forceinline__ float gp_ld(uint16_t v) { return BF16 ? __bfloat162float(__ushort_as_bfloat16(v)) : __half2float(__ushort_as_half(v)); }
template <bool BF16> __device__ __forceinline__ uint16_t gp_st(float v) { return BF16 ? __bfloat16_as_ushort(__float2bfloat16_rn(v)) : __half_as_ushort(__float2half_rn(v)); }
__device__ __forceinline__ float gp_ex2(float x) { return exp2f(x); }       // (a chunk's decay multiplies the state once a chunk: its error adds up)
__device__ __forceinline__ float gp_tf32(float x) { uint32_t y; asm("cvt.rna.tf32.f32 %0, %1;\n" : "=r"(y) : "f"(x)); return __uint_as_float(y); }
__device__ __forceinline__ void gp_split(float x, float& hi, float& lo) { hi = gp_tf32(x); lo = gp_tf32(x - hi); }
__device__ __forceinline__ void gp_mma_tf32(float* c, const float* a, float b0, float b1) {
  asm("mma.sync.aligned.m16n8k8.row.col.f32.tf32.tf32.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};\n"
               : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
               : "r"(__float_as_uint(a[0])), "r"(__float_as_uint(a[1])), "r"(__float_as_uint(a[2])), "r"(__float_as_uint(a[3])),
                 "r"(__float_as_uint(b0)), "r"(__float_as_uint(b1)));
}
template <bool BF16>
__device__ __forceinline__ void gp_mma_16(float* c, const uint32_t* a, uint32_t b0, uint32_t b1) {
  if (BF16)
    asm("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};\n"
                 : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3]) : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
  else
    asm("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};\n"
                 : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3]) : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
// the same with a sum that starts at zero
__device__ __forceinline__ void gp_mma0_tf32(float* c, const float* a, float b0, float b1) {
  asm("mma.sync.aligned.m16n8k8.row.col.f32.tf32.tf32.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%10,%10,%10,%10};\n"
      : "=f"(c[0]), "=f"(c[1]), "=f"(c[2]), "=f"(c[3])
      : "r"(__float_as_uint(a[0])), "r"(__float_as_uint(a[1])), "r"(__float_as_uint(a[2])), "r"(__float_as_uint(a[3])),
        "r"(__float_as_uint(b0)), "r"(__float_as_uint(b1)), "f"(0.f));
}
__device__ __forceinline__ void gp_mma0_bf16(float* c, const uint32_t* a, uint32_t b0, uint32_t b1) {
  asm("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%10,%10,%10,%10};\n"
      : "=f"(c[0]), "=f"(c[1]), "=f"(c[2]), "=f"(c[3]) : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1), "f"(0.f));
}
__device__ __forceinline__ void gp_add4(float* c, const float* t) {
  unpack_f32x2(add_f32x2(pack_f32x2(c[0], c[1]), pack_f32x2(t[0], t[1])), c[0], c[1]);
  unpack_f32x2(add_f32x2(pack_f32x2(c[2], c[3]), pack_f32x2(t[2], t[3])), c[2], c[3]);
}
// Two fp32 numbers as three bf16 terms each: all 24 bits.
__device__ __forceinline__ void gp_split_bf16(float x, float y, uint32_t& hi, uint32_t& mid, uint32_t& lo) {
  hi = pack_16<true>(x, y);
  const float2 f = unpack_16<true>(hi);
  x -= f.x; y -= f.y;
  mid = pack_16<true>(x, y);
  const float2 g = unpack_16<true>(mid);
  lo = pack_16<true>(x - g.x, y - g.y);
}
__device__ __forceinline__ void gp_ldsm4(uint32_t* r, const uint16_t* p) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];\n" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(smem_u32(p)) : "memory");
}
__device__ __forceinline__ void gp_ldsm4_t(uint32_t* r, const uint16_t* p) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];\n" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(smem_u32(p)) : "memory");
}
// 16 bytes global -> shared; `ok` false: zeros
__device__ __forceinline__ void gp_cp16(void* dst, const void* src, bool ok) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(smem_u32(dst)), "l"(src), "r"(ok ? 16 : 0) : "memory");
}
__device__ __forceinline__ void gp_cp_commit() { asm volatile("cp.async.commit_group;\n" ::: "memory"); }
template <int N> __device__ __forceinline__ void gp_cp_wait() { asm volatile("cp.async.wait_group %0;\n" ::"n"(N) : "memory"); }

// s / (1 + e^-s): the approximate reciprocal and one Newton step, within an fp32 rounding of the division.  (4001 x 8192 channels with the launch:
// 73 us; __expf and __fdividef 52 us, but 1.14 times as many results on the wrong 16-bit neighbour as fp32 operators; expf and a division 92 us.)
__device__ __forceinline__ float gp_silu(float s) {
  const float d = 1.f + expf(fminf(-s, 87.f));
  float y;
  asm("rcp.approx.ftz.f32 %0, %1;\n" : "=f"(y) : "f"(d));
  return s * fmaf(y, fmaf(-d, y, 1.f), y);
}

// ------------------------------------------------------------------------------------------------
// causal depth-wise convolution of four taps + SiLU.  A thread takes 8 channels of 16 tokens: bound by the rows it reads and writes once
// (4001 x 8192 channels: 131 MB).  The requests' windows are advanced by the kernel behind it, which this one must not overtake.
// ------------------------------------------------------------------------------------------------
constexpr int GP_CT = 16;
template <bool BF16>
__global__ void __launch_bounds__(256) gdn_conv_prompt_kernel(const uint16_t* __restrict__ x, long long ldx, const uint16_t* __restrict__ w,
                                                              const uint16_t* __restrict__ state, const int* __restrict__ chunks, uint16_t* __restrict__ out, int C) {
  pdl_launch_dependents();
  pdl_wait();
  const int c8 = blockIdx.x * 256 + threadIdx.x;
  const int* ch = chunks + 3 * blockIdx.y;
  const int row0 = ch[0], n = ch[1], slot = ch[2], t0 = blockIdx.z * GP_CT;
  if (c8 * 8 >= C || t0 >= n) return;
  float wf[8][4];
  {
    const uint4* wp = reinterpret_cast<const uint4*>(w + (size_t)c8 * 32);
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const uint4 v = wp[i];
      const uint32_t u[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
      for (int j = 0; j < 4; ++j) { const float2 f = unpack_16<BF16>(u[j]); wf[2 * i + (j >> 1)][2 * (j & 1)] = f.x; wf[2 * i + (j >> 1)][2 * (j & 1) + 1] = f.y; }
    }
  }
  float win[3][8];
  const bool first = slot >= 0 && t0 == 0;
#pragma unroll
  for (int j = 0; j < 3; ++j) {
    if (first) {
      const uint16_t* sp = state + ((size_t)slot * C + c8 * 8) * 3 + j;
#pragma unroll
      for (int e = 0; e < 8; ++e) win[j][e] = gp_ld<BF16>(sp[3 * e]);
    } else {
      const uint4 v = *reinterpret_cast<const uint4*>(x + (size_t)(row0 + t0 - 3 + j) * ldx + c8 * 8);
      const uint32_t u[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
      for (int e = 0; e < 4; ++e) { const float2 f = unpack_16<BF16>(u[e]); win[j][2 * e] = f.x; win[j][2 * e + 1] = f.y; }
    }
  }
  const int cnt = min(GP_CT, n - t0);
#pragma unroll 4
  for (int t = 0; t < cnt; ++t) {
    const uint4 v = *reinterpret_cast<const uint4*>(x + (size_t)(row0 + t0 + t) * ldx + c8 * 8);
    const uint32_t u[4] = {v.x, v.y, v.z, v.w};
    uint32_t o[4];
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      const float2 f = unpack_16<BF16>(u[e]);
      const float in[2] = {f.x, f.y};
      float r[2];
#pragma unroll
      for (int k = 0; k < 2; ++k) {
        const int c = 2 * e + k;
        const float s = fmaf(in[k], wf[c][3], fmaf(win[2][c], wf[c][2], fmaf(win[1][c], wf[c][1], win[0][c] * wf[c][0])));
        win[0][c] = win[1][c]; win[1][c] = win[2][c]; win[2][c] = in[k];
        r[k] = gp_silu(s);
      }
      o[e] = pack_16<BF16>(r[0], r[1]);
    }
    *reinterpret_cast<uint4*>(out + (size_t)(row0 + t0 + t) * C + c8 * 8) = make_uint4(o[0], o[1], o[2], o[3]);
  }
}

// the last three inputs of every request become its window
__global__ void __launch_bounds__(256) gdn_conv_state_kernel(const uint16_t* __restrict__ x, long long ldx, uint16_t* state, const int* __restrict__ chunks,
                                                             const int* __restrict__ reqs, int C) {
  const int c = blockIdx.x * 256 + threadIdx.x;
  if (c >= C) return;
  const int* rq = reqs + 4 * blockIdx.y;
  const int row0 = chunks[3 * rq[0]], n = rq[3];
  uint16_t* sp = state + ((size_t)rq[2] * C + c) * 3;
  const uint16_t h[3] = {sp[0], sp[1], sp[2]};
  uint16_t o[3];
#pragma unroll
  for (int j = 0; j < 3; ++j) {
    const int i = n + j;                          // place in [window | new inputs]
    o[j] = i < 3 ? h[i] : x[(size_t)(row0 + i - 3) * ldx + c];
  }
#pragma unroll
  for (int j = 0; j < 3; ++j) sp[j] = o[j];
}

// ------------------------------------------------------------------------------------------------
// gates, norms and T
// ------------------------------------------------------------------------------------------------
template <bool BF16>
__global__ void __launch_bounds__(128) gdn_chunk_inverse_kernel(const GdnPromptParams p) {
  __shared__ __align__(16) uint16_t ks[GP_T * GP_LDK];
  __shared__ __align__(16) float As[GP_T * (GP_T + 4)];
  __shared__ float sg[GP_T], sl[GP_T], sb[GP_T], rk[GP_T], rq[GP_T];
  __shared__ double part;
  constexpr int LDA = GP_T + 4;
  const int c = blockIdx.x, hl = blockIdx.y, h = p.h0 + hl, hk = h / (p.Hv / p.Hk);
  const int row0 = p.chunks[3 * c], n = p.chunks[3 * c + 1];
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const uint16_t* q0 = p.y + (size_t)row0 * p.ld_y + hk * GP_D;
  const uint16_t* k0 = q0 + p.Hk * GP_D;
  // half a warp a row: its keys into shared memory, squares of keys and queries
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    const int t = i * 8 + (tid >> 4), col = (tid & 15) * 8;
    uint4 kv = make_uint4(0u, 0u, 0u, 0u), qv = kv;
    if (t < n) {
      kv = *reinterpret_cast<const uint4*>(k0 + (size_t)t * p.ld_y + col);
      qv = *reinterpret_cast<const uint4*>(q0 + (size_t)t * p.ld_y + col);
    }
    *reinterpret_cast<uint4*>(ks + t * GP_LDK + col) = kv;
    float sk = 0.f, sq = 0.f;
    const uint32_t ku[4] = {kv.x, kv.y, kv.z, kv.w}, qu[4] = {qv.x, qv.y, qv.z, qv.w};
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      const float2 a = unpack_16<BF16>(ku[e]), b = unpack_16<BF16>(qu[e]);
      sk = fmaf(a.x, a.x, fmaf(a.y, a.y, sk));
      sq = fmaf(b.x, b.x, fmaf(b.y, b.y, sq));
    }
#pragma unroll
    for (int o = 8; o > 0; o >>= 1) { sk += __shfl_xor_sync(0xffffffffu, sk, o); sq += __shfl_xor_sync(0xffffffffu, sq, o); }
    if ((tid & 15) == 0) { rk[t] = 1.0f / sqrtf(sk + 1e-6f); rq[t] = 0.08838834764831845f / sqrtf(sq + 1e-6f); }
  }
  // running log2-decay, one token a thread; in 64 bits, for decays are exponentials of its differences (after 64 tokens that forget nearly
  // everything an fp32 sum has units of 2^-15)
  double G = 0.0;
  float beta = 0.f;
  if (tid < GP_T) {
    if (tid < n) {
      const size_t at = (size_t)(row0 + tid) * p.ld_ab + h;
      const float x = gp_ld<BF16>(p.a[at]) + p.dt_bias[h];
      G = (double)(-expf(p.A_log[h]) * (x > 20.f ? x : log1pf(expf(x)))) * 1.4426950408889634;
      beta = 1.0f / (1.0f + expf(-gp_ld<BF16>(p.b[at])));
    }
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) { const double u = __shfl_up_sync(0xffffffffu, G, o); if (lane >= o) G += u; }
    if (tid == 31) part = G;
  }
  __syncthreads();
  if (tid < GP_T) {
    if (warp == 1) G += part;
    sg[tid] = (float)G;
    sl[tid] = (float)(G - (double)sg[tid]);
    sb[tid] = beta;
  }
  __syncthreads();
  const size_t unit = (size_t)c * p.Hn + hl;
  if (tid < GP_T) {
    float* v = p.vecs + unit * GP_VECS * GP_T + tid;
    const double last = (double)sg[GP_T - 1] + (double)sl[GP_T - 1];
    const float eG = gp_ex2((float)G);
    v[GV_BETA * GP_T] = beta;
    v[GV_CB * GP_T] = beta * eG * rk[tid];
    v[GV_CD * GP_T] = rk[tid] * gp_ex2((float)(last - G));
    v[GV_EQ * GP_T] = rq[tid] * eG;
    v[GV_G * GP_T] = sg[tid];
    v[GV_GLO * GP_T] = sl[tid];
    v[GV_RK * GP_T] = rk[tid];
    v[GV_RQ * GP_T] = rq[tid];
    v[GV_LAST * GP_T] = gp_ex2((float)last);
  }
  // A, a warp 16 rows of it up to the diagonal
  {
    const int m0 = warp * 16, g = lane >> 2, q = lane & 3;
    uint32_t a[8][4];
#pragma unroll
    for (int kk = 0; kk < 8; ++kk) gp_ldsm4(a[kk], ks + (m0 + (lane & 15)) * GP_LDK + kk * 16 + (lane >> 4) * 8);
    for (int nt = 0; nt < 8; ++nt) {
      float acc[4] = {0.f, 0.f, 0.f, 0.f};
      if (nt <= 2 * warp + 1) {
#pragma unroll
        for (int kk = 0; kk < 8; kk += 2) {
          uint32_t b[4];
          gp_ldsm4(b, ks + (nt * 8 + (lane & 7)) * GP_LDK + kk * 16 + (lane >> 3) * 8);
          float t[4] = {0.f, 0.f, 0.f, 0.f}, v[4] = {0.f, 0.f, 0.f, 0.f};
          gp_mma_16<BF16>(t, a[kk], b[0], b[1]);
          gp_mma_16<BF16>(v, a[kk + 1], b[2], b[3]);
          gp_add4(t, v);
          gp_add4(acc, t);
        }
      }
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const int i = m0 + g + 8 * (e >> 1), j = nt * 8 + 2 * q + (e & 1);
        As[i * LDA + j] = j < i ? acc[e] * (sb[i] * rk[i]) * (rk[j] * gp_ex2((sg[i] - sg[j]) + (sl[i] - sl[j]))) : 0.f;
      }
    }
  }
  __syncthreads();
  if (tid < GP_T) {
    float t[GP_T];
    float* dst = p.inv + unit * GP_T * GP_T + tid;
#pragma unroll
    for (int i = 0; i < GP_T; ++i) {
      float s[4] = {i == tid ? 1.f : 0.f, 0.f, 0.f, 0.f};
#pragma unroll
      for (int j = 0; j < i; j += 4) {
        const float4 a = *reinterpret_cast<const float4*>(As + i * LDA + j);        // (zeros from column i on)
        s[0] = fmaf(-a.x, t[j], s[0]);
        if (j + 1 < i) s[1] = fmaf(-a.y, t[j + 1], s[1]);
        if (j + 2 < i) s[2] = fmaf(-a.z, t[j + 2], s[2]);
        if (j + 3 < i) s[3] = fmaf(-a.w, t[j + 3], s[3]);
      }
      t[i] = (s[0] + s[1]) + (s[2] + s[3]);
      dst[i * GP_T] = t[i];
    }
  }
}

// ------------------------------------------------------------------------------------------------
// the chain over a request's chunks: a CTA of eight warps takes 32 columns of a head's state, four warps 16 of them: each carries 32 of the 128 key
// channels.  They add up K S, a warp two of the eight token tiles, share out the columns of T's product (token tiles f and 7 - f: equal parts of its
// triangle) and exchange V', three times a chunk through shared memory.  Bound by the chain of a chunk: a warp issues 150 products of the tensor core and
// about 1000 instructions a chunk, two warps share a sub-core, and shared memory is busy half of the time.  Chain of 4001 tokens x 32 heads: 261 us with
// two warps per 16 columns, 229 with four, 207 with eight sums in flight between a product and the next one of its own sum, 198 with the state and V' stored as
// the accumulators hold them.  8 requests of 1000 tokens: 311 -> 284 us with the last two.
// ------------------------------------------------------------------------------------------------
constexpr int GS_THREADS = 256;
constexpr int GS_LDV = 40;
constexpr int GS_K = GP_T * GP_LDK * 2, GS_T = GP_T * GP_LDT * 4, GS_V = GP_T * GS_LDV * 2, GS_VEC = 3 * GP_T * 4;
constexpr int GS_STAGE = GS_K + GS_T + GS_V + GS_VEC;
constexpr int GS_STAGES = 2;
constexpr int GS_TILE = 32 * 16;                                  // bytes of a 16 x 8 fp32 tile as fragments
constexpr int GS_PART = 3 * 8 * GS_TILE;                          // of four warps: the partial sums of three others for every tile
constexpr int GS_SMEM = GS_STAGES * GS_STAGE + 2 * GS_PART;

template <bool BF16>
__global__ void __launch_bounds__(GS_THREADS, 2) gdn_chunk_scan_kernel(const GdnPromptParams p) {
  extern __shared__ __align__(16) uint8_t gs_smem[];
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, g = lane >> 2, q = lane & 3;
  const int four = warp >> 2, f = warp & 3, d0 = f * 32;
  const int hl = blockIdx.y, h = p.h0 + hl, hk = h / (p.Hv / p.Hk), v0 = blockIdx.x * 32;
  // [3][4 warps][2 tiles][32 lanes]: what three other warps have summed for a warp's tiles; once it has read them, the first third takes its rows of the
  // right-hand side and, after the barrier behind that, the rest takes V'
  float4* part = reinterpret_cast<float4*>(gs_smem + GS_STAGES * GS_STAGE + four * GS_PART) + lane;
  float4* vx = part + 8 * 32;
  auto meet = [&]() { asm volatile("bar.sync %0, 128;\n" ::"r"(1 + four) : "memory"); };
  const int* rq = p.reqs + 4 * blockIdx.z;
  const int c0 = rq[0], nc = rq[1], slot = rq[2];
  int row0 = p.chunks[3 * c0], n = p.chunks[3 * c0 + 1];           // of the chunk to be fetched next
  auto fetch = [&](int i) {
    uint8_t* st = gs_smem + (i % GS_STAGES) * GS_STAGE;
    const int c = c0 + i;
    const size_t unit = (size_t)c * p.Hn + hl;
    const uint16_t* kp = p.y + (size_t)row0 * p.ld_y + (p.Hk + hk) * GP_D;
    const uint16_t* vp = p.y + (size_t)row0 * p.ld_y + (size_t)2 * p.Hk * GP_D + (size_t)h * GP_D + v0;
    const float* tp = p.inv + unit * GP_T * GP_T;
    const float* gp = p.vecs + unit * GP_VECS * GP_T;
#pragma unroll
    for (int j = tid; j < GP_T * 16; j += GS_THREADS) {
      const int t = j >> 4, u = j & 15;
      gp_cp16(st + (t * GP_LDK + u * 8) * 2, kp + (size_t)(t < n ? t : 0) * p.ld_y + u * 8, t < n);
      gp_cp16(st + GS_K + (t * GP_LDT + u * 4) * 4, tp + t * GP_T + u * 4, true);
    }
    {
      const int t = tid >> 2, u = tid & 3;
      gp_cp16(st + GS_K + GS_T + (t * GS_LDV + u * 8) * 2, vp + (size_t)(t < n ? t : 0) * p.ld_y + u * 8, t < n);
    }
    if (tid < 48) gp_cp16(st + GS_K + GS_T + GS_V + tid * 16, gp + tid * 4, true);           // beta, cb, cd
    if (i + 1 < nc) { row0 = p.chunks[3 * c + 3]; n = p.chunks[3 * c + 4]; }
  };
  float s[4][4];                                  // S^T: rows v = g, g + 8, columns d = d0 + 8 i + 2 q, + 1
  float* S = p.state + ((size_t)slot * p.Hv + h) * GP_D * GP_D + (size_t)d0 * GP_D + v0 + four * 16;
#pragma unroll
  for (int i = 0; i < 4; ++i)
#pragma unroll
    for (int e = 0; e < 4; ++e) s[i][e] = S[(size_t)(8 * i + 2 * q + (e & 1)) * GP_D + g + 8 * (e >> 1)];
  fetch(0);
  gp_cp_commit();
  for (int i = 0; i < nc; ++i) {
    gp_cp_wait<0>();
    __syncthreads();                              // this chunk is there for all, and the other stage and the exchanged parts are done with
    if (i + 1 < nc) fetch(i + 1);
    gp_cp_commit();
    const uint8_t* st = gs_smem + (i % GS_STAGES) * GS_STAGE;
    const uint16_t* ks = reinterpret_cast<const uint16_t*>(st) + d0;
    const float* ts = reinterpret_cast<const float*>(st + GS_K);
    const uint16_t* vs = reinterpret_cast<const uint16_t*>(st + GS_K + GS_T);
    const float* vec = reinterpret_cast<const float*>(st + GS_K + GS_T + GS_V);
    const size_t unit = (size_t)(c0 + i) * p.Hn + hl;
    const float last = __ldg(p.vecs + (unit * GP_VECS + GV_LAST) * GP_T);
    const int vb = blockIdx.x * 2 + four;
    float4* s0 = p.s0 + (unit * 128 + vb * 16 + f * 4) * 32 + lane;
#pragma unroll
    for (int j = 0; j < 4; ++j) s0[j * 32] = make_float4(s[j][0], s[j][1], s[j][2], s[j][3]);
    // (K S)^T [16 v x 64 t] over this warp's channels
    float r[8][4];
    if (BF16) {
#pragma unroll
      for (int kk = 0; kk < 2; ++kk) {
        uint32_t hi[4], mid[4], lo[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) gp_split_bf16(s[2 * kk + (i >> 1)][2 * (i & 1)], s[2 * kk + (i >> 1)][2 * (i & 1) + 1], hi[i], mid[i], lo[i]);
        uint32_t b[4][4];
#pragma unroll
        for (int j = 0; j < 4; ++j) gp_ldsm4(b[j], ks + (8 * (2 * j + (lane >> 4)) + (lane & 7)) * GP_LDK + kk * 16 + ((lane >> 3) & 1) * 8);
        float t[8][4];                            // (eight sums at a time: a product waits for the one before it of its own sum)
#pragma unroll
        for (int j = 0; j < 8; ++j) gp_mma0_bf16(t[j], lo, b[j >> 1][2 * (j & 1)], b[j >> 1][2 * (j & 1) + 1]);
#pragma unroll
        for (int j = 0; j < 8; ++j) gp_mma_16<true>(t[j], mid, b[j >> 1][2 * (j & 1)], b[j >> 1][2 * (j & 1) + 1]);
#pragma unroll
        for (int j = 0; j < 8; ++j) gp_mma_16<true>(t[j], hi, b[j >> 1][2 * (j & 1)], b[j >> 1][2 * (j & 1) + 1]);
#pragma unroll
        for (int j = 0; j < 8; ++j) {
          if (kk == 0) { r[j][0] = t[j][0]; r[j][1] = t[j][1]; r[j][2] = t[j][2]; r[j][3] = t[j][3]; }
          else gp_add4(r[j], t[j]);
        }
      }
    } else {
#pragma unroll
      for (int kk = 0; kk < 4; ++kk) {
        float hi[4], lo[4];
        gp_split(s[kk][0], hi[0], lo[0]); gp_split(s[kk][2], hi[1], lo[1]); gp_split(s[kk][1], hi[2], lo[2]); gp_split(s[kk][3], hi[3], lo[3]);
        uint32_t b[8];
        gp_ldsm4(b, ks + lane * GP_LDK + kk * 8);
        gp_ldsm4(b + 4, ks + (32 + lane) * GP_LDK + kk * 8);
#pragma unroll
        for (int j = 0; j < 8; ++j) {
          const float2 k2 = unpack_16<BF16>(b[j]);
          float t[4];
          gp_mma0_tf32(t, lo, k2.x, k2.y);
          gp_mma_tf32(t, hi, k2.x, k2.y);
          if (kk == 0) { r[j][0] = t[0]; r[j][1] = t[1]; r[j][2] = t[2]; r[j][3] = t[3]; }
          else gp_add4(r[j], t);
        }
      }
    }
    float own[2][4];
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      const int to = j < 4 ? j : 7 - j, x = j >> 2;
      if (to == f) { own[x][0] = r[j][0]; own[x][1] = r[j][1]; own[x][2] = r[j][2]; own[x][3] = r[j][3]; }
      else part[((((f - to - 1) & 3) * 4 + to) * 2 + x) * 32] = make_float4(r[j][0], r[j][1], r[j][2], r[j][3]);
    }
    meet();
#pragma unroll
    for (int x = 0; x < 2; ++x) {
      const int t = 8 * (x == 0 ? f : 7 - f) + 2 * q;
      float4* pt = part + (f * 2 + x) * 32;
      const float4 a = pt[0], b = pt[8 * 32], c = pt[16 * 32];
      const float2 be = *reinterpret_cast<const float2*>(vec + t), cb = *reinterpret_cast<const float2*>(vec + GP_T + t);
      const uint16_t* vp = vs + t * GS_LDV + four * 16 + g;
      float4 o;
      o.x = fmaf(-cb.x, (own[x][0] + a.x) + (b.x + c.x), be.x * gp_ld<BF16>(vp[0]));
      o.y = fmaf(-cb.y, (own[x][1] + a.y) + (b.y + c.y), be.y * gp_ld<BF16>(vp[GS_LDV]));
      o.z = fmaf(-cb.x, (own[x][2] + a.z) + (b.z + c.z), be.x * gp_ld<BF16>(vp[8]));
      o.w = fmaf(-cb.y, (own[x][3] + a.w) + (b.w + c.w), be.y * gp_ld<BF16>(vp[GS_LDV + 8]));
      pt[0] = o;
    }
    meet();
    // V'^T = (right-hand side)^T T^T: token tiles f and 7 - f, 9 products of the triangle
    float w[2][4], wl[2][4], wm[2][4];            // products of first terms, the others'
#pragma unroll
    for (int x = 0; x < 2; ++x)
#pragma unroll
      for (int e = 0; e < 4; ++e) w[x][e] = wl[x][e] = wm[x][e] = 0.f;
#pragma unroll
    for (int kk = 0; kk < 8; ++kk) {
      if (kk > 7 - f) break;
      const float4 rv = part[((kk < 4 ? kk : 7 - kk) * 2 + (kk >> 2)) * 32];
      float hi[4], lo[4];
      gp_split(rv.x, hi[0], lo[0]); gp_split(rv.z, hi[1], lo[1]); gp_split(rv.y, hi[2], lo[2]); gp_split(rv.w, hi[3], lo[3]);
#pragma unroll
      for (int x = 0; x < 2; ++x) {
        if (x == 0 && kk > f) continue;
        const float2 tv = *reinterpret_cast<const float2*>(ts + (8 * (x == 0 ? f : 7 - f) + g) * GP_LDT + 8 * kk + 2 * q);
        float bh0, bl0, bh1, bl1;
        gp_split(tv.x, bh0, bl0);
        gp_split(tv.y, bh1, bl1);
        float t[4];
        gp_mma0_tf32(t, hi, bh0, bh1);
        gp_add4(w[x], t);
        gp_mma_tf32(wl[x], lo, bh0, bh1);
        gp_mma_tf32(wm[x], hi, bl0, bl1);
      }
    }
    float4* vn = p.vnew + (unit * 64 + vb * 8) * 32 + lane;
#pragma unroll
    for (int x = 0; x < 2; ++x) {
      const int tile = x == 0 ? f : 7 - f;
      gp_add4(wl[x], wm[x]);
      gp_add4(w[x], wl[x]);
      vn[tile * 32] = make_float4(w[x][0], w[x][1], w[x][2], w[x][3]);
      const float2 cd = *reinterpret_cast<const float2*>(vec + 2 * GP_T + 8 * tile + 2 * q);
      const float4 wd = make_float4(w[x][0] * cd.x, w[x][1] * cd.y, w[x][2] * cd.x, w[x][3] * cd.y);
      if (BF16) {                                 // half of a 16-token operand, in its three terms: [4 pairs of tiles][3][32 lanes]
        uint32_t hi[2], mid[2], lo[2];
        gp_split_bf16(wd.x, wd.y, hi[0], mid[0], lo[0]);
        gp_split_bf16(wd.z, wd.w, hi[1], mid[1], lo[1]);
        uint2* o = reinterpret_cast<uint2*>(vx + (tile >> 1) * 3 * 32) + (tile & 1);
        o[0] = make_uint2(hi[0], hi[1]); o[64] = make_uint2(mid[0], mid[1]); o[128] = make_uint2(lo[0], lo[1]);
      } else {
        vx[tile * 32] = wd;
      }
    }
    meet();
    // S^T <- e^(G_last) S^T + (decayed V')^T K
    float u[4][4];
    if (BF16) {
#pragma unroll
      for (int c = 0; c < 4; ++c) {               // 16 tokens
        const uint4 h4 = *reinterpret_cast<const uint4*>(vx + c * 96), m4 = *reinterpret_cast<const uint4*>(vx + c * 96 + 32),
                    l4 = *reinterpret_cast<const uint4*>(vx + c * 96 + 64);
        const uint32_t hi[4] = {h4.x, h4.y, h4.z, h4.w}, mid[4] = {m4.x, m4.y, m4.z, m4.w}, lo[4] = {l4.x, l4.y, l4.z, l4.w};
        uint32_t b[2][4];
#pragma unroll
        for (int j = 0; j < 2; ++j) gp_ldsm4_t(b[j], ks + (16 * c + (lane & 15)) * GP_LDK + (2 * j + (lane >> 4)) * 8);
        float t[4][4];
#pragma unroll
        for (int j = 0; j < 4; ++j) gp_mma0_bf16(t[j], lo, b[j >> 1][2 * (j & 1)], b[j >> 1][2 * (j & 1) + 1]);
#pragma unroll
        for (int j = 0; j < 4; ++j) gp_mma_16<true>(t[j], mid, b[j >> 1][2 * (j & 1)], b[j >> 1][2 * (j & 1) + 1]);
#pragma unroll
        for (int j = 0; j < 4; ++j) gp_mma_16<true>(t[j], hi, b[j >> 1][2 * (j & 1)], b[j >> 1][2 * (j & 1) + 1]);
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          if (c == 0) { u[j][0] = t[j][0]; u[j][1] = t[j][1]; u[j][2] = t[j][2]; u[j][3] = t[j][3]; }
          else gp_add4(u[j], t[j]);
        }
      }
    } else {
#pragma unroll
      for (int kk = 0; kk < 8; ++kk) {
        const float4 wv = vx[kk * 32];
        float hi[4], mid[4], lo[4];
        const float wd[4] = {wv.x, wv.z, wv.y, wv.w};
#pragma unroll
        for (int i = 0; i < 4; ++i) { gp_split(wd[i], hi[i], mid[i]); lo[i] = gp_tf32((wd[i] - hi[i]) - mid[i]); }
        uint32_t b[4];
        gp_ldsm4_t(b, ks + (8 * kk + (lane & 7)) * GP_LDK + (lane >> 3) * 8);
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          const float2 k2 = unpack_16<BF16>(b[e]);
          float t[4];
          gp_mma0_tf32(t, lo, k2.x, k2.y);
          gp_mma_tf32(t, mid, k2.x, k2.y);
          gp_mma_tf32(t, hi, k2.x, k2.y);
          if (kk == 0) { u[e][0] = t[0]; u[e][1] = t[1]; u[e][2] = t[2]; u[e][3] = t[3]; }
          else gp_add4(u[e], t);
        }
      }
    }
#pragma unroll
    for (int j = 0; j < 4; ++j)
#pragma unroll
      for (int e = 0; e < 4; ++e) s[j][e] = fmaf(s[j][e], last, u[j][e]);
  }
#pragma unroll
  for (int i = 0; i < 4; ++i)
#pragma unroll
    for (int e = 0; e < 4; ++e) S[(size_t)(8 * i + 2 * q + (e & 1)) * GP_D + g + 8 * (e >> 1)] = s[i][e];
}

// ------------------------------------------------------------------------------------------------
// outputs of a chunk: warps 2 x 4 over (32 tokens, 32 columns).  The state comes in quarters of 32 channels and V' in halves of 32 tokens through a ring of
// three buffers, two ahead of the products; two CTAs share an SM.  Bound by the issue of instructions (splits into tf32 terms, the gate).  4001 tokens x 32 heads:
// 160 us with one buffer that every step waited for, 147 with the ring, 126 with gates read ahead and without exact exponentials and divisions.
// ------------------------------------------------------------------------------------------------
constexpr int GO_THREADS = 256;
constexpr int GO_QK = GP_T * GP_LDK * 2, GO_P = GP_T * GP_LDT * 4, GO_B = 8 * 4 * 32 * 16, GO_RING = 3;
constexpr int GO_SMEM = 2 * GO_QK + GO_P + GO_RING * GO_B + GP_T * 4 * 4;

template <bool BF16>
__global__ void __launch_bounds__(GO_THREADS, 2) gdn_chunk_out_kernel(const GdnPromptParams p) {
  extern __shared__ __align__(16) uint8_t go_smem[];
  uint16_t* qs = reinterpret_cast<uint16_t*>(go_smem);
  uint16_t* ks = reinterpret_cast<uint16_t*>(go_smem + GO_QK);
  float* Ps = reinterpret_cast<float*>(go_smem + 2 * GO_QK);
  float4* Bs = reinterpret_cast<float4*>(go_smem + 2 * GO_QK + GO_P);             // [3][8 blocks of 16 v][4 tiles of 8][32 lanes]
  float* red = reinterpret_cast<float*>(go_smem + 2 * GO_QK + GO_P + GO_RING * GO_B);       // [64][4]
  const int c = blockIdx.x, hl = blockIdx.y, h = p.h0 + hl, hk = h / (p.Hv / p.Hk);
  const int row0 = p.chunks[3 * c], n = p.chunks[3 * c + 1];
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, g = lane >> 2, q = lane & 3;
  const size_t unit = (size_t)c * p.Hn + hl;
  const float* vec = p.vecs + unit * GP_VECS * GP_T;
  const uint16_t* qp = p.y + (size_t)row0 * p.ld_y + hk * GP_D;
  for (int j = tid; j < GP_T * 16; j += GO_THREADS) {
    const int t = j >> 4, u = j & 15;
    const uint16_t* src = qp + (size_t)(t < n ? t : 0) * p.ld_y + u * 8;
    gp_cp16(qs + t * GP_LDK + u * 8, src, t < n);
    gp_cp16(ks + t * GP_LDK + u * 8, src + p.Hk * GP_D, t < n);
  }
  gp_cp_commit();
  const float4 *s0 = p.s0 + unit * 128 * 32, *vnew = p.vnew + unit * 64 * 32;
  auto fetch = [&](int step) {                    // quarters of the state, then halves of V'
    const float4* src = step < 4 ? s0 + step * 128 : vnew + (step - 4) * 128;
    const int ld = step < 4 ? 16 * 32 : 8 * 32;
#pragma unroll
    for (int j = tid; j < 8 * 128; j += GO_THREADS) gp_cp16(Bs + (step % GO_RING) * 1024 + j, src + (j >> 7) * ld + (j & 127), true);
    gp_cp_commit();
  };
  fetch(0);
  fetch(1);
  gp_cp_wait<2>();
  __syncthreads();
  {                                               // decayed scores, 16 tokens x 32 keys a warp
    const int m0 = (warp & 3) * 16, n0 = (warp >> 2) * 4;
    uint32_t a[8][4];
#pragma unroll
    for (int kk = 0; kk < 8; ++kk) gp_ldsm4(a[kk], qs + (m0 + (lane & 15)) * GP_LDK + kk * 16 + (lane >> 4) * 8);
    const float gi[2] = {__ldg(vec + GV_G * GP_T + m0 + g), __ldg(vec + GV_G * GP_T + m0 + g + 8)};
    const float li[2] = {__ldg(vec + GV_GLO * GP_T + m0 + g), __ldg(vec + GV_GLO * GP_T + m0 + g + 8)};
    const float ri[2] = {__ldg(vec + GV_RQ * GP_T + m0 + g), __ldg(vec + GV_RQ * GP_T + m0 + g + 8)};
#pragma unroll
    for (int x = 0; x < 4; ++x) {
      const int nt = n0 + x;
      float acc[4] = {0.f, 0.f, 0.f, 0.f};
      if (nt * 8 < m0 + 16) {
#pragma unroll
        for (int kk = 0; kk < 8; kk += 2) {
          uint32_t b[4];
          gp_ldsm4(b, ks + (nt * 8 + (lane & 7)) * GP_LDK + kk * 16 + (lane >> 3) * 8);
          gp_mma_16<BF16>(acc, a[kk], b[0], b[1]);
          gp_mma_16<BF16>(acc, a[kk + 1], b[2], b[3]);
        }
      }
      const int j = nt * 8 + 2 * q;
      const float2 lj = __ldg(reinterpret_cast<const float2*>(vec + GV_GLO * GP_T + j));
      const float2 gj = __ldg(reinterpret_cast<const float2*>(vec + GV_G * GP_T + j)), rj = __ldg(reinterpret_cast<const float2*>(vec + GV_RK * GP_T + j));
#pragma unroll
      for (int e = 0; e < 2; ++e) {
        const int i = m0 + g + 8 * e;
        float2 o;
        o.x = j <= i ? acc[2 * e] * ri[e] * (rj.x * gp_ex2((gi[e] - gj.x) + (li[e] - lj.x))) : 0.f;
        o.y = j + 1 <= i ? acc[2 * e + 1] * ri[e] * (rj.y * gp_ex2((gi[e] - gj.y) + (li[e] - lj.y))) : 0.f;
        *reinterpret_cast<float2*>(Ps + i * GP_LDT + j) = o;
      }
    }
  }
  const int tg = warp >> 2, vg = warp & 3;
  float acc[2][4][4];
#pragma unroll
  for (int m = 0; m < 2; ++m)
#pragma unroll
    for (int j = 0; j < 4; ++j) acc[m][j][0] = acc[m][j][1] = acc[m][j][2] = acc[m][j][3] = 0.f;
  auto terms = [&](const float4* bs, float (*hb)[2], float (*lb)[2]) {            // of 8 rows of B for this warp's 32 columns
#pragma unroll
    for (int j = 0; j < 4; j += 2) {
      const float4 v = bs[(j >> 1) * 128];
      gp_split(v.x, hb[j][0], lb[j][0]); gp_split(v.y, hb[j][1], lb[j][1]); gp_split(v.z, hb[j + 1][0], lb[j + 1][0]); gp_split(v.w, hb[j + 1][1], lb[j + 1][1]);
    }
  };
  uint32_t zr[2][2][4];                           // gates of this thread's outputs, asked for ahead of the last products
  const bool pairs = ((reinterpret_cast<uintptr_t>(p.z) | (uintptr_t)(2 * p.ld_z)) & 3) == 0;
#pragma unroll
  for (int step = 0; step < 6; ++step) {
    if (step == 5) gp_cp_wait<0>(); else gp_cp_wait<1>();
    __syncthreads();                              // this step's operands are there for all, the ones of the step before are done with
    if (step + 2 < 6) fetch(step + 2);
    const float4* bs = Bs + (step % GO_RING) * 1024 + vg * 256 + lane;
    if (step < 4) {
#pragma unroll
      for (int kk = 0; kk < 4; kk += 2) {
        uint32_t a[2][4];                         // rows 0-7 | 8-15 of k step kk, then of kk + 1
#pragma unroll
        for (int m = 0; m < 2; ++m) gp_ldsm4(a[m], qs + (tg * 32 + m * 16 + (lane & 15)) * GP_LDK + step * 32 + (kk + (lane >> 4)) * 8);
#pragma unroll
        for (int x = 0; x < 2; ++x) {
          float af[2][4], hb[4][2], lb[4][2];
#pragma unroll
          for (int m = 0; m < 2; ++m) {
            const float2 f0 = unpack_16<BF16>(a[m][2 * x]), f1 = unpack_16<BF16>(a[m][2 * x + 1]);
            af[m][0] = f0.x; af[m][1] = f1.x; af[m][2] = f0.y; af[m][3] = f1.y;
          }
          terms(bs + (kk + x) * 32, hb, lb);
#pragma unroll
          for (int j = 0; j < 8; ++j) gp_mma_tf32(acc[j & 1][j >> 1], af[j & 1], hb[j >> 1][0], hb[j >> 1][1]);
#pragma unroll
          for (int j = 0; j < 8; ++j) gp_mma_tf32(acc[j & 1][j >> 1], af[j & 1], lb[j >> 1][0], lb[j >> 1][1]);
        }
      }
      if (step == 3) {
#pragma unroll
        for (int m = 0; m < 2; ++m)
#pragma unroll
          for (int e = 0; e < 2; ++e) {
            const int t = tg * 32 + m * 16 + g + 8 * e;
            const uint16_t* zp = p.z + (size_t)(row0 + (t < n ? t : 0)) * p.ld_z + (size_t)h * GP_D + vg * 32 + 2 * q;
#pragma unroll
            for (int j = 0; j < 4; ++j) zr[m][e][j] = pairs ? *reinterpret_cast<const uint32_t*>(zp + 8 * j) : (uint32_t)zp[8 * j] | (uint32_t)zp[8 * j + 1] << 16;
          }
#pragma unroll
        for (int m = 0; m < 2; ++m) {
          const float e0 = __ldg(vec + GV_EQ * GP_T + tg * 32 + m * 16 + g), e1 = __ldg(vec + GV_EQ * GP_T + tg * 32 + m * 16 + g + 8);
#pragma unroll
          for (int j = 0; j < 4; ++j) { acc[m][j][0] *= e0; acc[m][j][1] *= e0; acc[m][j][2] *= e1; acc[m][j][3] *= e1; }
        }
      }
    } else if (step - 4 <= tg) {                  // (scores behind the diagonal are zeros)
#pragma unroll
      for (int kk = 0; kk < 4; ++kk) {
        float hi[2][4], lo[2][4], hb[4][2], lb[4][2];
#pragma unroll
        for (int m = 0; m < 2; ++m) {
          const float* pp = Ps + (tg * 32 + m * 16 + g) * GP_LDT + (step - 4) * 32 + kk * 8 + 2 * q;
          const float2 f0 = *reinterpret_cast<const float2*>(pp), f1 = *reinterpret_cast<const float2*>(pp + 8 * GP_LDT);
          gp_split(f0.x, hi[m][0], lo[m][0]); gp_split(f1.x, hi[m][1], lo[m][1]); gp_split(f0.y, hi[m][2], lo[m][2]); gp_split(f1.y, hi[m][3], lo[m][3]);
        }
        terms(bs + kk * 32, hb, lb);
#pragma unroll
        for (int j = 0; j < 8; ++j) gp_mma_tf32(acc[j & 1][j >> 1], hi[j & 1], hb[j >> 1][0], hb[j >> 1][1]);
#pragma unroll
        for (int j = 0; j < 8; ++j) gp_mma_tf32(acc[j & 1][j >> 1], lo[j & 1], hb[j >> 1][0], hb[j >> 1][1]);
#pragma unroll
        for (int j = 0; j < 8; ++j) gp_mma_tf32(acc[j & 1][j >> 1], hi[j & 1], lb[j >> 1][0], lb[j >> 1][1]);
      }
    }
  }
  // RMS norm of the head's row and the gate, with the roundings of the separate operators (16-bit row, normalised row, weighted row)
  float o16[2][4][4];
#pragma unroll
  for (int m = 0; m < 2; ++m) {
    float ss[2] = {0.f, 0.f};
#pragma unroll
    for (int j = 0; j < 4; ++j)
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const float f = gp_ld<BF16>(gp_st<BF16>(acc[m][j][e]));
        o16[m][j][e] = f;
        ss[e >> 1] = fmaf(f, f, ss[e >> 1]);
      }
#pragma unroll
    for (int e = 0; e < 2; ++e) {
      ss[e] += __shfl_xor_sync(0xffffffffu, ss[e], 1);
      ss[e] += __shfl_xor_sync(0xffffffffu, ss[e], 2);
      if (q == 0) red[(tg * 32 + m * 16 + g + 8 * e) * 4 + vg] = ss[e];
    }
  }
  __syncthreads();
#pragma unroll
  for (int m = 0; m < 2; ++m)
#pragma unroll
    for (int e = 0; e < 2; ++e) {
      const int t = tg * 32 + m * 16 + g + 8 * e;
      if (t >= n) continue;
      const float4 r4 = *reinterpret_cast<const float4*>(red + t * 4);
      const float inv = 1.0f / sqrtf(((r4.x + r4.y) + (r4.z + r4.w)) * (1.0f / 128.0f) + p.eps);
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const int v = vg * 32 + j * 8 + 2 * q;
        const float2 nw = unpack_16<BF16>(*reinterpret_cast<const uint32_t*>(p.norm_w + v));
        const float2 y1 = unpack_16<BF16>(pack_16<BF16>(o16[m][j][2 * e] * inv, o16[m][j][2 * e + 1] * inv));
        const float2 y2 = unpack_16<BF16>(pack_16<BF16>(nw.x * y1.x, nw.y * y1.y));
        const float2 z = unpack_16<BF16>(zr[m][e][j]);
        *reinterpret_cast<uint32_t*>(p.out + ((size_t)(row0 + t) * p.Hv + h) * GP_D + v) =
            pack_16<BF16>(y2.x * gp_silu(z.x), y2.y * gp_silu(z.y));
      }
    }
}

}  // namespace fb

using namespace fb;

// x [T, C] 16-bit rows (stride ldx, a multiple of 8 elements, 16-byte aligned), w [C, 4], state [slots, C, 3]; chunks / reqs as in
// GdnPromptParams; out [T, C].  C % 8 == 0.
extern "C" int fb_gdn_conv_prompt(const void* x, long long ldx, const void* w, void* state, const int* chunks, int n_chunks, const int* reqs, int n_reqs, void* out,
                                  int C, int dtype, void* stream_) {
  if (n_chunks <= 0 || n_reqs <= 0) return 0;
  if (C % 8 != 0 || ldx % 8 != 0 || (dtype != 0 && dtype != 1) || n_chunks > 65535 || n_reqs > 65535) return -1;
  cudaStream_t s = reinterpret_cast<cudaStream_t>(stream_);
  const dim3 grid((C / 8 + 255) / 256, n_chunks, GP_T / GP_CT);
  if (dtype == 1)
    launch_k(gdn_conv_prompt_kernel<true>, grid, dim3(256), 0, s, 0, (const uint16_t*)x, ldx, (const uint16_t*)w, (const uint16_t*)state, chunks, (uint16_t*)out, C);
  else
    launch_k(gdn_conv_prompt_kernel<false>, grid, dim3(256), 0, s, 0, (const uint16_t*)x, ldx, (const uint16_t*)w, (const uint16_t*)state, chunks, (uint16_t*)out, C);
  gdn_conv_state_kernel<<<dim3((C + 255) / 256, n_reqs), 256, 0, s>>>((const uint16_t*)x, ldx, (uint16_t*)state, chunks, reqs, C);
  return (int)cudaGetLastError();
}

// One pass of the chunked rule over the heads [h0, h0 + Hn); see GdnPromptParams for the operands.  Scratch: inv n_chunks * Hn * 4096,
// vecs * 576, vnew * 8192, s0 * 16384 floats.
extern "C" int fb_gdn_prompt(const void* y, long long ld_y, const void* a, const void* b, long long ld_ab, const void* z, long long ld_z, const float* A_log,
                             const float* dt_bias, const void* norm_w, float* state, void* out, const int* chunks, int n_chunks, const int* reqs, int n_reqs,
                             float* inv, float* vecs, float* vnew, float* s0, int Hk, int Hv, int h0, int Hn, float eps, int dtype, void* stream_) {
  if (n_chunks <= 0 || n_reqs <= 0 || Hn <= 0) return 0;
  if (Hk <= 0 || Hv % Hk != 0 || ld_y % 8 != 0 || (dtype != 0 && dtype != 1) || Hn > 65535 || n_reqs > 65535) return -1;
  GdnPromptParams p = {};
  p.y = (const uint16_t*)y; p.ld_y = ld_y; p.a = (const uint16_t*)a; p.b = (const uint16_t*)b; p.ld_ab = ld_ab; p.z = (const uint16_t*)z; p.ld_z = ld_z;
  p.A_log = A_log; p.dt_bias = dt_bias; p.norm_w = (const uint16_t*)norm_w; p.state = state; p.out = (uint16_t*)out; p.chunks = chunks; p.reqs = reqs;
  p.inv = inv; p.vecs = vecs; p.vnew = reinterpret_cast<float4*>(vnew); p.s0 = reinterpret_cast<float4*>(s0); p.Hk = Hk; p.Hv = Hv; p.h0 = h0; p.Hn = Hn; p.eps = eps;
  cudaStream_t s = reinterpret_cast<cudaStream_t>(stream_);
  static DeviceOnce once;
  if (once.need()) {
    cudaError_t e = cudaSuccess;
    const void* scan[2] = {(const void*)gdn_chunk_scan_kernel<true>, (const void*)gdn_chunk_scan_kernel<false>};
    const void* outk[2] = {(const void*)gdn_chunk_out_kernel<true>, (const void*)gdn_chunk_out_kernel<false>};
    for (int i = 0; i < 2 && e == cudaSuccess; ++i) {
      e = cudaFuncSetAttribute(scan[i], cudaFuncAttributeMaxDynamicSharedMemorySize, GS_SMEM);
      if (e == cudaSuccess) e = cudaFuncSetAttribute(outk[i], cudaFuncAttributeMaxDynamicSharedMemorySize, GO_SMEM);
    }
    if (e != cudaSuccess) return (int)e;
  }
  const dim3 units(n_chunks, Hn), scan(GP_D / 32, Hn, n_reqs);
  if (dtype == 1) {
    gdn_chunk_inverse_kernel<true><<<units, 128, 0, s>>>(p);
    gdn_chunk_scan_kernel<true><<<scan, GS_THREADS, GS_SMEM, s>>>(p);
    gdn_chunk_out_kernel<true><<<units, GO_THREADS, GO_SMEM, s>>>(p);
  } else {
    gdn_chunk_inverse_kernel<false><<<units, 128, 0, s>>>(p);
    gdn_chunk_scan_kernel<false><<<scan, GS_THREADS, GS_SMEM, s>>>(p);
    gdn_chunk_out_kernel<false><<<units, GO_THREADS, GO_SMEM, s>>>(p);
  }
  return (int)cudaGetLastError();
}
