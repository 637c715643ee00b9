// int4-group-128 weights x int8 activations for up to 32 rows (sm_100a): packed weights from global memory straight into the fragments of warp-level
// integer products.
//
// Bound: latency and issue, then the weight stream.  The tcgen05 route (gemm_i8.cu) unpacks nibbles through shared memory and promotes every k block out of
// TMEM, a chain that takes 0.65 us per 128 of k whatever the number of rows, beside 6.5 us of prologue and cluster reduction.  A warp-level product reads its
// operands from registers, and the order of k inside a sum is free as long as both operands agree: a lane loads 16 packed bytes of a row (32 of k), the high
// nibbles of a word are one operand register (weights 0, 2, 4, 6 of eight), the low ones the other (1, 3, 5, 7), and the activation bytes are picked to
// match: three operations for eight weights and no shared memory.  The sums of a k block are exact int32 and promoted where they lie:
//     acc[m][n] += (sum * s[n,kb] + min[n,kb] * xs[m,kb]) * a[m,kb]          (the arithmetic of gemm_i8.cu)
// A CTA takes 16 weight rows; its eight warps share out k and meet once, in shared memory, in the order of k.  Requests for DEPTH k blocks of weights
// are in flight per lane from before the dependency wait on, and several CTAs an SM cover one another's ends.
// us, gemm_i8.cu -> here, weights from HBM: 16 rows 6144 x 4096 9.4 -> 6.1, 4096 x 4096 8.0 -> 4.6, 28672 x 4096 26.4 -> 22.7, 4096 x 14336 15.3 -> 12.4;
// 8 rows 9.1 -> 5.0, 7.6 -> 3.9, 26.1 -> 16.5, 15.1 -> 10.7; 32 rows 4096 x 4096 9.7 -> 7.0.  Also tried: 32 weight rows a CTA (28672 x 4096 at 16 rows
// 23.2); one persistent CTA an SM whose warps keep their activations in registers (19.1, but 4096 x 4096 5.4) or in shared memory, with reducer warps (23.5,
// 6.1), or with TMA rings for the weights (23.3, 7.2); sums that start at the bits of 1.5 * 2^23 in place of 0 (26.6: the registers live longer).
// SwiGLU layout (64 gate rows, then their 64 up rows): the lower half of a 16-row tile is gate rows, the upper half the up rows that belong to them.
#include "gemm_smallm.cuh"
#include "launch.h"

FB_DEFINE_ERROR_API(gemm_i4_rows)

namespace fb {

struct I4RowsParams {
  const int8_t* xq; int ldq;                                // activations [M, K]
  const float* a_scale; const float* a_sum; int ld_a;       // [K / 128, ld_a], ld_a >= M + 32
  const uint8_t* w;                                         // [N, K / 2]
  const float2* pairs;                                      // (scale, min) [K / 128, N]
  void* out; int ld_out;
  const uint16_t* bias; const uint16_t* residual; int ld_res;
  int M, N, K, flags;
};
constexpr int I4R_WARPS = 8;

__device__ __forceinline__ uint4 ld_stream_b128(const void* p) {      // read once: no L1 allocation
  uint4 v;
  asm volatile("ld.global.nc.L1::no_allocate.v4.u32 {%0,%1,%2,%3}, [%4];\n" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "l"(p));
  return v;
}
__device__ __forceinline__ void mma_s8(int (&c)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
  asm volatile("mma.sync.aligned.m16n8k32.row.col.s32.s8.s8.s32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};\n"
               : "+r"(c[0]), "+r"(c[1]), "+r"(c[2]), "+r"(c[3])
               : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}
// |v| < 2^22 (15 * 127 * 128): v + 0x4B400000 is the bit pattern of 1.5 * 2^23 + v
__device__ __forceinline__ float i4_sum_to_float(int v) { return __int_as_float(v + 0x4B400000) - 12582912.0f; }
__device__ __forceinline__ uint32_t word_of(const uint4& v, int i) { return i == 0 ? v.x : i == 1 ? v.y : i == 2 ? v.z : v.w; }

// NT: tiles of eight tokens; CTAS: meant to be resident on an SM
template <int NT, int DEPTH, int CTAS, bool BF16>
__global__ void __launch_bounds__(I4R_WARPS * 32, CTAS) i4_rows_kernel(const I4RowsParams p) {
  __shared__ float red[I4R_WARPS][NT][4][32];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, g = lane >> 2, q = lane & 3;
  const bool swiglu = (p.flags & GEMM_SWIGLU) != 0;
  const int kb_total = p.K >> 7, half = p.K >> 1;
  const int kb0 = warp * kb_total / I4R_WARPS, kb1 = (warp + 1) * kb_total / I4R_WARPS;
  pdl_launch_dependents();

  const uint8_t* wp[2];
  const float2* sp[2];
#pragma unroll
  for (int h = 0; h < 2; ++h) {
    const int o = blockIdx.x * 8 + g;                       // SwiGLU: output column
    int row = swiglu ? (o >> 6) * 128 + (o & 63) + h * 64 : blockIdx.x * 16 + h * 8 + g;
    row = min(row, p.N - 1);                                // (past the end: dropped below)
    wp[h] = p.w + (size_t)row * half + q * 16;
    sp[h] = p.pairs + row;
  }
  uint4 wr[DEPTH][2];
  float2 sc[DEPTH][2];
  auto load = [&](int d, int kb) {
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      wr[d][h] = ld_stream_b128(wp[h] + kb * 64);
      sc[d][h] = __ldg(sp[h] + (size_t)kb * p.N);
    }
  };
#pragma unroll
  for (int d = 0; d < DEPTH; ++d)
    if (kb0 + d < kb1) load(d, kb0 + d);
  pdl_wait();

  float acc[NT][4];
#pragma unroll
  for (int j = 0; j < NT; ++j)
#pragma unroll
    for (int c = 0; c < 4; ++c) acc[j][c] = 0.f;
  const int8_t* xp[NT];
#pragma unroll
  for (int j = 0; j < NT; ++j) xp[j] = p.xq + (size_t)min(j * 8 + g, p.M - 1) * p.ldq + q * 32;      // (columns past M: dropped below)

  for (int kb = kb0; kb < kb1; kb += DEPTH) {
#pragma unroll
    for (int d = 0; d < DEPTH; ++d) {
      const int k = kb + d;
      if (k >= kb1) break;
      uint4 x0[NT], x1[NT];
#pragma unroll
      for (int j = 0; j < NT; ++j) {
        x0[j] = *reinterpret_cast<const uint4*>(xp[j] + k * 128);
        x1[j] = *reinterpret_cast<const uint4*>(xp[j] + k * 128 + 16);
      }
      int c[NT][4];
#pragma unroll
      for (int j = 0; j < NT; ++j)
#pragma unroll
        for (int i = 0; i < 4; ++i) c[j][i] = 0;
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        uint32_t b0[NT], b1[NT];
#pragma unroll
        for (int j = 0; j < NT; ++j) {
          const uint4& x = e < 2 ? x0[j] : x1[j];
          const uint32_t lo = word_of(x, 2 * (e & 1)), hi = word_of(x, 2 * (e & 1) + 1);
          b0[j] = __byte_perm(lo, hi, 0x6420);
          b1[j] = __byte_perm(lo, hi, 0x7531);
        }
        const uint32_t u = word_of(wr[d][0], e), v = word_of(wr[d][1], e);
        const uint32_t a0 = (u >> 4) & 0x0F0F0F0Fu, a1 = (v >> 4) & 0x0F0F0F0Fu, a2 = u & 0x0F0F0F0Fu, a3 = v & 0x0F0F0F0Fu;
#pragma unroll
        for (int j = 0; j < NT; ++j) mma_s8(c[j], a0, a1, a2, a3, b0[j], b1[j]);
      }
#pragma unroll
      for (int j = 0; j < NT; ++j) {
        const float2 a = *reinterpret_cast<const float2*>(p.a_scale + (size_t)k * p.ld_a + j * 8 + q * 2);
        const float2 x = *reinterpret_cast<const float2*>(p.a_sum + (size_t)k * p.ld_a + j * 8 + q * 2);
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          const float2 s = sc[d][h];
          acc[j][2 * h] = fmaf(fmaf(i4_sum_to_float(c[j][2 * h]), s.x, s.y * x.x), a.x, acc[j][2 * h]);
          acc[j][2 * h + 1] = fmaf(fmaf(i4_sum_to_float(c[j][2 * h + 1]), s.x, s.y * x.y), a.y, acc[j][2 * h + 1]);
        }
      }
      if (k + DEPTH < kb1) load(d, k + DEPTH);
    }
  }
#pragma unroll
  for (int j = 0; j < NT; ++j)
#pragma unroll
    for (int c = 0; c < 4; ++c) red[warp][j][c][lane] = acc[j][c];
  __syncthreads();

  const int sh = swiglu ? 3 : 4, cols = 1 << sh;            // output columns of this CTA
  auto to_f = [](uint16_t b) { return unpack_16<BF16>((uint32_t)b).x; };
  for (int i = threadIdx.x; i < p.M * cols; i += I4R_WARPS * 32) {
    const int m = i >> sh, r = i & (cols - 1), j = m >> 3, odd = m & 1;
    const int n = blockIdx.x * cols + r;
    if (n >= (swiglu ? p.N >> 1 : p.N)) continue;
    const int h = swiglu ? 0 : r >> 3, l = (r & 7) * 4 + ((m & 7) >> 1);
    float v = 0.f, u = 0.f;
#pragma unroll
    for (int w = 0; w < I4R_WARPS; ++w) {
      v += red[w][j][2 * h + odd][l];
      if (swiglu) u += red[w][j][2 + odd][l];
    }
    if (swiglu) {
      if (p.flags & GEMM_BIAS) {
        const int row = (n >> 6) * 128 + (n & 63);
        v += to_f(p.bias[row]); u += to_f(p.bias[row + 64]);
      }
      v = silu_f(v) * u;
    } else if (p.flags & GEMM_BIAS) {
      v += to_f(p.bias[n]);
    }
    if (p.flags & GEMM_RESIDUAL) v += to_f(p.residual[(size_t)m * p.ld_res + n]);
    if (p.flags & GEMM_OUT_F32) reinterpret_cast<float*>(p.out)[(size_t)m * p.ld_out + n] = v;
    else reinterpret_cast<uint16_t*>(p.out)[(size_t)m * p.ld_out + n] = (uint16_t)pack_16<BF16>(v, 0.f);
  }
}

template <int NT, int DEPTH, int CTAS>
static int launch_i4_rows(const I4RowsParams& p, int dtype, cudaStream_t stream) {
  return (int)launch_k<PDL_GEMM>(dtype == 1 ? i4_rows_kernel<NT, DEPTH, CTAS, true> : i4_rows_kernel<NT, DEPTH, CTAS, false>, dim3((p.N + 15) / 16),
                                 dim3(I4R_WARPS * 32), 0, stream, 0, p);
}

}  // namespace fb

// Operands as for fb_gemm_i8 with int4 groups of 128 (plain, not grouped); M <= 32, N % 8 == 0 (SwiGLU: 128), K % 128 == 0.  -1: not a product for this kernel.
extern "C" int fb_gemm_i4_rows(const void* xq, int ldq, const float* a_scale, const float* a_sum, int ld_a, const void* Wq, const float* pairs, void* out,
                               const void* bias, const void* residual, int M, int N, int K, int ld_out, int ld_res, int dtype, int flags, void* stream_) {
  using namespace fb;
  if (M <= 0) return 0;
  if (M > 32 || K <= 0 || K % 128 != 0 || N <= 0 || N % 8 != 0 || ldq % 16 != 0 || ld_a % 2 != 0 || ld_a < M + 32 || (dtype != 0 && dtype != 1)) return -1;
  if ((flags & ~(GEMM_BIAS | GEMM_RESIDUAL | GEMM_SWIGLU | GEMM_OUT_F32)) || ((flags & GEMM_SWIGLU) && N % 128 != 0)) return -1;
  if ((reinterpret_cast<uintptr_t>(xq) & 15) || (reinterpret_cast<uintptr_t>(Wq) & 15) || (reinterpret_cast<uintptr_t>(a_scale) & 7) ||
      (reinterpret_cast<uintptr_t>(a_sum) & 7) || (reinterpret_cast<uintptr_t>(pairs) & 7)) return -1;
  I4RowsParams p;
  p.xq = (const int8_t*)xq; p.ldq = ldq; p.a_scale = a_scale; p.a_sum = a_sum; p.ld_a = ld_a; p.w = (const uint8_t*)Wq;
  p.pairs = reinterpret_cast<const float2*>(pairs); p.out = out; p.ld_out = ld_out; p.bias = (const uint16_t*)bias;
  p.residual = (const uint16_t*)residual; p.ld_res = ld_res; p.M = M; p.N = N; p.K = K; p.flags = flags;
  cudaStream_t s = reinterpret_cast<cudaStream_t>(stream_);
  int sms = 0, dev = 0;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  // Where all CTAs of a matrix are resident two to an SM, each keeps the most requests in flight; larger matrices live on more CTAs an SM.  us at 16 / 8 rows,
  // two / three / four CTAs: 4096 x 14336 12.4 16.0 - / 10.7 14.4 13.9, 6144 x 4096 7.8 6.1 - / 6.5 5.0 5.4, 28672 x 4096 25.5 22.7 - / 18.9 20.3 16.5.
  // 17 to 32 rows: 4096 x 14336 18.1 against 19.6 in gemm_i8.cu, 28672 x 4096 38 against 36.
  const int ctas = (N + 15) / 16;
  const bool resident = ctas <= 2 * sms;
  if (M > 16) return resident ? launch_i4_rows<4, 2, 2>(p, dtype, s) : -1;
  if (M > 8) return resident ? launch_i4_rows<2, 4, 2>(p, dtype, s) : launch_i4_rows<2, 2, 3>(p, dtype, s);
  return resident ? launch_i4_rows<1, 4, 2>(p, dtype, s) : ctas <= 3 * sms ? launch_i4_rows<1, 4, 3>(p, dtype, s) : launch_i4_rows<1, 2, 4>(p, dtype, s);
}
