// Causal attention forward of short sequences: a block per (sequence, head), a warp per 16 query rows, everything of a head in
// shared memory and the score rows of a warp in registers, on mma.sync.
//
// What bounds so small a problem is latency, not arithmetic.  The tcgen05 kernel passes its tile through tensor memory and
// back twice, with a barrier each way, and its softmax threads take whole rows of 128 scores, masked or not; here a warp waits
// once for its operands and has scores, probabilities and output in its own registers.  5 x 24 tokens, 12 heads of 64: 6.1 -> 2.7
// us a launch, in the chain of a sampling pass 5.1 -> 2.0; 512 x 32, 4 heads of 32, 29.0 -> 5.5; beside the rule in attention.cu
// where it ends.  Products are added up in the order of attention_fwd_kernel, 16 at a time, and row sums in its four chains, so
// the results are the same bits.
#pragma once
#include "ptx.cuh"
#include "launch.h"

namespace dsw {

constexpr int SHORT_MAX_T = 128;

__device__ __forceinline__ void ldmatrix4(uint32_t (&r)[4], uint32_t addr) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0, %1, %2, %3}, [%4];" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr));
}
__device__ __forceinline__ void ldmatrix4_trans(uint32_t (&r)[4], uint32_t addr) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0, %1, %2, %3}, [%4];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr));
}
// c (16 x 8) += a (16 x 16) b (16 x 8)
__device__ __forceinline__ void mma_bf16(float (&c)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
  asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};"
               : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
               : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}

// Byte offset of 16-byte chunk `chunk` of row `row`: eight neighbouring rows of one chunk lie in different banks.
template <int HS>
__device__ __forceinline__ uint32_t short_offset(int row, int chunk) {
  return HS == 64 ? row * 128 + ((chunk ^ (row & 7)) << 4) : row * 64 + ((chunk ^ ((row >> 1) & 3)) << 4);
}

// NB: blocks of 16 rows that a sequence may have; HS: head size.
template <int NB, int HS>
__global__ void __launch_bounds__(NB <= 4 ? 128 : 256, NB <= 4 ? 1 : 2)
attention_short_kernel(const __nv_bfloat16* qkv, __nv_bfloat16* __restrict__ out, float* __restrict__ lse_out, int T, int nh, int n_bh,
                       float scale_log2) {
  constexpr int CH = HS / 8;                           // chunks of a row
  constexpr int PART = NB * 16 * HS * 2;               // bytes of Q, K or V
  extern __shared__ __align__(128) uint8_t short_smem[];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, d = nh * HS;
  const int blocks = (T + 15) >> 4, bh = blockIdx.x, b = bh / nh, h = bh - b * nh;
  pdl_wait();
  pdl_launch();
  const __nv_bfloat16* src = qkv + (long long)b * T * 3 * d + h * HS;
  for (int i = threadIdx.x; i < blocks * 16 * CH; i += blockDim.x) {
    const int row = i / CH, ch = i - row * CH;
    const bool in = row < T;                           // rows past the sequence are zeros
    const __nv_bfloat16* p = src + (in ? (long long)row * 3 * d + ch * 8 : 0);
#pragma unroll
    for (int part = 0; part < 3; ++part) cp_async16(short_smem + part * PART + short_offset<HS>(row, ch), p + part * d, in);
  }
  asm volatile("cp.async.wait_all;" ::: "memory");
  __syncthreads();
  const uint32_t sq = smem_u32(short_smem), sk = sq + PART, sv = sk + PART;
  for (int qb = warp; qb < blocks; qb += blockDim.x >> 5) {
    float s[2 * NB][4];                                // scores of 16 rows: s[n] columns 8 n .., in the accumulator's layout
#pragma unroll
    for (int n = 0; n < 2 * NB; ++n)
#pragma unroll
      for (int e = 0; e < 4; ++e) s[n][e] = 0.f;
    uint32_t q[HS / 16][4];
#pragma unroll
    for (int k = 0; k < HS / 16; ++k) ldmatrix4(q[k], sq + short_offset<HS>(qb * 16 + (lane & 15), k * 2 + (lane >> 4)));
#pragma unroll
    for (int m = 0; m < NB; ++m) {
      if (m > qb) break;                               // blocks of keys up to the diagonal
#pragma unroll
      for (int k = 0; k < HS / 16; ++k) {
        uint32_t f[4];
        ldmatrix4(f, sk + short_offset<HS>(m * 16 + (lane & 7) + ((lane >> 4) << 3), k * 2 + ((lane >> 3) & 1)));
        mma_bf16(s[2 * m], q[k], f[0], f[1]);
        mma_bf16(s[2 * m + 1], q[k], f[2], f[3]);
      }
    }
    // rows g and g + 8 of the block; the block on the diagonal is masked, those right of it were never computed
    const int g = lane >> 2, t = (lane & 3) * 2;
    float mx[2] = {-INFINITY, -INFINITY};
#pragma unroll
    for (int n = 0; n < 2 * NB; ++n) {
      if (n > 2 * qb + 1) break;
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const int col = n * 8 + t + (e & 1), row = qb * 16 + g + (e >> 1) * 8;
        if (n >= 2 * qb && col > row) s[n][e] = -INFINITY;
        mx[e >> 1] = fmaxf(mx[e >> 1], s[n][e]);
      }
    }
    // Row sums: four chains, columns 0, 1, 2 and 3 modulo 4 in ascending order, as attention_fwd_kernel adds them.  The lanes that
    // hold the first half of eight columns (t < 4) add those of the second half, which they are handed.
    float l[2][2] = {{0.f, 0.f}, {0.f, 0.f}};
#pragma unroll
    for (int r = 0; r < 2; ++r) {
      mx[r] = fmaxf(mx[r], __shfl_xor_sync(0xffffffffu, mx[r], 1));
      mx[r] = fmaxf(mx[r], __shfl_xor_sync(0xffffffffu, mx[r], 2)) * scale_log2;
    }
    float o[CH][4];
#pragma unroll
    for (int n = 0; n < CH; ++n)
#pragma unroll
      for (int e = 0; e < 4; ++e) o[n][e] = 0.f;
#pragma unroll
    for (int m = 0; m < NB; ++m) {
      if (m > qb) break;
      uint32_t p[4];
#pragma unroll
      for (int u = 0; u < 2; ++u) {
        float e[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) e[i] = ex2_approx(fmaf(s[2 * m + u][i], scale_log2, -mx[i >> 1]));
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          const float second = __shfl_down_sync(0xffffffffu, e[i], 2);
          l[i >> 1][i & 1] = (l[i >> 1][i & 1] + e[i]) + second;
        }
        p[2 * u] = pack_bf16(e[0], e[1]);
        p[2 * u + 1] = pack_bf16(e[2], e[3]);
      }
#pragma unroll
      for (int n = 0; n < CH; n += 2) {
        uint32_t f[4];
        ldmatrix4_trans(f, sv + short_offset<HS>(m * 16 + (lane & 15), n + (lane >> 4)));
        mma_bf16(o[n], p, f[0], f[1]);
        mma_bf16(o[n + 1], p, f[2], f[3]);
      }
    }
#pragma unroll
    for (int r = 0; r < 2; ++r) {
      const int lane0 = lane & ~3;          // chains 0 and 1 are its, 2 and 3 its neighbour's
      const float even = __shfl_sync(0xffffffffu, l[r][0], lane0) + __shfl_sync(0xffffffffu, l[r][0], lane0 + 1);
      const float odd = __shfl_sync(0xffffffffu, l[r][1], lane0) + __shfl_sync(0xffffffffu, l[r][1], lane0 + 1);
      const float sum = even + odd;
      const int row = qb * 16 + g + r * 8;
      if (row >= T) continue;
      const float inv = 1.f / sum;
      uint32_t* dst = reinterpret_cast<uint32_t*>(out + ((long long)b * T + row) * d + h * HS + t);
#pragma unroll
      for (int n = 0; n < CH; ++n) dst[n * 4] = pack_bf16(o[n][2 * r] * inv, o[n][2 * r + 1] * inv);
      if ((lane & 3) == 0) lse_out[(long long)bh * T + row] = (mx[r] + log2f(sum)) * 0.6931471805599453f;
    }
  }
}

template <int NB, int HS>
inline int launch_attention_short(const __nv_bfloat16* qkv, __nv_bfloat16* out, float* lse, int T, int nh, int n_bh, float scale_log2,
                                  cudaStream_t st) {
  return launch(attention_short_kernel<NB, HS>, n_bh, NB <= 4 ? 128 : 256, 3 * NB * 16 * HS * 2, st, 1, qkv, out, lse, T, nh, n_bh,
                scale_log2) == cudaSuccess ? 0 : -3;
}
template <int HS>
inline int attention_short(const __nv_bfloat16* qkv, __nv_bfloat16* out, float* lse, int T, int nh, int n_bh, float scale_log2, cudaStream_t st) {
  if (T <= 32) return launch_attention_short<2, HS>(qkv, out, lse, T, nh, n_bh, scale_log2, st);
  if (T <= 64) return launch_attention_short<4, HS>(qkv, out, lse, T, nh, n_bh, scale_log2, st);
  return launch_attention_short<8, HS>(qkv, out, lse, T, nh, n_bh, scale_log2, st);
}

inline int load_attention_short() {
  cudaFuncAttributes a;
  const auto bad = [&](auto kernel) { return cudaFuncGetAttributes(&a, kernel) != cudaSuccess; };
  return bad(attention_short_kernel<2, 64>) | bad(attention_short_kernel<4, 64>) | bad(attention_short_kernel<8, 64>) |
         bad(attention_short_kernel<2, 32>) | bad(attention_short_kernel<4, 32>) | bad(attention_short_kernel<8, 32>);
}

}  // namespace dsw
