// GEMM for few rows and a short K on mma.sync: 32 x 32 tiles, both operands of a tile in shared memory at once, optionally with
// the LayerNorm that makes the activations.
//
// What bounds these is the latency of one launch after the other.  The cluster kernel (gemm_split.cuh) spends some 3 us on
// setting up tensor memory and barriers, a TMA round trip, the products' and the exchange's; here the operands come by plain
// asynchronous copies, the weights' before the kernel ahead has ended, and the sums are in registers.  A tile of 32 rows takes
// a whole row of a narrow model, so its LayerNorm costs no launch and no exchange: every column tile makes it again.  In the
// chain of a sampling pass of the tiny model (5 x 24 tokens, width 128) LayerNorm and the product behind it took 1.75 + 3.0 us,
// here 2.5; the pass 90.1 -> 69.0.  Few rows of a wider model whose blocks are all resident gain less
// (GPT-2 small: 120 x 2304 5.4 -> 4.65, 120 x 768 from 768 4.5 -> 3.7 in the chain, where the launch behind loses most of it again:
// the pass 352.8 -> 350.3); where the line to the cluster kernel lies stands beside narrow_fits.
//
// The results are the cluster kernel's, bit for bit: the same slices of K, 16 values at a time, and their sums added up in the
// same order, the owner's first (narrow_sum).
#pragma once
#include "gemm_split.cuh"
#include "attention_short.cuh"

namespace dsw {

constexpr int NARROW_ROWS = 32, NARROW_COLS = 32, NARROW_THREADS = 256;
constexpr int NARROW_MAX_K = 1024;

struct NarrowArgs {
  const __nv_bfloat16 *a, *w;          // activations [M, K] (LN: what is normalised), weights [N, K] or [K, N]
  long long lda, ldw;
  int ref_width;                       // tile width of the cluster kernel, which says who owns a column's sum
  const __nv_bfloat16* a_lo;           // LN: low half of the rows, or null
  const float *gamma, *beta;
  float eps;
  __nv_bfloat16* ln_out;               // LN: where the normalised rows and their statistics are kept, or null
  float *mean_out, *rstd_out;
};

// Byte offset of 16-byte chunk `chunk` of row `row` of K values.
__device__ __forceinline__ uint32_t narrow_offset(int K, int row, int chunk) { return row * K * 2 + ((chunk ^ (row & 7)) << 4); }

// MN: weights [K, N].  LN: K <= 128.  g.split_k slices of K.
template <int MODE, bool MN, bool LN>
__global__ void __launch_bounds__(NARROW_THREADS)
gemm_narrow_kernel(GemmArgs g, NarrowArgs n) {
  extern __shared__ __align__(128) uint8_t narrow_smem[];
  const int K = g.K, S = g.split_k, lgS = 31 - __clz(S);
  uint8_t* sa = narrow_smem;                                         // [32 rows][K]
  uint8_t* sw = sa + NARROW_ROWS * K * 2;                            // [32][K], MN: [K][32]
  float* part = reinterpret_cast<float*>(sw + NARROW_COLS * K * 2);  // [S][32][32]
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int m0 = blockIdx.x * NARROW_ROWS, n0 = blockIdx.y * NARROW_COLS;
  static_assert(NARROW_THREADS == 8 * NARROW_ROWS && NARROW_ROWS == NARROW_COLS, "eight threads to a row of either operand");
  const int lr = threadIdx.x >> 3, lc = threadIdx.x & 7;
  const auto load_w = [&] {
    if constexpr (!MN) {
      const bool in = n0 + lr < g.N;
      const __nv_bfloat16* p = n.w + (in ? (long long)(n0 + lr) * n.ldw : 0);
#pragma unroll 2
      for (int ch = lc; ch < K >> 3; ch += 8) cp_async16(sw + narrow_offset(K, lr, ch), p + (in ? ch * 8 : 0), in);
    } else {
      for (int i = threadIdx.x; i < K * 4; i += NARROW_THREADS) {
        const int k = i >> 2, ch = i & 3, col = n0 + ch * 8;
        cp_async16(sw + k * 64 + ((ch ^ ((k >> 1) & 3)) << 4), n.w + (col < g.N ? (long long)k * n.ldw + col : 0), col < g.N);
      }
    }
  };
  // The unit of eight columns that this thread finishes, and what its sum needs besides
  const int ur = threadIdx.x >> 2, uc = threadIdx.x & 3, row = m0 + ur, col = n0 + uc * 8;
  const bool mine = threadIdx.x < NARROW_ROWS * 4 && row < g.M && col < g.N;
  float bias[8];
#pragma unroll
  for (int e = 0; e < 8; ++e) bias[e] = 0.f;
  if (g.b_static) load_w();
  if (mine && g.bias != nullptr) {
    const float4 lo = __ldg(reinterpret_cast<const float4*>(g.bias + col)), hi = __ldg(reinterpret_cast<const float4*>(g.bias + col) + 1);
    bias[0] = lo.x; bias[1] = lo.y; bias[2] = lo.z; bias[3] = lo.w;
    bias[4] = hi.x; bias[5] = hi.y; bias[6] = hi.z; bias[7] = hi.w;
  }
  [[maybe_unused]] float gm[8], bt[8];
  constexpr int LPR = 16;              // lanes per row, as in layernorm_fwd_kernel
  const int lcol = (threadIdx.x & (LPR - 1)) * 8;
  if constexpr (LN) {
#pragma unroll
    for (int j = 0; j < 8; ++j) { gm[j] = 0.f; bt[j] = 0.f; }
    if (lcol < K) {
#pragma unroll
      for (int j = 0; j < 8; j += 4) {
        const float4 a = *reinterpret_cast<const float4*>(n.gamma + lcol + j);
        gm[j] = a.x; gm[j + 1] = a.y; gm[j + 2] = a.z; gm[j + 3] = a.w;
        if (n.beta) {
          const float4 b = *reinterpret_cast<const float4*>(n.beta + lcol + j);
          bt[j] = b.x; bt[j + 1] = b.y; bt[j + 2] = b.z; bt[j + 3] = b.w;
        }
      }
    }
  }
  pdl_wait();
  pdl_launch();
  if (!g.b_static) load_w();
  if constexpr (!LN) {
    const bool in = m0 + lr < g.M;
    const __nv_bfloat16* p = n.a + (in ? (long long)(m0 + lr) * n.lda : 0);
#pragma unroll 2
    for (int ch = lc; ch < K >> 3; ch += 8) cp_async16(sa + narrow_offset(K, lr, ch), p + (in ? ch * 8 : 0), in);
  }
  constexpr bool EXTRA = MODE == EPI_RESID || MODE == EPI_MUL;
  uint4 x = make_uint4(0, 0, 0, 0), t = x;
  if constexpr (EXTRA) {
    if (mine) {
      x = *reinterpret_cast<const uint4*>(MODE == EPI_RESID ? g.resid + (long long)row * g.ldr + col : g.aux_in + (long long)row * g.ldaux + col);
      if (MODE == EPI_RESID && g.aux_in != nullptr) t = *reinterpret_cast<const uint4*>(g.aux_in + (long long)row * g.ldaux + col);
    }
  }
  if constexpr (LN) {
    // the arithmetic of layernorm_fwd_kernel, 16 lanes to a row
    constexpr int P = NARROW_ROWS * LPR / NARROW_THREADS;
    uint4 hi[P], lo[P];
#pragma unroll
    for (int i = 0; i < P; ++i) {
      const int r = m0 + i * (NARROW_THREADS / LPR) + threadIdx.x / LPR;
      const bool in = r < g.M && lcol < K;
      hi[i] = in ? *reinterpret_cast<const uint4*>(n.a + (long long)r * n.lda + lcol) : make_uint4(0, 0, 0, 0);
      lo[i] = in && n.a_lo ? *reinterpret_cast<const uint4*>(n.a_lo + (long long)r * n.lda + lcol) : make_uint4(0, 0, 0, 0);
    }
    const float inv_d = 1.f / K;
#pragma unroll
    for (int i = 0; i < P; ++i) {
      const int rl = i * (NARROW_THREADS / LPR) + threadIdx.x / LPR, r = m0 + rl;
      const uint32_t hw[4] = {hi[i].x, hi[i].y, hi[i].z, hi[i].w}, lw[4] = {lo[i].x, lo[i].y, lo[i].z, lo[i].w};
      float v[8];
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const float2 a = unpack_bf16(hw[j]);
        v[2 * j] = a.x; v[2 * j + 1] = a.y;
        if (n.a_lo) {
          const float2 b = unpack_bf16(lw[j]);
          v[2 * j] += b.x; v[2 * j + 1] += b.y;
        }
      }
      float s = 0.f;
#pragma unroll
      for (int j = 0; j < 8; ++j) s += v[j];
#pragma unroll
      for (int o = LPR / 2; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
      const float mean = s * inv_d;
      float q = 0.f;
      if (lcol < K) {
#pragma unroll
        for (int j = 0; j < 8; ++j) { const float e = v[j] - mean; q += e * e; }
      }
#pragma unroll
      for (int o = LPR / 2; o > 0; o >>= 1) q += __shfl_xor_sync(0xffffffffu, q, o);
      const float rstd = rsqrtf(q * inv_d + n.eps);
      if (lcol < K) {
        float o[8];
#pragma unroll
        for (int j = 0; j < 8; ++j) o[j] = fmaf((v[j] - mean) * rstd, gm[j], bt[j]);
        const uint4 y = make_uint4(pack_bf16(o[0], o[1]), pack_bf16(o[2], o[3]), pack_bf16(o[4], o[5]), pack_bf16(o[6], o[7]));
        *reinterpret_cast<uint4*>(sa + narrow_offset(K, rl, lcol >> 3)) = y;
        if (n.ln_out != nullptr && blockIdx.y == 0 && r < g.M) *reinterpret_cast<uint4*>(n.ln_out + (long long)r * K + lcol) = y;
      }
      if (n.ln_out != nullptr && blockIdx.y == 0 && lcol == 0 && r < g.M) { n.mean_out[r] = mean; n.rstd_out[r] = rstd; }
    }
  }
  asm volatile("cp.async.wait_all;" ::: "memory");
  __syncthreads();
  // warp = 16 rows, 16 columns, every second slice of K
  const int wr = warp & 1, wc = (warp >> 1) & 1;
  const uint32_t pa = smem_u32(sa), pw = smem_u32(sw);
  const int kb = (K + BK - 1) / BK;
  for (int ks = warp >> 2; ks < S; ks += NARROW_THREADS / 128) {
    const int k0 = (((kb * ks) >> lgS)) * (BK / 16), k1 = ((kb * (ks + 1)) >> lgS) * (BK / 16);
    float c[2][4] = {{0.f, 0.f, 0.f, 0.f}, {0.f, 0.f, 0.f, 0.f}};
#pragma unroll 4
    for (int k = k0; k < k1; ++k) {
      uint32_t af[4], bf[4];
      ldmatrix4(af, pa + narrow_offset(K, wr * 16 + (lane & 15), k * 2 + (lane >> 4)));
      if constexpr (!MN) {
        ldmatrix4(bf, pw + narrow_offset(K, wc * 16 + (lane & 7) + ((lane >> 4) << 3), k * 2 + ((lane >> 3) & 1)));
      } else {
        const int kr = k * 16 + (lane & 15), ch = wc * 2 + (lane >> 4);
        ldmatrix4_trans(bf, pw + kr * 64 + ((ch ^ ((kr >> 1) & 3)) << 4));
      }
      mma_bf16(c[0], af, bf[0], bf[1]);
      mma_bf16(c[1], af, bf[2], bf[3]);
    }
    float* to = part + ks * NARROW_ROWS * NARROW_COLS + (wr * 16 + (lane >> 2)) * NARROW_COLS + wc * 16 + (lane & 3) * 2;
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      *reinterpret_cast<float2*>(to + h * 8) = make_float2(c[h][0], c[h][1]);
      *reinterpret_cast<float2*>(to + h * 8 + 8 * NARROW_COLS) = make_float2(c[h][2], c[h][3]);
    }
  }
  __syncthreads();
  if (!mine) return;
  float f[8];
  const auto slice = [&](int ks, float (&v)[8]) {
    const float4* p = reinterpret_cast<const float4*>(part + (ks * NARROW_ROWS + ur) * NARROW_COLS + uc * 8);
    const float4 lo = p[0], hi = p[1];
    v[0] = lo.x; v[1] = lo.y; v[2] = lo.z; v[3] = lo.w; v[4] = hi.x; v[5] = hi.y; v[6] = hi.z; v[7] = hi.w;
  };
  const int owner = (((col & (n.ref_width - 1)) >> 3) << lgS) >> (28 - __clz(n.ref_width));
  slice(owner, f);
  for (int ks = 0; ks < S; ++ks) {
    if (ks == owner) continue;
    float v[8];
    slice(ks, v);
#pragma unroll
    for (int e = 0; e < 8; ++e) f[e] += v[e];
  }
#pragma unroll
  for (int e = 0; e < 8; ++e) f[e] += bias[e];
  finish_unit<MODE>(g, row, col, f, x, t);
}

inline int narrow_smem_bytes(int K, int splits) { return (NARROW_ROWS + NARROW_COLS) * K * 2 + splits * NARROW_ROWS * NARROW_COLS * 4; }
int launch_narrow(const GemmArgs& g, const NarrowArgs& n, bool layernorm, cudaStream_t st);

}  // namespace dsw
