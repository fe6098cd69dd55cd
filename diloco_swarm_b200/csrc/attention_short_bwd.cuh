// Causal attention backward of short sequences on mma.sync: Q, K, V and dO of a head in shared memory, a warp per 16 key rows (dK and
// dV) or 16 query rows (dQ); no sums cross a warp.
//
// The tcgen05 kernel for sequences of one tile (attention_bwd_kernel<true>) does one item at a time on an SM, in some 5 us however
// short the sequence is: a chain of loads, two products, the row algebra, three products and three stores with a barrier between
// any two.  For a little more than a tile it does three pairs of whole tiles, with dQ summed up in memory and two kernels around
// it.  Here scores and their gradients are computed twice, once by rows and once by columns, so that every product's operand is in
// the registers of the warp that needs it; only blocks of 16 under the diagonal are computed, and several blocks share an SM.
// us a launch: 64 x 16 tokens, 12 heads of 64, 32.8 -> 6.0; 1 x 128, 4 heads of 32, 8.0 -> 4.8; 200 x 133 of those 68.7 -> 30.3.  Work that
// grows with the square of the length on the slower instruction ends it: beside the rule in attention.cu.
//
// Products are added up 16 at a time in the order of attention_bwd_kernel, dQ by tiles of 128 keys, with its row algebra and its
// order of additions in D = rowsum(dO O), so the results are the same bits.
#pragma once
#include "attention_short.cuh"

namespace dsw {

struct ShortBwdArgs {
  const __nv_bfloat16 *qkv, *out, *dout;
  const float* lse;
  __nv_bfloat16* dqkv;
  float* colsum;                 // optional: += column sums of dqkv
  int T, nh;
  float scale;
};

constexpr int SHORT_BWD_MAX_T = 192;          // heads of 32 (of 64: 64)
// Blocks for a head (each loads it), warps of a block (0: the other kernel), and whether a warp loads its own rows' operands again
// for every block of 16 it meets: with them in registers two blocks of eight warps do not fit on an SM.
struct ShortBwdPlan { int parts, warps; bool reload; };

// HS: head size; LONG: more than 128 keys.
template <int HS, bool LONG, bool RELOAD>
__global__ void __launch_bounds__(RELOAD ? 512 : 256, 1)
attention_short_bwd_kernel(ShortBwdArgs a) {
  constexpr int CH = HS / 8, LPR = CH;
  extern __shared__ __align__(128) uint8_t short_smem[];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, d = a.nh * HS, T = a.T;
  const int blocks = (T + 15) >> 4, bh = blockIdx.x, b = bh / a.nh, h = bh - b * a.nh;
  const int PART = blocks * 16 * HS * 2;
  float* const s_lse = reinterpret_cast<float*>(short_smem + 4 * PART);          // log-sum-exp in base 2, +inf past the sequence
  float* const s_d = s_lse + blocks * 16;                                        // -D * scale
  float* const s_sum = s_d + blocks * 16 + warp * 3 * HS;                        // column sums of the warp's dQ, dK, dV
  for (int i = lane; i < 3 * HS; i += 32) s_sum[i] = 0.f;
  const float scale_log2 = a.scale * 1.4426950408889634f;
  pdl_wait();
  pdl_launch();
  const __nv_bfloat16* src = a.qkv + (long long)b * T * 3 * d + h * HS;
  const long long row0 = (long long)b * T * d + h * HS;              // of out and dout
  for (int i = threadIdx.x; i < blocks * 16 * CH; i += blockDim.x) {
    const int row = i / CH, ch = i - row * CH;
    const bool in = row < T;                                         // rows past the sequence are zeros
    const __nv_bfloat16* p = src + (in ? (long long)row * 3 * d + ch * 8 : 0);
#pragma unroll
    for (int part = 0; part < 3; ++part) cp_async16(short_smem + part * PART + short_offset<HS>(row, ch), p + part * d, in);
    cp_async16(short_smem + 3 * PART + short_offset<HS>(row, ch), a.dout + row0 + (in ? (long long)row * d + ch * 8 : 0), in);
  }
  // D by CH lanes to a row, dO and O from memory, while the tiles are on their way
  for (int i = threadIdx.x; i < blocks * 16 * CH; i += blockDim.x) {
    const int row = i / CH, ch = i - row * CH;
    const bool in = row < T;
    const long long at = row0 + (in ? (long long)row * d + ch * 8 : 0);
    const uint4 z = make_uint4(0, 0, 0, 0);
    const uint4 o = in ? *reinterpret_cast<const uint4*>(a.out + at) : z, g = in ? *reinterpret_cast<const uint4*>(a.dout + at) : z;
    float v = dot8(o, g);
#pragma unroll
    for (int x = LPR / 2; x > 0; x >>= 1) v += __shfl_xor_sync(0xffffffffu, v, x);
    if (ch == 0) {
      s_d[row] = -v * a.scale;
      s_lse[row] = in ? a.lse[(long long)bh * T + row] * 1.4426950408889634f : INFINITY;
    }
  }
  asm volatile("cp.async.wait_all;" ::: "memory");
  __syncthreads();
  const uint32_t sq = smem_u32(short_smem), sk = sq + PART, sv = sk + PART, so = sv + PART;
  const int g = lane >> 2, t = (lane & 3) * 2;
  const auto rows_a = [&](uint32_t (&f)[4], uint32_t base, int blk, int k) {          // A operand: 16 rows, 16 columns of the head
    ldmatrix4(f, base + short_offset<HS>(blk * 16 + (lane & 15), k * 2 + (lane >> 4)));
  };
  const auto rows_b = [&](uint32_t (&f)[4], uint32_t base, int blk, int k) {          // B operand: n = the 16 rows, K = 16 columns
    ldmatrix4(f, base + short_offset<HS>(blk * 16 + (lane & 7) + ((lane >> 4) << 3), k * 2 + ((lane >> 3) & 1)));
  };
  const auto cols_b = [&](uint32_t (&f)[4], uint32_t base, int blk, int n) {          // B operand: n = 16 columns, K = the 16 rows
    ldmatrix4_trans(f, base + short_offset<HS>(blk * 16 + (lane & 15), n + (lane >> 4)));
  };
  // what a warp has summed up over its 16 rows goes out, part 0: dQ, 1: dK, 2: dV
  const auto store = [&](const float (&c)[CH][4], int blk, int part) {
#pragma unroll
    for (int r = 0; r < 2; ++r) {
      const int row = blk * 16 + g + r * 8;
      if (row >= T) continue;
      uint32_t* dst = reinterpret_cast<uint32_t*>(a.dqkv + ((long long)b * T + row) * 3 * d + part * d + h * HS + t);
#pragma unroll
      for (int n = 0; n < CH; ++n) dst[n * 4] = pack_bf16(c[n][2 * r], c[n][2 * r + 1]);
    }
    if (a.colsum == nullptr) return;
    // over the eight rows that share a column, a warp's sums added up without atomics (with them and a shuffle per step and column
    // 12 x 90 tokens, 12 heads of 64, took 14 us instead of 8): each step with half as many columns; rows past the sequence are zeros
    float v[2 * CH];
#pragma unroll
    for (int n = 0; n < CH; ++n) { v[2 * n] = c[n][0] + c[n][2]; v[2 * n + 1] = c[n][1] + c[n][3]; }
    int first_col = 0;
#pragma unroll
    for (int m = CH, x = 16; x >= 4; m >>= 1, x >>= 1) {
      const bool up = lane & x;
#pragma unroll
      for (int i = 0; i < m; ++i) {
        const float keep = up ? v[i + m] : v[i], send = up ? v[i] : v[i + m];
        v[i] = keep + __shfl_xor_sync(0xffffffffu, send, x);
      }
      first_col += up ? m : 0;
    }
#pragma unroll
    for (int i = 0; i < CH / 4; ++i) s_sum[part * HS + ((first_col + i) >> 1) * 8 + t + ((first_col + i) & 1)] += v[i];
  };
  // the warps of a head's blocks take its 2 * blocks tasks, keys first: with as many warps as blocks of 16 each has dK and dV of one
  // and then dQ of the same one, and all have about the same to do
  const int step = gridDim.y * (blockDim.x >> 5);
  for (int task = blockIdx.y + gridDim.y * warp; task < 2 * blocks; task += step) {
    const bool keys = task < blocks;
    const int blk = keys ? task : task - blocks;
    if (keys) {
      // ---------------------------------------------------------------- dK and dV of 16 key rows
      uint32_t ka[HS / 16][4], va[HS / 16][4];
#pragma unroll
      for (int k = 0; k < (RELOAD ? 0 : HS / 16); ++k) { rows_a(ka[k], sk, blk, k); rows_a(va[k], sv, blk, k); }
      float dk[CH][4], dv[CH][4];
#pragma unroll
      for (int n = 0; n < CH; ++n)
#pragma unroll
        for (int e = 0; e < 4; ++e) { dk[n][e] = 0.f; dv[n][e] = 0.f; }
      for (int i = blk; i < blocks; ++i) {
        float s[2][4] = {{0.f, 0.f, 0.f, 0.f}, {0.f, 0.f, 0.f, 0.f}}, dp[2][4] = {{0.f, 0.f, 0.f, 0.f}, {0.f, 0.f, 0.f, 0.f}};
#pragma unroll
        for (int k = 0; k < HS / 16; ++k) {
          uint32_t f[4];
          if (RELOAD) { rows_a(ka[k], sk, blk, k); rows_a(va[k], sv, blk, k); }
          rows_b(f, sq, i, k);
          mma_bf16(s[0], ka[k], f[0], f[1]);
          mma_bf16(s[1], ka[k], f[2], f[3]);
          rows_b(f, so, i, k);
          mma_bf16(dp[0], va[k], f[0], f[1]);
          mma_bf16(dp[1], va[k], f[2], f[3]);
        }
        uint32_t pa[4], da[4];
#pragma unroll
        for (int u = 0; u < 2; ++u) {
          const int q0 = i * 16 + u * 8 + t;
          const float2 l2 = *reinterpret_cast<const float2*>(s_lse + q0), nd = *reinterpret_cast<const float2*>(s_d + q0);
          float p[4], ds[4];
#pragma unroll
          for (int e = 0; e < 4; ++e) {
            const int q = q0 + (e & 1), key = blk * 16 + g + (e >> 1) * 8;
            p[e] = ex2_approx(fmaf(s[u][e], scale_log2, -((e & 1) ? l2.y : l2.x)));
            if (key > q) p[e] = 0.f;
            ds[e] = p[e] * fmaf(dp[u][e], a.scale, (e & 1) ? nd.y : nd.x);
          }
          pa[2 * u] = pack_bf16(p[0], p[1]);
          pa[2 * u + 1] = pack_bf16(p[2], p[3]);
          da[2 * u] = pack_bf16(ds[0], ds[1]);
          da[2 * u + 1] = pack_bf16(ds[2], ds[3]);
        }
#pragma unroll
        for (int n = 0; n < CH; n += 2) {
          uint32_t f[4];
          cols_b(f, so, i, n);
          mma_bf16(dv[n], pa, f[0], f[1]);
          mma_bf16(dv[n + 1], pa, f[2], f[3]);
          cols_b(f, sq, i, n);
          mma_bf16(dk[n], da, f[0], f[1]);
          mma_bf16(dk[n + 1], da, f[2], f[3]);
        }
      }
      store(dk, blk, 1);
      store(dv, blk, 2);
    } else {
      // ---------------------------------------------------------------- dQ of 16 query rows
      uint32_t qa[HS / 16][4], oa[HS / 16][4];
#pragma unroll
      for (int k = 0; k < (RELOAD ? 0 : HS / 16); ++k) { rows_a(qa[k], sq, blk, k); rows_a(oa[k], so, blk, k); }
      float dq[CH][4], first[LONG ? CH : 1][4];
#pragma unroll
      for (int n = 0; n < CH; ++n)
#pragma unroll
        for (int e = 0; e < 4; ++e) dq[n][e] = 0.f;
      const float l2[2] = {s_lse[blk * 16 + g], s_lse[blk * 16 + g + 8]}, nd[2] = {s_d[blk * 16 + g], s_d[blk * 16 + g + 8]};
      for (int i = 0; i <= blk; ++i) {
        if (LONG && i == 8)
#pragma unroll
          for (int n = 0; n < CH; ++n)
#pragma unroll
            for (int e = 0; e < 4; ++e) { first[LONG ? n : 0][e] = dq[n][e]; dq[n][e] = 0.f; }
        float s[2][4] = {{0.f, 0.f, 0.f, 0.f}, {0.f, 0.f, 0.f, 0.f}}, dp[2][4] = {{0.f, 0.f, 0.f, 0.f}, {0.f, 0.f, 0.f, 0.f}};
#pragma unroll
        for (int k = 0; k < HS / 16; ++k) {
          uint32_t f[4];
          if (RELOAD) { rows_a(qa[k], sq, blk, k); rows_a(oa[k], so, blk, k); }
          rows_b(f, sk, i, k);
          mma_bf16(s[0], qa[k], f[0], f[1]);
          mma_bf16(s[1], qa[k], f[2], f[3]);
          rows_b(f, sv, i, k);
          mma_bf16(dp[0], oa[k], f[0], f[1]);
          mma_bf16(dp[1], oa[k], f[2], f[3]);
        }
        uint32_t da[4];
#pragma unroll
        for (int u = 0; u < 2; ++u) {
          float ds[4];
#pragma unroll
          for (int e = 0; e < 4; ++e) {
            const int key = i * 16 + u * 8 + t + (e & 1), q = blk * 16 + g + (e >> 1) * 8;
            float p = ex2_approx(fmaf(s[u][e], scale_log2, -l2[e >> 1]));
            if (key > q) p = 0.f;
            ds[e] = p * fmaf(dp[u][e], a.scale, nd[e >> 1]);
          }
          da[2 * u] = pack_bf16(ds[0], ds[1]);
          da[2 * u + 1] = pack_bf16(ds[2], ds[3]);
        }
#pragma unroll
        for (int n = 0; n < CH; n += 2) {
          uint32_t f[4];
          cols_b(f, sk, i, n);
          mma_bf16(dq[n], da, f[0], f[1]);
          mma_bf16(dq[n + 1], da, f[2], f[3]);
        }
      }
      if (LONG && blk >= 8)
#pragma unroll
        for (int n = 0; n < CH; ++n)
#pragma unroll
          for (int e = 0; e < 4; ++e) dq[n][e] += first[LONG ? n : 0][e];
      store(dq, blk, 0);
    }
  }
  if (a.colsum == nullptr) return;
  __syncthreads();
  for (int i = threadIdx.x; i < 3 * HS; i += blockDim.x) {
    float v = 0.f;
    for (int w = 0; w < (int)(blockDim.x >> 5); ++w) v += s_sum[(w - warp) * 3 * HS + i];
    atomicAdd(a.colsum + i / HS * d + h * HS + i % HS, v);
  }
}

template <int HS, bool LONG, bool RELOAD>
inline int launch_attention_short_bwd(const ShortBwdArgs& a, int n_bh, int parts, int warps, cudaStream_t st) {
  constexpr int ROW = 4 * HS * 2 + 2 * 4, MAX_T = LONG ? SHORT_BWD_MAX_T : HS == 32 ? 128 : 64, SUMS = 3 * HS * 4;
  static bool attr_set[64] = {false};
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return -2;
  const auto kernel = attention_short_bwd_kernel<HS, LONG, RELOAD>;
  if (!attr_set[dev]) {
    if (cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, MAX_T * ROW + SUMS * 16) != cudaSuccess) return -2;
    attr_set[dev] = true;
  }
  return launch(kernel, dim3(n_bh, parts), warps * 32, (a.T + 15) / 16 * 16 * ROW + SUMS * warps, st, 1, a) == cudaSuccess ? 0 : -3;
}
template <int HS>
inline int attention_short_bwd(const ShortBwdArgs& a, const ShortBwdPlan& p, int n_bh, cudaStream_t st) {
  if constexpr (HS == 32)
    if (a.T > 128) return launch_attention_short_bwd<HS, true, true>(a, n_bh, p.parts, p.warps, st);
  return p.reload ? launch_attention_short_bwd<HS, false, true>(a, n_bh, p.parts, p.warps, st)
                  : launch_attention_short_bwd<HS, false, false>(a, n_bh, p.parts, p.warps, st);
}
inline int load_attention_short_bwd() {
  cudaFuncAttributes a;
  const auto bad = [&](auto kernel) { return cudaFuncGetAttributes(&a, kernel) != cudaSuccess; };
  return bad(attention_short_bwd_kernel<64, false, false>) | bad(attention_short_bwd_kernel<64, false, true>) |
         bad(attention_short_bwd_kernel<32, false, false>) | bad(attention_short_bwd_kernel<32, false, true>) |
         bad(attention_short_bwd_kernel<32, true, true>);
}

}  // namespace dsw
