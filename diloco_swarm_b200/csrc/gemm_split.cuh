// GEMM for few rows: 128 x BN tiles on one CTA each, K split over the CTAs of a cluster.
//
// What bounds such a GEMM is neither arithmetic nor bandwidth but latency and how many bytes are in flight: 120 rows of
// GPT-2 small through the MLP's second projection (N 768, K 3072) are six 128-wide tiles, so six SMs walked 48 k-blocks
// one after the other (17.2 us with 4.7 MB of weights cold in L2, 7.9 here).  Here a tile is 32, 64 or 128 columns wide and its K range is
// divided over up to eight CTAs, enough of them to fill the SMs; every CTA has most of its share in flight at once.
// The partial sums meet inside the cluster: a CTA owns BN / S of the tile's columns, receives the other CTAs' fp32
// sums of those through distributed shared memory and runs the epilogue on them.  No atomics, no second launch, and a
// fixed order of additions.
//
// The weights do not depend on the kernel before (LaunchMode::static_b), so their loads go out before pdl_wait(): the
// predecessor's tail covers their DRAM latency.  At most 110 KB of shared memory up to BN = 64, so that the CTAs of two
// consecutive GEMMs share an SM while the second one fills its stages.
#pragma once
#include "gemm_kernels.cuh"

namespace dsw {

// Warps 0-7 epilogue (two per TMEM lane quarter, each takes half of the tile's columns), 8 TMA, 9 MMA.  With one warp per
// quarter, and the bias and the residual's low half asked for only when the sums were there, what followed the last
// product was the longest part of a short launch: 120 x 3072 from 768 with GELU 8.3 -> 7.0 us, 120 x 2304 7.0 -> 6.3,
// 120 x 512 from 128 4.9 -> 3.9, 120 x 768 from 3072 8.6 -> 7.9 (32 weight matrices in turn, one graph).
constexpr int SPLIT_EPI_WARPS = 8, SPLIT_TMA_WARP = 8, SPLIT_MMA_WARP = 9;
constexpr int SPLIT_THREADS = 32 * (SPLIT_EPI_WARPS + 2);

template <int BN>
struct SplitSmem {
  static constexpr int NSTAGE = BN == 32 ? 4 : BN == 64 ? 3 : 4;
  static constexpr int A_BYTES = BM * BK * 2;
  static constexpr int B_BYTES = BN * BK * 2;
  static constexpr int STAGE_BYTES = A_BYTES + B_BYTES;
  static constexpr int RECV_OFFSET = NSTAGE * STAGE_BYTES;       // fp32 [source][BN / S / 4][128 rows][4]
  static constexpr int BIAS_OFFSET = RECV_OFFSET + BM * BN * 4;  // per epilogue warp: the bias of its columns
  static constexpr int BAR_OFFSET = BIAS_OFFSET + SPLIT_EPI_WARPS * (BN / 2) * 4;
  static constexpr int TOTAL = BAR_OFFSET + 128 + 1024;          // + alignment slack
};

__device__ __forceinline__ void st_cluster_v4(uint32_t addr, uint32_t a, uint32_t b, uint32_t c, uint32_t d) {
  asm volatile("st.shared::cluster.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(addr), "r"(a), "r"(b), "r"(c), "r"(d) : "memory");
}

// Eight columns of a row, f: the finished sum with bias, x: residual or factor, t: the residual's low half.  f is left as what
// was rounded.
template <int MODE>
__device__ __forceinline__ void finish_unit(const GemmArgs& g, int row, int col, float (&f)[8], const uint4& x, const uint4& t) {
  uint32_t w[4];
  if constexpr (MODE == EPI_GELU) {
    uint32_t dw[4];
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      f2 ga, da;
      gelu_pair(f[2 * e], f[2 * e + 1], ga, da);
      w[e] = pack_bf16_f2(ga);
      dw[e] = pack_bf16_f2(da);
    }
    if (g.aux_out != nullptr)
      *reinterpret_cast<uint4*>(g.aux_out + (long long)row * g.ldaux + col) = make_uint4(dw[0], dw[1], dw[2], dw[3]);
  } else {
    if constexpr (MODE == EPI_RESID || MODE == EPI_MUL || MODE == EPI_MUL_SUM) {
      const uint32_t xu[4] = {x.x, x.y, x.z, x.w};
      uint32_t tu[4] = {0, 0, 0, 0};
      if constexpr (MODE == EPI_RESID) { tu[0] = t.x; tu[1] = t.y; tu[2] = t.z; tu[3] = t.w; }
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const float2 b = unpack_bf16(xu[e]), c = unpack_bf16(tu[e]);
        f[2 * e] = MODE == EPI_RESID ? f[2 * e] + (b.x + c.x) : f[2 * e] * b.x;
        f[2 * e + 1] = MODE == EPI_RESID ? f[2 * e + 1] + (b.y + c.y) : f[2 * e + 1] * b.y;
      }
    }
#pragma unroll
    for (int e = 0; e < 4; ++e) w[e] = pack_bf16(f[2 * e], f[2 * e + 1]);
    if (MODE == EPI_RESID && g.aux_out != nullptr) {
      uint32_t lo[4];
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const float2 h = unpack_bf16(w[e]);
        lo[e] = pack_bf16(f[2 * e] - h.x, f[2 * e + 1] - h.y);
      }
      *reinterpret_cast<uint4*>(g.aux_out + (long long)row * g.ldaux + col) = make_uint4(lo[0], lo[1], lo[2], lo[3]);
    }
  }
  *reinterpret_cast<uint4*>(reinterpret_cast<__nv_bfloat16*>(g.out) + (long long)row * g.ldo + col) = make_uint4(w[0], w[1], w[2], w[3]);
}

// Cluster size (splits) is a launch attribute: 1, 2, 4 or 8, with BN / splits >= 8.
template <int BN, int MODE>
__global__ void __launch_bounds__(SPLIT_THREADS, BN <= 64 ? 2 : 1)
gemm_split_kernel(const __grid_constant__ CUtensorMap tmap_a, const __grid_constant__ CUtensorMap tmap_b, GemmArgs g) {
  using L = SplitSmem<BN>;
  constexpr int NSTAGE = L::NSTAGE;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint64_t* full_bar = reinterpret_cast<uint64_t*>(smem + L::BAR_OFFSET);
  uint64_t* empty_bar = full_bar + NSTAGE;
  uint64_t* acc_full = empty_bar + NSTAGE;
  uint32_t* tmem_holder = reinterpret_cast<uint32_t*>(acc_full + 1);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_holder + 1);

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int S = g.split_k;
  const int ks = int(blockIdx.x) & (S - 1);                // rank in the cluster = slice of K
  const int tile = int(blockIdx.x) / S;
  const int tiles_m = (g.M + BM - 1) / BM;
  const int m0 = (tile % tiles_m) * BM, n0 = (tile / tiles_m) * BN;
  const int kb_total = (g.K + BK - 1) / BK;
  // slices differ by at most one k-block; the launcher sees to it that none is empty
  const int kb0 = int((long long)kb_total * ks / S), kb1 = int((long long)kb_total * (ks + 1) / S);

  if (threadIdx.x == 0) {
    for (int s = 0; s < NSTAGE; ++s) { mbar_init(&full_bar[s], 1); mbar_init(&empty_bar[s], 1); }
    mbar_init(acc_full, 1);
    *abort_flag = 0;
    mbar_fence_init();
    fence_proxy_async();
  }
  if (warp == SPLIT_MMA_WARP) {
    tmem_alloc(tmem_holder, BN);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  if (S > 1) cluster_arrive();          // phase 1: every CTA of the cluster has started
  const uint32_t tmem_base = *tmem_holder;

  // Output units of eight columns; CTA ks of the cluster finishes units [ks * UW, (ks + 1) * UW).
  constexpr int U = BN / 8;
  const int lgS = 31 - __clz(S), UW = U >> lgS;
  const auto owner_of = [lgS](int u) { return (u << lgS) / U; };
  bool ok = true;

  if (warp == SPLIT_TMA_WARP) {
    // ------------------------------------------------------------ producer (the whole warp, one lane issues)
    const auto load_b = [&](int i) {
      uint8_t* sb = smem + (i % NSTAGE) * L::STAGE_BYTES + L::A_BYTES;
      uint64_t* bar = &full_bar[i % NSTAGE];
      const int k0 = (kb0 + i) * BK;
      if (!g.b_mn_major) {
        tma_load_2d(sb, &tmap_b, bar, k0, n0);
      } else {
#pragma unroll
        for (int c = 0; c < (BN + 63) / 64; ++c) tma_load_2d(sb + c * 8192, &tmap_b, bar, n0 + 64 * c, k0);
      }
    };
    const int nkb = kb1 - kb0;
    int early = 0;                      // stages whose B operand is already on its way
    if (g.b_static) {
      early = nkb < NSTAGE ? nkb : NSTAGE;
      if (elect_one()) {
        for (int i = 0; i < early; ++i) { mbar_expect_tx(&full_bar[i], L::STAGE_BYTES); load_b(i); }
        for (int i = early; i < nkb; ++i) {                       // the rest is asked into L2
          const int k0 = (kb0 + i) * BK;
          if (!g.b_mn_major) {
            tma_prefetch_l2_2d(&tmap_b, k0, n0);
          } else {
#pragma unroll
            for (int c = 0; c < (BN + 63) / 64; ++c) tma_prefetch_l2_2d(&tmap_b, n0 + 64 * c, k0);
          }
        }
      }
      __syncwarp();
    }
    pdl_wait();
    pdl_launch();
    for (int i = 0; i < nkb; ++i) {
      const int s = i % NSTAGE;
      if (i >= NSTAGE && !mbar_wait_warp(&empty_bar[s], ((i / NSTAGE) & 1) ^ 1, abort_flag, g.status)) break;
      if (elect_one()) {
        if (i >= early) { mbar_expect_tx(&full_bar[s], L::STAGE_BYTES); load_b(i); }
        tma_load_2d(smem + s * L::STAGE_BYTES, &tmap_a, &full_bar[s], (kb0 + i) * BK, m0);
      }
      __syncwarp();
    }
  } else if (warp == SPLIT_MMA_WARP) {
    // ------------------------------------------------------------ MMA issuer (the whole warp, one lane issues)
    const uint32_t idesc = make_idesc_bf16(BM, BN, 0, g.b_mn_major);
    const uint32_t desc_hi = smem_desc_hi(1024);
    const uint32_t b_lbo = g.b_mn_major ? 8192 : 16, b_step = g.b_mn_major ? (2048 >> 4) : (32 >> 4);
    for (int i = 0; i < kb1 - kb0; ++i) {
      const int s = i % NSTAGE;
      if (!mbar_wait_warp(&full_bar[s], (i / NSTAGE) & 1, abort_flag, g.status)) { ok = false; break; }
      const uint32_t sa = smem_u32(smem + s * L::STAGE_BYTES);
      const uint32_t a_lo = smem_desc_lo(sa, 16), b_lo = smem_desc_lo(sa + L::A_BYTES, b_lbo);
      if (elect_one()) {
#pragma unroll
        for (int k = 0; k < BK / UMMA_K; ++k)
          umma_bf16_lohi(tmem_base, a_lo + k * (32 >> 4), b_lo + k * b_step, desc_hi, idesc, i > 0 || k > 0);
        umma_commit(&empty_bar[s]);
      }
      __syncwarp();
    }
    if (ok && elect_one()) umma_commit(acc_full);
    __syncwarp();
  }

  if (warp < SPLIT_EPI_WARPS) {
    // ------------------------------------------------------------ epilogue: thread = row and half of the columns
    const int quarter = warp & 3, half = warp >> 2;
    const int r = quarter * 32 + lane, row = m0 + r;
    constexpr int UT = U / 2;           // units of this thread: u0 .. u0 + UT - 1
    const int u0 = half * UT;
    constexpr bool EXTRA = MODE == EPI_RESID || MODE == EPI_MUL || MODE == EPI_MUL_SUM;
    uint4 x[EXTRA ? UT : 1], t[MODE == EPI_RESID ? UT : 1];
    // Everything from global memory is asked for before the accumulator is waited for, the bias (older than the kernel
    // before, like the weights) even before that kernel has ended.
    float* bias = reinterpret_cast<float*>(smem + L::BIAS_OFFSET) + warp * (BN / 2);
    const auto load_bias = [&] {
#pragma unroll
      for (int c = lane; c < BN / 2; c += 32) {
        const int col = n0 + u0 * 8 + c;
        bias[c] = g.bias != nullptr && col < g.N ? __ldg(g.bias + col) : 0.f;
      }
      __syncwarp();
    };
    if (g.b_static) load_bias();
    pdl_wait();
    if (!g.b_static) load_bias();
    if constexpr (EXTRA) {
      const __nv_bfloat16* src = MODE == EPI_RESID ? g.resid : g.aux_in;
      const long long ld = MODE == EPI_RESID ? g.ldr : g.ldaux;
#pragma unroll
      for (int i = 0; i < UT; ++i) {
        const int col = n0 + (u0 + i) * 8;
        const bool in = owner_of(u0 + i) == ks && row < g.M && col < g.N;
        x[i] = in ? *reinterpret_cast<const uint4*>(src + (long long)row * ld + col) : make_uint4(0, 0, 0, 0);
        if constexpr (MODE == EPI_RESID)
          t[i] = in && g.aux_in != nullptr ? *reinterpret_cast<const uint4*>(g.aux_in + (long long)row * g.ldaux + col)
                                           : make_uint4(0, 0, 0, 0);
      }
    }
    ok = mbar_wait(acc_full, 0, abort_flag, g.status);
    tc_fence_after();
    uint32_t v[UT * 8];
    const uint32_t t_addr = tmem_base + (uint32_t(quarter * 32) << 16) + u0 * 8;
    if constexpr (UT == 2) tmem_ld_32x16(t_addr, v);
    else if constexpr (UT == 4) tmem_ld_32x32(t_addr, v);
    else {
      tmem_ld_32x32(t_addr, *reinterpret_cast<uint32_t(*)[32]>(v));
      tmem_ld_32x32(t_addr + 32, *reinterpret_cast<uint32_t(*)[32]>(v + 32));
    }
    tmem_ld_wait();
    uint8_t* recv = smem + L::RECV_OFFSET;
    if (S > 1) {
      // the other CTAs' columns go to their owners: 16 bytes per lane, one row after the other
      const uint32_t recv_addr = smem_u32(recv);
      cluster_wait();
#pragma unroll
      for (int i = 0; i < UT; ++i) {
        const int u = u0 + i, owner = owner_of(u);
        if (owner != ks) {
          const int slot = ks < owner ? ks : ks - 1;              // sources in rank order, the owner left out
          const uint32_t at = map_to_cta(recv_addr, owner) + ((slot * UW + (u - owner * UW)) * 2 * BM + r) * 16;
          const uint32_t* q = &v[i * 8];
          st_cluster_v4(at, q[0], q[1], q[2], q[3]);
          st_cluster_v4(at + BM * 16, q[4], q[5], q[6], q[7]);
        }
      }
      cluster_arrive();                 // phase 2: all partial sums have been delivered
      cluster_wait();
    }
#pragma unroll
    for (int i = 0; i < UT; ++i) {
      const int u = u0 + i, col = n0 + u * 8;
      float out8[MODE == EPI_MUL_SUM ? 8 : 1];          // of a row that exists, else zeros
      if constexpr (MODE == EPI_MUL_SUM) {
#pragma unroll
        for (int e = 0; e < 8; ++e) out8[e] = 0.f;
      }
      if (owner_of(u) == ks && row < g.M && col < g.N && ok) {
        const uint32_t* q = &v[i * 8];
        float f[8];
#pragma unroll
        for (int e = 0; e < 8; ++e) f[e] = __uint_as_float(q[e]);
        for (int src = 0; src < S - 1; ++src) {
          const float4* p = reinterpret_cast<const float4*>(recv + ((src * UW + (u - ks * UW)) * 2 * BM + r) * 16);
          const float4 lo = p[0], hi = p[BM];
          f[0] += lo.x; f[1] += lo.y; f[2] += lo.z; f[3] += lo.w;
          f[4] += hi.x; f[5] += hi.y; f[6] += hi.z; f[7] += hi.w;
        }
        {
          const float4 lo = *reinterpret_cast<const float4*>(bias + i * 8), hi = *reinterpret_cast<const float4*>(bias + i * 8 + 4);
          f[0] += lo.x; f[1] += lo.y; f[2] += lo.z; f[3] += lo.w;
          f[4] += hi.x; f[5] += hi.y; f[6] += hi.z; f[7] += hi.w;
        }
        if constexpr (EXTRA) finish_unit<MODE>(g, row, col, f, x[i], t[MODE == EPI_RESID ? i : 0]);
        else finish_unit<MODE>(g, row, col, f, make_uint4(0, 0, 0, 0), make_uint4(0, 0, 0, 0));
        if constexpr (MODE == EPI_MUL_SUM) {
#pragma unroll
          for (int e = 0; e < 8; ++e) out8[e] = f[e];
        }
      }
      if constexpr (MODE == EPI_MUL_SUM) {
        if (owner_of(u) == ks && col < g.N) {          // the same for the whole warp
          const float sum = warp_sums(out8);
          if ((lane & 3) == 0) atomicAdd(g.colsum + col + (lane >> 2), sum);
        }
      }
    }
  } else if (S > 1) {
    cluster_wait();
    cluster_arrive();
    cluster_wait();
  }

  tc_fence_before();
  __syncthreads();
  if (warp == SPLIT_MMA_WARP) {
    tc_fence_after();
    tmem_dealloc(tmem_base, BN);
  }
}

int launch_split(int bn, const CUtensorMap& ta, const CUtensorMap& tb, const GemmArgs& g, cudaStream_t st);
int load_split_kernels();

}  // namespace dsw
