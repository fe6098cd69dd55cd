// Causal flash attention forward on tcgen05 tensor cores, head size 64 or 32.
//
// Replaces the reference's F.scaled_dot_product_attention(q, k, v, is_causal=True)
// (src/model.py:66-67).  Input is the packed [B*T, 3*d] output of the QKV
// projection (Q | K | V, head h at columns h*hs of each part); output is the
// [B*T, d] tensor that feeds the output projection, plus the per-row log-sum-exp
// that the backward pass needs.
//
// A work item is (128 query rows, batch, head); persistent CTAs walk the items.
// Warps 0-3 own one query row per thread: they read the score row from tensor
// memory once, do the online softmax on it in registers and write P to tensor
// memory.  The output row stays in tensor memory: every P V product accumulates
// onto it, and the row threads rescale it in place only when the running maximum
// has grown by more than 2^8 since the last rescale (until then P is computed
// against the older maximum, which is exact algebra and safe in bf16/fp32 range).
// Warp 4 issues the MMAs, warp 5 the TMA loads.
//   S = Q K_j^T          A = Q  [128 x 64]  K-major,  B = K_j [128 x 64] K-major   -> TMEM, 128 columns
//   O_j = P V_j          A = P  [128 x 128] in TMEM, 64 columns of bf16 pairs,  B = V_j [128 x 64] N-major -> TMEM, 64 columns
// P by way of shared memory cost 64 KB of its bandwidth per tile, written and read by the product, of the 144 KB that a tile took
// (128 bytes per clock; us, before / now: 32 x 1024 tokens, 12 heads of 64, 121.7 / 115.4; 8 x 1024, 16 heads 44.6 / 42.3; 16 x 133,
// 12 heads 12.6 / 12.1; 64 x 1024, 4 heads of 32, 80.6 / 76.5).  A quarter to a half of the exponentials on the FMA pipe instead: slower
// by 6 to 20 %, here as in the backward.
// K/V tiles are double buffered; two CTAs fit on an SM (97 KB shared memory,
// 256 TMEM columns each), so one CTA's MMAs run under the other's softmax.
// Only kv tiles up to the diagonal are visited; the diagonal tile is masked.
//
// The tensor maps describe the matrices as (head's columns, head, row, sequence).  Head size 32 (the 4-head, 128-wide
// test model) runs the same tiles: the 64-column box reaches past the head, so TMA fills the right half of each
// operand tile with zeros.  Q K^T and dO V^T are unchanged by the zero columns, the output tiles get zero
// right halves, and only the first 32 columns are written.
#include <cuda.h>
#include "ptx.cuh"
#include "launch.h"
#include "tmap.h"
#include "attention_short_bwd.cuh"
#include "dswarm.h"

namespace dsw {

// [128 x 64] operand tile of column block `cb` (= part * heads + head) at `row` of sequence b.  The sequence is a dimension
// of the maps, so a tile that reaches past its sequence's end holds zeros there and never a row of the next one, whose
// infinities or NaN would spoil this one's products (0 x Inf); stores and reductions end there as well.
// Per call against maps over all rows at once: forward unchanged; backward of 32 x 1024 tokens, 12 heads of 64, 370 -> 336 us,
// 16 x 133 29.9 -> 28.5, 64 x 1024, 4 heads of 32, whose dK and dV had left row by row, 205 -> 186.
__device__ __forceinline__ void att_load_tile(void* dst, const CUtensorMap* tm, uint64_t* bar, int cb, int row, int b) {
  tma_load_4d(dst, tm, bar, 0, cb, row, b);
}

// Optional in-kernel timeline for tuning: when a trace buffer is registered (dsw_attention_set_trace),
// CTA 0 stores %globaltimer values at its phase boundaries: [0,256) row-warp 0, [256,512) MMA thread.
__device__ __forceinline__ long long gtimer() {
  long long t;
  asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
  return t;
}
// In-kernel timeline stamps exist only in the tracing build (-DDSWARM_TRACE, benchmarks/timelines.py).
#ifdef DSWARM_TRACE
#define ATT_TRACE(buf, base, slot) do { if ((buf) != nullptr && (slot) < 256) (buf)[(base) + (slot)++] = gtimer(); } while (0)
#else
#define ATT_TRACE(buf, base, slot) do { } while (0)
#endif

constexpr int ATT_BQ = 128;        // query rows per work item
constexpr int ATT_BK = 128;        // kv rows per step
constexpr int ATT_HS = 64;
constexpr int ATT_THREADS = 256;          // warps 0-3 softmax, 4 MMA, 5 TMA, 6-7 only lend their registers
constexpr int ATT_TILE_BYTES = 128 * 64 * 2;     // one [128 x 64] bf16 tile

struct AttSmem {
  static constexpr int Q_OFF = 0;
  static constexpr int K_OFF = Q_OFF + ATT_TILE_BYTES;            // 2 stages
  static constexpr int V_OFF = K_OFF + 2 * ATT_TILE_BYTES;        // 2 stages
  static constexpr int O_OFF = V_OFF + 2 * ATT_TILE_BYTES;        // output rows on their way out, [128 rows][64]
  static constexpr int BAR_OFF = O_OFF + ATT_TILE_BYTES;
  // Two CTAs share an SM only if each stays under (227 KB - 2 KB) / 2 = 115200 bytes, so
  // there is no room for alignment slack: the dynamic segment is declared 1024-aligned
  // and the kernel checks that it really is.
  static constexpr int TOTAL = BAR_OFF + 128;
};

// max(a, b, c) in one instruction (sm_100 has the three-input form)
__device__ __forceinline__ float fmax3(float a, float b, float c) {
  float d;
  asm("max.f32 %0, %1, %2, %3;" : "=f"(d) : "f"(a), "f"(b), "f"(c));
  return d;
}

__device__ __forceinline__ float fast_exp2(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}

// byte offset of element (row, col) of a [128 x 128] bf16 operand stored as two
// 64-column k-blocks in the 128-byte-swizzled K-major layout
__device__ __forceinline__ uint32_t p_offset(int row, int col) {
  const int kb = col >> 6, c = col & 63;
  return kb * ATT_TILE_BYTES + row * 128 + ((((c >> 3) ^ (row & 7)) << 4) | ((c & 7) << 1));
}

// Work items of a persistent launch: item = (query or kv tile, batch*head), listed heaviest first; CTA c of G
// takes items c, 2G-1-c, 2G+c, ... (a snake over the rounds), which evens out the tile counts per CTA.
// Returns false when round r holds no item for this CTA.
__device__ __forceinline__ bool att_item(int r, int c, int G, int total, int& idx) {
  idx = r * G + ((r & 1) ? G - 1 - c : c);
  return idx < total;
}

// SOLO: no more items than SMs.  A row then goes straight from its thread, 16 bytes at a time: staged through shared memory as
// the rows of more items are, it leaves some 0.4 us later (1 x 24 tokens, 4 heads of 32, before sequences of one tile had a
// kernel of their own: 6.4 -> 6.0 us a launch; 5 x 24, 12 heads of 64: 6.5 -> 6.1).  With two CTAs on an SM the stores of a row per lane get in each other's way: 16 x 128, 12 heads,
// 192 items, 9.1 us staged, 10.0 not.
template <bool SOLO>
__global__ void __launch_bounds__(ATT_THREADS, 2)
attention_fwd_kernel(const __grid_constant__ CUtensorMap tmap_qkv, __nv_bfloat16* __restrict__ out,
                     float* __restrict__ lse_out, int T, int nh, int n_bh, int hs, float scale_log2, int* status,
                     long long* trace) {
  extern __shared__ __align__(1024) uint8_t smem_raw[];
  uint8_t* smem = smem_raw;
  if (smem_u32(smem) & 1023) {            // swizzled operand tiles need 1024-byte alignment
    if (threadIdx.x == 0 && status) atomicCAS(status, 0, ST_BAD_ARG);
    return;
  }
  // Every barrier below completes one phase per kv tile (q_full / q_empty: per work item), counted over the
  // whole life of the CTA: g is the number of tiles, w the number of items this CTA has finished.
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + AttSmem::BAR_OFF);
  uint64_t* q_full = bars;            // Q of the item loaded
  uint64_t* kv_full = bars + 1;       // 2 stages
  uint64_t* kv_empty = bars + 3;      // 2 stages
  uint64_t* s_full = bars + 5;        // S ready in TMEM
  uint64_t* p_full = bars + 6;        // P written to TMEM (4 warps arrive)
  uint64_t* o_full = bars + 7;        // P V accumulated in TMEM
  uint64_t* o_free = bars + 8;        // per item: the output rows have been read out of TMEM (4 warps arrive)
  uint64_t* s_free = bars + 9;        // S read out of TMEM (4 warps arrive)
  uint64_t* q_empty = bars + 10;      // all S products of the item done: Q may be overwritten
  uint32_t* tmem_holder = reinterpret_cast<uint32_t*>(bars + 11);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_holder + 1);

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int nq = (T + ATT_BQ - 1) / ATT_BQ;
  const int total = nq * n_bh;
  const int G = gridDim.x, cta = blockIdx.x;
  const int rounds = (total + G - 1) / G;
  const int d = nh * hs;
  long long* tr = blockIdx.x == 0 ? trace : nullptr;
  int tslot = 0;

  if (threadIdx.x == 0) {
    mbar_init(q_full, 1); mbar_init(q_empty, 1);
    for (int i = 0; i < 2; ++i) { mbar_init(&kv_full[i], 1); mbar_init(&kv_empty[i], 1); }
    mbar_init(s_full, 1); mbar_init(p_full, 4); mbar_init(o_full, 1); mbar_init(o_free, 4);
    mbar_init(s_free, 4);
    *abort_flag = 0;
    mbar_fence_init();
    fence_proxy_async();
  }
  if (warp == 4) {
    tmem_alloc(tmem_holder, 256);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  // Two CTAs share the SM's registers: 128 per thread at launch.  The softmax warps keep a whole score row
  // (128 values) in registers, so their warpgroup takes 216 and the other warpgroup (one MMA-issuing and one
  // TMA-issuing thread) drops to 40.
  // (each role changes its own allotment at the top of its branch)
  const uint32_t tmem_base = *tmem_holder;
  const uint32_t tmem_s = tmem_base;            // 128 columns
  const uint32_t tmem_o = tmem_base + 128;      // 64 columns
  const uint32_t tmem_p = tmem_base + 192;      // 64 columns: P, two bf16 values to a column

  if (warp >= 4) {
    asm volatile("setmaxnreg.dec.sync.aligned.u32 40;");          // the whole warpgroup, one instruction
  }
  if (warp >= 6) {
    // nothing to do: these warps exist so that the register hand-over works on whole warpgroups
  } else if (warp == 5) {
    // ------------------------------------------------------------ TMA producer (the whole warp, one lane issues)
    if (elect_one()) tma_prefetch_desc(&tmap_qkv);
    pdl_wait();
    uint32_t g = 0, w = 0;
    bool ok = true;
    for (int r = 0; r < rounds && ok; ++r) {
      int idx;
      if (!att_item(r, cta, G, total, idx)) continue;
      const int qi = nq - 1 - idx / n_bh, bh = idx % n_bh;
      const int b = bh / nh, h = bh - b * nh;
      if (w > 0 && !mbar_wait_warp(q_empty, (w - 1) & 1, abort_flag, status)) break;
      if (elect_one()) {
        mbar_expect_tx(q_full, ATT_TILE_BYTES);
        att_load_tile(smem + AttSmem::Q_OFF, &tmap_qkv, q_full, h, qi * ATT_BQ, b);
      }
      __syncwarp();
      for (int j = 0; j <= qi; ++j, ++g) {
        const int s = g & 1;
        if (!mbar_wait_warp(&kv_empty[s], ((g >> 1) & 1) ^ 1, abort_flag, status)) { ok = false; break; }
        const int kvrow = j * ATT_BK;
        if (elect_one()) {
          mbar_expect_tx(&kv_full[s], 2 * ATT_TILE_BYTES);
          att_load_tile(smem + AttSmem::K_OFF + s * ATT_TILE_BYTES, &tmap_qkv, &kv_full[s], nh + h, kvrow, b);
          att_load_tile(smem + AttSmem::V_OFF + s * ATT_TILE_BYTES, &tmap_qkv, &kv_full[s], 2 * nh + h, kvrow, b);
        }
        __syncwarp();
      }
      ++w;
    }
    pdl_launch();
  } else if (warp == 4) {
    // ------------------------------------------------------------ MMA issuer (the whole warp, one lane issues)
    if (lane != 0) tr = nullptr;
    const uint32_t idesc_s = make_idesc_bf16(128, 128, 0, 0);
    const uint32_t idesc_o = make_idesc_bf16(128, 64, 0, 1);
    const uint32_t desc_hi = smem_desc_hi(1024);
    const uint32_t q_lo = smem_desc_lo(smem_u32(smem + AttSmem::Q_OFF), 16);
    // S of global tile gt = Q K^T into the (single) score buffer; `first` / `last`: position in its item wi
    auto issue_s = [&](uint32_t gt, uint32_t wi, bool first, bool last) -> bool {
      if (first && !mbar_wait_warp(q_full, wi & 1, abort_flag, status)) return false;
      const int st = gt & 1;
      if (!mbar_wait_warp(&kv_full[st], (gt >> 1) & 1, abort_flag, status)) return false;
      const uint32_t k_lo = smem_desc_lo(smem_u32(smem + AttSmem::K_OFF + st * ATT_TILE_BYTES), 16);
      if (elect_one()) {
#pragma unroll
        for (int k = 0; k < ATT_HS / 16; ++k)
          umma_bf16_lohi(tmem_s, q_lo + k * 2, k_lo + k * 2, desc_hi, idesc_s, k > 0);
        umma_commit(s_full);
        if (last) umma_commit(q_empty);
      }
      __syncwarp();
      ATT_TRACE(tr, 256, tslot);          // S issued
      return true;
    };
    uint32_t g = 0, w = 0;
    bool ok = true;
    for (int r = 0; r < rounds && ok; ++r) {
      int idx;
      if (!att_item(r, cta, G, total, idx)) continue;
      const int n_kv = nq - idx / n_bh;
      // the item after this one (its first score tile is issued during this item's last tile)
      int next_n_kv = 0;
      for (int r2 = r + 1, idx2; r2 < rounds; ++r2)
        if (att_item(r2, cta, G, total, idx2)) { next_n_kv = nq - idx2 / n_bh; break; }
      if (g == 0) ok = issue_s(0, 0, true, n_kv == 1);
      for (int j = 0; j < n_kv && ok; ++j, ++g) {
        const int s = g & 1;
        const uint32_t v_lo = smem_desc_lo(smem_u32(smem + AttSmem::V_OFF + s * ATT_TILE_BYTES), ATT_TILE_BYTES);
        // The next score tile goes first, as soon as the softmax warps have read this one for the last
        // time (they are still turning its last columns into P): they need the next S next, while the
        // P V product is only folded in after their first pass over it.
        const bool more = j + 1 < n_kv;
        if (more || next_n_kv > 0) {
          if (!mbar_wait_warp(s_free, g & 1, abort_flag, status)) { ok = false; break; }
          tc_fence_after();
          const bool okk = more ? issue_s(g + 1, w, false, j + 2 == n_kv) : issue_s(g + 1, w + 1, true, next_n_kv == 1);
          if (!okk) { ok = false; break; }
        }
        // P of this tile is in tensor memory (and the output rows are rescaled if they had to be)
        if (!mbar_wait_warp(p_full, g & 1, abort_flag, status)) { ok = false; break; }
        ATT_TRACE(tr, 256, tslot);          // P ready
        // a new item starts its output from zero: the previous item's must have been read out
        if (j == 0 && w > 0 && !mbar_wait_warp(o_free, (w - 1) & 1, abort_flag, status)) { ok = false; break; }
        tc_fence_after();
        if (elect_one()) {
#pragma unroll
          for (int k = 0; k < ATT_BK / 16; ++k)
            umma_bf16_ts(tmem_o, tmem_p + k * 8, v_lo + k * (2048 >> 4), desc_hi, idesc_o, (j > 0 || k > 0));
          umma_commit(o_full);
          umma_commit(&kv_empty[s]);
        }
        __syncwarp();
        ATT_TRACE(tr, 256, tslot);          // PV issued
      }
      ++w;
    }
  } else {
    // ------------------------------------------------------------ softmax + output (thread = query row)
    asm volatile("setmaxnreg.inc.sync.aligned.u32 216;");
    const int r = warp * 32 + lane;                      // row within the tile = TMEM lane
    const uint32_t lane_addr = uint32_t(warp * 32) << 16;
    if (threadIdx.x != 0) tr = nullptr;
    uint32_t g = 0;
    bool ok = true;
    for (int rr = 0; rr < rounds && ok; ++rr) {
      int idx;
      if (!att_item(rr, cta, G, total, idx)) continue;
      const int qi = nq - 1 - idx / n_bh, bh = idx % n_bh;
      const int b = bh / nh, h = bh - b * nh;
      const int n_kv = qi + 1;
      float m = -INFINITY, l = 0.f;           // m: the maximum P is computed against (log2 units)
      for (int j = 0; j < n_kv && ok; ++j, ++g) {
        ATT_TRACE(tr, 0, tslot);              // waiting for S
        if (!mbar_wait(s_full, g & 1, abort_flag, status)) { ok = false; break; }
        tc_fence_after();
        ATT_TRACE(tr, 0, tslot);              // S arrived
        // the whole score row into registers; the score buffer is free for the next tile at once
        uint32_t v[4][32];
#pragma unroll
        for (int c = 0; c < 4; ++c) tmem_ld_32x32(tmem_s + lane_addr + c * 32, v[c]);
        tmem_ld_wait();
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(s_free);
        const bool diag = j == qi;
        // Row maximum (four independent chains).  On the diagonal tile only columns <= r count: of the warp's four
        // 32-column chunks those left of its rows are whole, the one above its rows is masked column by column, and
        // those right of it are empty and cost nothing (masking all four made a diagonal tile, every 4.5th of 1024
        // tokens, the dearest one).
        const int whole = diag ? warp : 4;
        float mx4[4] = {-INFINITY, -INFINITY, -INFINITY, -INFINITY};
#pragma unroll
        for (int c = 0; c < 4; ++c) {
          if (c < whole) {
#pragma unroll
            for (int i = 0; i < 32; i += 8) {
              mx4[0] = fmax3(mx4[0], __uint_as_float(v[c][i]), __uint_as_float(v[c][i + 1]));
              mx4[1] = fmax3(mx4[1], __uint_as_float(v[c][i + 2]), __uint_as_float(v[c][i + 3]));
              mx4[2] = fmax3(mx4[2], __uint_as_float(v[c][i + 4]), __uint_as_float(v[c][i + 5]));
              mx4[3] = fmax3(mx4[3], __uint_as_float(v[c][i + 6]), __uint_as_float(v[c][i + 7]));
            }
          } else if (c == whole) {
#pragma unroll
            for (int i = 0; i < 32; ++i)
              if (i <= lane) mx4[i & 3] = fmaxf(mx4[i & 3], __uint_as_float(v[c][i]));
          }
        }
        const float mx = fmaxf(fmaxf(mx4[0], mx4[1]), fmaxf(mx4[2], mx4[3])) * scale_log2;
        ATT_TRACE(tr, 0, tslot);              // maximum done
        if (j == 0) {
          m = mx;
        } else {
          // the previous product must be done: it reads the P that is about to be overwritten, and it
          // accumulates onto the output rows that may be rescaled here
          if (!mbar_wait(o_full, (g - 1) & 1, abort_flag, status)) { ok = false; break; }
          const bool grow = mx > m + 8.f;
          if (__any_sync(0xffffffffu, grow)) {          // rare after the first tiles
            tc_fence_after();
            const float alpha = grow ? fast_exp2(m - mx) : 1.f;
            if (grow) { m = mx; l *= alpha; }
#pragma unroll
            for (int c0 = 0; c0 < ATT_HS; c0 += 32) {
              uint32_t ov[32];
              tmem_ld_32x32(tmem_o + lane_addr + c0, ov);
              tmem_ld_wait();
#pragma unroll
              for (int i = 0; i < 32; ++i) ov[i] = __float_as_uint(__uint_as_float(ov[i]) * alpha);
              tmem_st_32x32(tmem_o + lane_addr + c0, ov);
            }
            tmem_st_wait();
          }
        }
        ATT_TRACE(tr, 0, tslot);              // output rows ready for the next product
        // probabilities -> tensor memory (bf16), row sum
        f2 sum2[2] = {f2_bcast(0.f), f2_bcast(0.f)};      // packed pairs (two columns per instruction)
        const f2 sc2 = f2_bcast(scale_log2), nm2 = f2_bcast(-m);
#pragma unroll
        for (int c = 0; c < 4; ++c) {
          uint32_t pk[16];
          if (c <= whole) {
            const bool masked = c == whole;
#pragma unroll
            for (int i = 0; i < 32; i += 2) {
              float x0, x1;
              f2_split(f2_fma(f2_make(__uint_as_float(v[c][i]), __uint_as_float(v[c][i + 1])), sc2, nm2), x0, x1);
              float p0 = fast_exp2(x0), p1 = fast_exp2(x1);
              if (masked) {
                p0 = i <= lane ? p0 : 0.f;
                p1 = i + 1 <= lane ? p1 : 0.f;
              }
              sum2[(i >> 1) & 1] = f2_add(sum2[(i >> 1) & 1], f2_make(p0, p1));
              pk[i >> 1] = pack_bf16(p0, p1);
            }
          } else {
#pragma unroll
            for (int i = 0; i < 16; ++i) pk[i] = 0;
          }
          tmem_st_32x16(tmem_p + lane_addr + c * 16, pk);
        }
        {
          float a0, a1;
          f2_split(f2_add(sum2[0], sum2[1]), a0, a1);
          l += a0 + a1;
        }
        ATT_TRACE(tr, 0, tslot);              // P written
        tmem_st_wait();
        tc_fence_before();            // orders P and the rescaled output rows before the product that follows the arrive
        __syncwarp();
        if (lane == 0) mbar_arrive(p_full);
      }
      if (!ok || !mbar_wait(o_full, (g - 1) & 1, abort_flag, status)) { ok = false; break; }
      tc_fence_after();
      const float inv = 1.f / l;
      const bool in_seq = qi * ATT_BQ + r < T;             // a last tile may reach past the sequence's end
      uint32_t ov[2][32];
      tmem_ld_32x32(tmem_o + lane_addr, ov[0]);
      tmem_ld_32x32(tmem_o + lane_addr + 32, ov[1]);
      tmem_ld_wait();
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(o_free);          // the next item's first product may overwrite the rows
      if constexpr (SOLO) {
        __nv_bfloat16* dst = out + ((long long)b * T + qi * ATT_BQ + r) * d + h * hs;
#pragma unroll
        for (int c = 0; c < 8; ++c)
          if (c * 8 < hs && in_seq) {
            const uint32_t* o = ov[c >> 2] + (c & 3) * 8;
            *reinterpret_cast<uint4*>(dst + c * 8) = make_uint4(pack_bf16(__uint_as_float(o[0]) * inv, __uint_as_float(o[1]) * inv),
                                                                pack_bf16(__uint_as_float(o[2]) * inv, __uint_as_float(o[3]) * inv),
                                                                pack_bf16(__uint_as_float(o[4]) * inv, __uint_as_float(o[5]) * inv),
                                                                pack_bf16(__uint_as_float(o[6]) * inv, __uint_as_float(o[7]) * inv));
          }
      } else {
        // The warp's 32 rows pass through shared memory, so that a store
        // covers four whole rows of 128 bytes: a lane that stores its own row 16 bytes at a time touches 32 lines with
        // every instruction (32 x 1024 tokens, 12 heads of 64: 135.6 -> 129.0 us; 16 x 1024: 72.9 -> 68.6).
        uint8_t* so = smem + AttSmem::O_OFF + warp * 32 * 128;
#pragma unroll
        for (int c = 0; c < 8; ++c) {
          const uint32_t* o = ov[c >> 2] + (c & 3) * 8;
          *reinterpret_cast<uint4*>(so + lane * 128 + ((c ^ (lane & 7)) << 4)) =
              make_uint4(pack_bf16(__uint_as_float(o[0]) * inv, __uint_as_float(o[1]) * inv),
                         pack_bf16(__uint_as_float(o[2]) * inv, __uint_as_float(o[3]) * inv),
                         pack_bf16(__uint_as_float(o[4]) * inv, __uint_as_float(o[5]) * inv),
                         pack_bf16(__uint_as_float(o[6]) * inv, __uint_as_float(o[7]) * inv));
        }
        __syncwarp();
        const int ch = lane & 7, t0 = qi * ATT_BQ + warp * 32 + (lane >> 3);
        __nv_bfloat16* dst = out + ((long long)b * T + t0) * d + h * hs + ch * 8;
#pragma unroll
        for (int i = 0; i < 8; ++i) {
          const int rl = i * 4 + (lane >> 3);
          const uint4 w = *reinterpret_cast<const uint4*>(so + rl * 128 + ((ch ^ (rl & 7)) << 4));
          if (t0 + i * 4 < T && ch * 8 < hs) *reinterpret_cast<uint4*>(dst + (long long)i * 4 * d) = w;
        }
        __syncwarp();                                // read out before the next item's rows are written here
      }
      // natural-log LSE of the scaled scores
      if (in_seq) lse_out[(long long)bh * T + qi * ATT_BQ + r] = (m + log2f(l)) * 0.6931471805599453f;
    }
  }

  tc_fence_before();
  __syncthreads();
  if (warp == 4) {
    tc_fence_after();
    tmem_dealloc(tmem_base, 256);
  }
}


// ------------------------------------------------------------------ backward
// One CTA per (128 kv rows, batch, head); it walks the query tiles i >= j (causal).
// Per query tile, with thread = query row for the softmax algebra:
//   S  = Q_i K_j^T,  dP = dO_i V_j^T                         -> TMEM (2 x 128 columns)
//   P  = exp(S*scale - lse),  dS = P * (dP - D) * scale      -> shared memory, bf16, swizzled
//   dV += P^T dO_i,  dK += dS^T Q_i   (accumulate in TMEM over i),  dQ_i = dS K_j (fresh)
// The P / dS tiles are written once and read through two descriptors: K-major
// (rows = queries) for dQ, and M-major (rows of the transposed operand = kv) for dV / dK;
// the [128 x 64] Q_i, dO_i, K_j tiles likewise serve as K-major A and as N-major B.
// dQ is accumulated across kv tiles with fp32 bulk reductions into a scratch tensor
// and converted to bf16 afterwards; dK and dV leave as two bulk stores per item.
//
// Eleven warps.  Row warps 0-7 (thread = query row, two threads per row, 64 columns each):
// wait sdp_full, take S and dP out of TMEM in one load group, arrive sdp_read, compute P / dS
// in registers, wait dq_full of the step before (its products read P / dS), write P / dS,
// arrive pds_full, then stage the dQ of the step before for the reducer.  MMA warp (a whole
// warp on uniform values, a lane elected around each instruction): issues the S / dP pair of
// step i+1 as soon as sdp_read of step i is complete (also for the first step of the next work
// item: K and V are double-buffered by item parity), then, on pds_full, dV, dK (releasing the
// Q / dO stage), dQ.  TMA warp (likewise): K / V of the item into the buffer of its parity,
// Q / dO pairs into two stages.  Reducer warp (one lane): one bulk reduce-add per staged dQ tile, two bulk stores per item for dK / dV
// (staged by the row warps in the P buffer).
// Sequences of one tile have an instantiation of their own (ONE, below); where the caller asks for the column sums of dqkv
// (LaunchMode::colsum), the row threads leave those of dK and dV in shared memory with the tiles.
// Every wait is bounded; a wait that runs out sets the CTA's abort flag and the status word.
struct AttBwdSmem {
  static constexpr int KV_BYTES = 2 * ATT_TILE_BYTES;               // K_j then V_j
  static constexpr int K_OFF = 0;                                   // 2 buffers (item parity) of (K, V)
  static constexpr int V_OFF = K_OFF + ATT_TILE_BYTES;
  static constexpr int QSTAGES = 2;                                 // (Q_i, dO_i) pairs in flight
  static constexpr int Q_OFF = K_OFF + 2 * KV_BYTES;
  static constexpr int DO_OFF = Q_OFF + QSTAGES * ATT_TILE_BYTES;
  static constexpr int P_OFF = DO_OFF + QSTAGES * ATT_TILE_BYTES;   // 2 k-blocks
  static constexpr int DS_OFF = P_OFF + 2 * ATT_TILE_BYTES;         // 2 k-blocks
  static constexpr int DQ_OFF = DS_OFF + 2 * ATT_TILE_BYTES;        // fp32 [2 halves][128 rows][32], 128-byte swizzled
  static constexpr int BAR_OFF = DQ_OFF + 2 * ATT_TILE_BYTES;
  static constexpr int SUM_OFF = BAR_OFF + 256;                     // column sums of dK and dV: fp32 [lane quarter][2][64]
  // no room for alignment slack: the segment is declared 1024-aligned, and the kernel checks that it is
  static constexpr int TOTAL = SUM_OFF + 4 * 2 * 64 * 4;
  // sequences of one tile stage dQ in half of its buffer; behind that dQ's column sums, D, and rows of O for the next D
  static constexpr int ONE_SUM_OFF = DQ_OFF + ATT_TILE_BYTES;       // fp32 [lane quarter][64]
  static constexpr int ONE_D_OFF = ONE_SUM_OFF + 1024;              // fp32 [2 item parities][128 rows]
  static constexpr int ONE_O_OFF = ONE_D_OFF + 1024;                // [8 row warps][3 pieces][32 lanes] of 16 bytes
};

// D[bh, t] = sum_c dO[t, h*hs + c] * O[t, h*hs + c], and dq_acc[t, :] = 0.  One warp per token row: 16-byte
// loads, one head's hs columns lie in hs/8 neighbouring lanes (hs = 64 or 32), which a few shuffles add up.
__global__ void __launch_bounds__(256)
attention_bwd_prep_kernel(const __nv_bfloat16* out, const __nv_bfloat16* dout,
                          float* __restrict__ D, float* __restrict__ dq_acc, int B, int T, int nh, int hs) {
  const int lane = threadIdx.x & 31;
  const int d = nh * hs, chunks = d >> 3, lanes_per_head = hs >> 3;
  const long long rows = (long long)B * T;
  pdl_wait();
  pdl_launch();
  const long long warps = ((long long)gridDim.x * blockDim.x) >> 5;
  for (long long row = ((long long)blockIdx.x * blockDim.x + threadIdx.x) >> 5; row < rows; row += warps) {
    const int b = int(row / T), t = int(row - (long long)b * T);
    const uint4* po = reinterpret_cast<const uint4*>(out + row * d);
    const uint4* pg = reinterpret_cast<const uint4*>(dout + row * d);
    float4* pz = reinterpret_cast<float4*>(dq_acc + row * d);
    for (int u0 = 0; u0 < chunks; u0 += 32) {
      const int u = u0 + lane;
      float v = 0.f;
      if (u < chunks) {
        v = dot8(po[u], pg[u]);
        pz[2 * u] = make_float4(0.f, 0.f, 0.f, 0.f);
        pz[2 * u + 1] = make_float4(0.f, 0.f, 0.f, 0.f);
      }
      for (int o = lanes_per_head >> 1; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
      if (u < chunks && (lane & (lanes_per_head - 1)) == 0) D[((long long)b * nh + u / lanes_per_head) * T + t] = v;
    }
  }
}

// dqkv[:, 0:d] = bf16(dq_acc); a thread keeps to eight columns, whose sums over all rows go to colsum (optional).
// A block has `width` threads to a row, and a grid column for every 8 * width columns.
__global__ void __launch_bounds__(512)
attention_dq_convert_kernel(const float* dq_acc, __nv_bfloat16* __restrict__ dqkv, long long rows, int d, int width, float* colsum) {
  extern __shared__ float cvt_sums[];                // [rows per step][8 * width], with colsum
  pdl_wait();
  pdl_launch();
  const int per_step = blockDim.x / width, rl = threadIdx.x / width, cl = (threadIdx.x - rl * width) * 8;
  const int col0 = blockIdx.y * width * 8, col = col0 + cl;
  float s[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
  const long long step = (long long)gridDim.x * per_step;
#pragma unroll 4
  for (long long row = (long long)blockIdx.x * per_step + rl; row < rows && col < d; row += step) {
    const float4 a = *reinterpret_cast<const float4*>(dq_acc + row * d + col);
    const float4 b = *reinterpret_cast<const float4*>(dq_acc + row * d + col + 4);
    *reinterpret_cast<uint4*>(dqkv + row * 3 * d + col) =
        make_uint4(pack_bf16(a.x, a.y), pack_bf16(a.z, a.w), pack_bf16(b.x, b.y), pack_bf16(b.z, b.w));
    s[0] += a.x; s[1] += a.y; s[2] += a.z; s[3] += a.w;
    s[4] += b.x; s[5] += b.y; s[6] += b.z; s[7] += b.w;
  }
  if (colsum == nullptr) return;
  float4* mine = reinterpret_cast<float4*>(cvt_sums + rl * width * 8 + cl);
  mine[0] = make_float4(s[0], s[1], s[2], s[3]);
  mine[1] = make_float4(s[4], s[5], s[6], s[7]);
  __syncthreads();
  for (int c = threadIdx.x; c < width * 8 && col0 + c < d; c += blockDim.x) {
    float v = 0.f;
    for (int k = 0; k < per_step; ++k) v += cvt_sums[k * width * 8 + c];
    atomicAdd(colsum + col0 + c, v);
  }
}

// 32 columns of one query row: P = exp2(S * scale_log2 - lse2), dS = P * (dP - D) * scale, both packed to bf16
// pairs.  MASKED: columns past `r` (above the diagonal) give zero.
template <bool MASKED, int N>
__device__ __forceinline__ void bwd_row_chunk(const uint32_t (&sv)[N], const uint32_t (&dpv)[N], uint32_t* pk_p,
                                              uint32_t* pk_ds, int c0, int r, float scale_log2, float lse2,
                                              float Dr, float scale) {
  // packed fp32 pairs: one instruction per two columns for everything but the exponentials and the packing
  const f2 sc = f2_bcast(scale_log2), nl = f2_bcast(-lse2), s2 = f2_bcast(scale), nd = f2_bcast(-Dr * scale);
#pragma unroll
  for (int c = 0; c < N; c += 2) {
    const f2 x = f2_fma(f2_make(__uint_as_float(sv[c]), __uint_as_float(sv[c + 1])), sc, nl);
    float x0, x1;
    f2_split(x, x0, x1);
    float p0 = fast_exp2(x0), p1 = fast_exp2(x1);
    if (MASKED) {
      p0 = c0 + c <= r ? p0 : 0.f;
      p1 = c0 + c + 1 <= r ? p1 : 0.f;
    }
    const f2 u = f2_fma(f2_make(__uint_as_float(dpv[c]), __uint_as_float(dpv[c + 1])), s2, nd);    // (dP - D) * scale
    pk_p[c >> 1] = pack_bf16(p0, p1);
    pk_ds[c >> 1] = pack_bf16_f2(f2_mul(f2_make(p0, p1), u));
  }
}

constexpr int ATT_BWD_ROW_WARPS = 8;     // two per TMEM lane quarter: each thread takes half of its row's columns
constexpr int ATT_BWD_THREADS = 32 * (ATT_BWD_ROW_WARPS + 3);    // + MMA issuer, TMA producer, dQ reducer

// Column sums of dqkv (a bias gradient) meet in global memory by bulk reductions that the reducer warp issues, 64 columns
// of 32 rows each: a row thread that adds to global memory itself finds its next barrier waiting for that (32 x 1024
// tokens: 328 -> 387 us; with a warp of its own that read the staged tiles 396, since the next item's P waits for it).
__device__ __forceinline__ void bulk_add(float* to, const void* from, int bytes) {
  asm volatile("cp.reduce.async.bulk.global.shared::cta.bulk_group.add.f32 [%0], [%1], %2;" ::"l"(to), "r"(smem_u32(from)), "r"(bytes)
               : "memory");
}
// The sums over the warp's 32 rows of a thread's 32 columns, a column per lane.
__device__ __forceinline__ float column_sum(const uint32_t (&row)[32]) {
  float v[32];
#pragma unroll
  for (int i = 0; i < 32; ++i) v[i] = __uint_as_float(row[i]);
  return warp_sums(v);
}

// D = rowsum(dO O) of 16 rows of a sequence of one tile by a warp, LPR lanes (hs / 8) to a row, added up in the order of
// attention_bwd_prep_kernel.  piece(i, r, o, g): a lane's eight values of O and dO in row r (of the 16), the i-th it has.
template <int LPR, class F>
__device__ __forceinline__ void row_dots16(float* to, int lane, F&& piece) {
  constexpr int N = LPR / 2, RPI = 32 / LPR;          // pieces, rows per piece
  float v[N];
#pragma unroll
  for (int i = 0; i < N; ++i) {
    uint4 o, g;
    piece(i, i * RPI + lane / LPR, o, g);
    v[i] = dot8(o, g);
  }
  // over the lanes of a row, each step with half as many rows
#pragma unroll
  for (int n = N / 2, x = LPR / 2; n >= 1; n >>= 1, x >>= 1) {
    const bool up = lane & x;
#pragma unroll
    for (int i = 0; i < n; ++i) {
      const float keep = up ? v[i + n] : v[i], send = up ? v[i] : v[i + n];
      v[i] = keep + __shfl_xor_sync(0xffffffffu, send, x);
    }
  }
  v[0] += __shfl_xor_sync(0xffffffffu, v[0], 1);
  if (!(lane & 1)) to[((lane & (LPR - 1)) >> 1) * RPI + lane / LPR] = v[0];
}

// A row warp's 16 rows of D, item by item.  O of an item is asked for a whole item ahead: three of a lane's four pieces
// into shared memory, where there is no room for four, and one into registers; dO is in its stage.  Loaded when they are
// wanted, the pieces came from DRAM while the row warps waited (64 x 128 tokens, 12 heads of 64: 45 us a launch, this
// way 37; by a warp of its own 38).
template <int LPR>
struct ItemDots {
  static __device__ __forceinline__ uint4 load(const __nv_bfloat16* p, int r, int d, int rows, int lane) {
    return r < rows ? *reinterpret_cast<const uint4*>(p + (long long)r * d + (lane & (LPR - 1)) * 8) : make_uint4(0, 0, 0, 0);
  }
  // o, g: the head's columns of the first of the 16 rows; `rows` of them lie within the sequence
  static __device__ __forceinline__ void first(const __nv_bfloat16* o, const __nv_bfloat16* g, int d, int rows, float* to, int lane) {
    row_dots16<LPR>(to, lane, [&](int, int r, uint4& ov, uint4& gv) { ov = load(o, r, d, rows, lane); gv = load(g, r, d, rows, lane); });
  }
  static __device__ __forceinline__ void fetch(const __nv_bfloat16* o, int d, int rows, uint4* mine, uint4& last, int lane) {
#pragma unroll
    for (int i = 0; i < LPR / 2; ++i) {
      const int r = i * (32 / LPR) + lane / LPR;
      if (i < 3) cp_async16(mine + i * 32, r < rows ? o + (long long)r * d + (lane & (LPR - 1)) * 8 : o, r < rows);
      else       last = load(o, r, d, rows, lane);
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  }
  // tile: the 128 rows of dO, row0: the first of the 16
  static __device__ __forceinline__ void finish(const uint8_t* tile, int row0, const uint4* mine, const uint4& last, float* to, int lane) {
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    row_dots16<LPR>(to, lane, [&](int i, int r, uint4& ov, uint4& gv) {
      ov = i < 3 ? mine[i * 32] : last;
      gv = *reinterpret_cast<const uint4*>(tile + (row0 + r) * 128 + (((lane & (LPR - 1)) ^ ((row0 + r) & 7)) << 4));
    });
  }
};

// ONE: sequences of a single tile (T <= 128), heads of 64 (of 32: attention_short_bwd.cuh).  Every item is one step, and dQ
// needs no sum over kv tiles, so it leaves as bf16 with dK and dV.  D is computed by the row warps, 16 rows each, that of the
// next item under the products of this one.  No accumulator, and neither of the kernels around this one (which clear it and
// compute D, and convert it).  The results are those of the three kernels, bit for bit: 64 x 128 tokens, 12 heads of 64,
// 45.7 -> 36.8 us; 16 x 128, 16 heads, 23.9 -> 16.9; 200 x 64, 12 heads, 95.4 -> 84.0.  (With D as the row sum of P dP, which is
// another rounding and has the two warps of a row wait for each other inside the row algebra: 33.1, 15.4, 77.0.)
template <bool ONE>
__global__ void __launch_bounds__(ATT_BWD_THREADS, 1)
attention_bwd_kernel(const __grid_constant__ CUtensorMap tmap_qkv, const __grid_constant__ CUtensorMap tmap_do,
                     const __grid_constant__ CUtensorMap tmap_dq, const __grid_constant__ CUtensorMap tmap_dkv,
                     const __nv_bfloat16* out, const __nv_bfloat16* dout, const float* lse, const float* Dvec, int T, int nh,
                     int n_bh, int hs, int item0, int total, float scale, float* colsum, int* status, long long* trace) {
  using L = AttBwdSmem;
  extern __shared__ __align__(1024) uint8_t smem_raw[];
  uint8_t* smem = smem_raw;
  if (smem_u32(smem) & 1023) {
    if (threadIdx.x == 0 && status) atomicCAS(status, 0, ST_BAD_ARG);
    return;
  }
  // Persistent: one CTA per SM walks work items (kv tile, batch*head).  The per-step barriers complete one
  // phase per step, kv_full / kv_empty / dkv_free one per item, counted over the life of the CTA
  // (g = steps done, w = items done).
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + L::BAR_OFF);
  uint64_t* kv_full = bars;            // 2: K, V of the item loaded (buffer = item parity)
  uint64_t* kv_empty = bars + 2;       // 2: every MMA of the item done: its K, V may be overwritten
  uint64_t* q_full = bars + 4;         // QSTAGES stages of (Q_i, dO_i)
  uint64_t* q_empty = bars + 6;        // QSTAGES
  uint64_t* sdp_full = bars + 8;       // S and dP ready
  uint64_t* pds_full = bars + 9;       // P and dS in shared memory (8 warps arrive)
  uint64_t* dq_full = bars + 10;       // dV/dK/dQ MMAs of this step done
  uint64_t* dq_free = bars + 11;       // dQ read out of TMEM (8 warps arrive)
  uint64_t* dkv_free = bars + 12;      // dK, dV of the item read out of TMEM (8 warps arrive)
  uint64_t* sdp_read = bars + 13;      // S and dP of this step read out of TMEM (8 warps arrive)
  uint64_t* dq_staged = bars + 14;     // dQ of this step staged in shared memory (8 warps arrive)
  uint64_t* dq_stage_free = bars + 15; // the reduction of this step's dQ has read the staging tile
  uint64_t* dkv_staged = bars + 16;    // dK, dV of the item staged in the P buffer (8 warps arrive; hs = 64)
  uint64_t* dkv_stored = bars + 17;    // their bulk stores have read the P buffer
  uint64_t* dots_full = bars + 18;     // D of the item in shared memory (8 warps arrive; ONE)
  uint32_t* tmem_holder = reinterpret_cast<uint32_t*>(bars + 19);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_holder + 1);

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int nq = (T + ATT_BQ - 1) / ATT_BQ;
  // items item0 .. item0 + total - 1, heaviest first: kv tile 0 meets every query tile
  const auto next_item = [=](int r, int& idx) {
    const bool is = att_item(r, int(blockIdx.x), int(gridDim.x), total, idx);
    idx += item0;
    return is;
  };
  const int rounds = (total + int(gridDim.x) - 1) / int(gridDim.x);
  const int d = nh * hs;
  const float scale_log2 = scale * 1.4426950408889634f;
  long long* tr = blockIdx.x == 0 ? trace : nullptr;
  int tslot = 0;

  if (threadIdx.x == 0) {
    for (int i = 0; i < 2; ++i) { mbar_init(&kv_full[i], 1); mbar_init(&kv_empty[i], 1); }
    for (int i = 0; i < L::QSTAGES; ++i) { mbar_init(&q_full[i], 1); mbar_init(&q_empty[i], 1); }
    mbar_init(sdp_full, 1); mbar_init(pds_full, ATT_BWD_ROW_WARPS); mbar_init(dq_full, 1);
    mbar_init(dq_free, ATT_BWD_ROW_WARPS); mbar_init(dkv_free, ATT_BWD_ROW_WARPS);
    mbar_init(sdp_read, ATT_BWD_ROW_WARPS);
    mbar_init(dq_staged, ATT_BWD_ROW_WARPS); mbar_init(dq_stage_free, 1);
    mbar_init(dkv_staged, ATT_BWD_ROW_WARPS); mbar_init(dkv_stored, 1);
    mbar_init(dots_full, ATT_BWD_ROW_WARPS);
    *abort_flag = 0;
    mbar_fence_init();
    fence_proxy_async();
  }
  constexpr int MMA_WARP = ATT_BWD_ROW_WARPS, TMA_WARP = ATT_BWD_ROW_WARPS + 1, RED_WARP = ATT_BWD_ROW_WARPS + 2;
  if (warp == MMA_WARP) {
    tmem_alloc(tmem_holder, 512);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_holder;
  const uint32_t tm_s = tmem_base, tm_dp = tmem_base + 128, tm_dv = tmem_base + 256, tm_dk = tmem_base + 320,
                 tm_dq = tmem_base + 384;

  if (warp == TMA_WARP) {
    // ------------------------------------------------------------ TMA producer (the whole warp, one lane issues)
    if (elect_one()) {
      tma_prefetch_desc(&tmap_qkv);
      tma_prefetch_desc(&tmap_do);
    }
    pdl_wait();
    uint32_t g = 0, w = 0;
    bool ok = true;
    for (int r = 0; r < rounds && ok; ++r) {
      int idx;
      if (!next_item(r, idx)) continue;
      const int j = idx / n_bh, bh = idx % n_bh;
      const int b = bh / nh, h = bh - b * nh;
      const int steps = nq - j;
      // K and V of the item go into the buffer of its parity, free since the item two back finished: they
      // are on their way while the item before still runs
      const int kb = w & 1;
      if (!mbar_wait_warp(&kv_empty[kb], ((w >> 1) & 1) ^ 1, abort_flag, status)) break;
      const int kvrow = j * ATT_BK;
      if (elect_one()) {
        mbar_expect_tx(&kv_full[kb], 2 * ATT_TILE_BYTES);
        att_load_tile(smem + L::K_OFF + kb * L::KV_BYTES, &tmap_qkv, &kv_full[kb], nh + h, kvrow, b);
        att_load_tile(smem + L::V_OFF + kb * L::KV_BYTES, &tmap_qkv, &kv_full[kb], 2 * nh + h, kvrow, b);
      }
      __syncwarp();
      for (int it = 0; it < steps; ++it, ++g) {
        const int s = g % L::QSTAGES;
        if (!mbar_wait_warp(&q_empty[s], ((g / L::QSTAGES) & 1) ^ 1, abort_flag, status)) { ok = false; break; }
        const int qrow = (j + it) * ATT_BQ;
        if (elect_one()) {
          mbar_expect_tx(&q_full[s], 2 * ATT_TILE_BYTES);
          att_load_tile(smem + L::Q_OFF + s * ATT_TILE_BYTES, &tmap_qkv, &q_full[s], h, qrow, b);
          att_load_tile(smem + L::DO_OFF + s * ATT_TILE_BYTES, &tmap_do, &q_full[s], h, qrow, b);
          // The pair two steps on is asked into L2 now: its load can only start when its stage is released, and
          // the time from there to the data is on the issuing thread's path.
          if (hs == 64 && it + 2 < steps) {
            tma_prefetch_l2_4d(&tmap_qkv, 0, h, qrow + 2 * ATT_BQ, b);
            tma_prefetch_l2_4d(&tmap_do, 0, h, qrow + 2 * ATT_BQ, b);
          }
        }
        __syncwarp();
      }
      ++w;
    }
    pdl_launch();
  } else if (warp == MMA_WARP) {
    // ------------------------------------------------------------ MMA issuer (the whole warp, one lane issues)
    if (lane != 0) tr = nullptr;
    const uint32_t id_s = make_idesc_bf16(128, 128, 0, 0);      // Q K^T and dO V^T
    const uint32_t id_t = make_idesc_bf16(128, 64, 1, 1);       // P^T dO and dS^T Q : A M-major, B N-major
    const uint32_t id_q = make_idesc_bf16(128, 64, 0, 1);       // dS K : A K-major, B N-major
    // Descriptor low words: K-major operands (leading offset 16) step 32 bytes per MMA, M/N-major ones
    // (leading offset = one tile) step 16 rows of 128 bytes; the high word is the same for all.
    constexpr uint32_t KSTEP = 32 >> 4, MNSTEP = 2048 >> 4, TILE16 = ATT_TILE_BYTES >> 4;
    const uint32_t desc_hi = smem_desc_hi(1024);
    // K and V descriptors of buffer 0; buffer 1 lies KVBUF16 further
    const uint32_t k_km0 = smem_desc_lo(smem_u32(smem + L::K_OFF), 16), v_km0 = smem_desc_lo(smem_u32(smem + L::V_OFF), 16);
    const uint32_t k_mn0 = smem_desc_lo(smem_u32(smem + L::K_OFF), ATT_TILE_BYTES);
    constexpr uint32_t KVBUF16 = L::KV_BYTES >> 4;
    const uint32_t p_mn = smem_desc_lo(smem_u32(smem + L::P_OFF), ATT_TILE_BYTES);
    const uint32_t ds_mn = smem_desc_lo(smem_u32(smem + L::DS_OFF), ATT_TILE_BYTES);
    const uint32_t ds_km = smem_desc_lo(smem_u32(smem + L::DS_OFF), 16);
    uint32_t g = 0, w = 0;
    bool ok = true;
    // S = Q K^T and dP = dO V^T of global step gs, which belongs to item wi (operands: Q/dO stage
    // gs % QSTAGES, K/V buffer wi & 1).  The row threads must have read the pair of the step before out of
    // TMEM; the first step of an item also waits for its K and V.
    auto issue_sdp = [&](uint32_t gs, uint32_t wi, bool first_of_item) -> bool {
      const int st = gs % L::QSTAGES, kb = wi & 1;
      if (gs > 0 && !mbar_wait_warp(sdp_read, (gs - 1) & 1, abort_flag, status)) return false;
      if (first_of_item && !mbar_wait_warp(&kv_full[kb], (wi >> 1) & 1, abort_flag, status)) return false;
      if (!mbar_wait_warp(&q_full[st], (gs / L::QSTAGES) & 1, abort_flag, status)) return false;
      tc_fence_after();
      const uint32_t q_km = smem_desc_lo(smem_u32(smem + L::Q_OFF + st * ATT_TILE_BYTES), 16);
      const uint32_t do_km = smem_desc_lo(smem_u32(smem + L::DO_OFF + st * ATT_TILE_BYTES), 16);
      const uint32_t k_km = k_km0 + kb * KVBUF16, v_km = v_km0 + kb * KVBUF16;
      if (elect_one()) {
#pragma unroll
        for (int k = 0; k < 4; ++k) umma_bf16_lohi(tm_s, q_km + k * KSTEP, k_km + k * KSTEP, desc_hi, id_s, k > 0);
#pragma unroll
        for (int k = 0; k < 4; ++k) umma_bf16_lohi(tm_dp, do_km + k * KSTEP, v_km + k * KSTEP, desc_hi, id_s, k > 0);
        umma_commit(sdp_full);
      }
      __syncwarp();
      ATT_TRACE(tr, 256, tslot);          // S, dP issued
      return true;
    };
    for (int r = 0; r < rounds && ok; ++r) {
      int idx;
      if (!next_item(r, idx)) continue;
      const int steps = nq - idx / n_bh;
      bool more = false;                  // does this CTA have another item after this one?
      for (int r2 = r + 1; r2 < rounds && !more; ++r2) {
        int idx2;
        more = next_item(r2, idx2);
      }
      const int kb = w & 1;
      const uint32_t k_mn = k_mn0 + kb * KVBUF16;
      if (w == 0) ok = issue_sdp(0, 0, true);
      for (int it = 0; it < steps && ok; ++it, ++g) {
        const int s = g % L::QSTAGES;
        const uint32_t sq = smem_u32(smem + L::Q_OFF + s * ATT_TILE_BYTES);
        const uint32_t sdo = smem_u32(smem + L::DO_OFF + s * ATT_TILE_BYTES);
        const uint32_t q_mn = smem_desc_lo(sq, ATT_TILE_BYTES), do_mn = smem_desc_lo(sdo, ATT_TILE_BYTES);
        // The next step's pair goes as soon as the row threads have S and dP of this one in registers, while
        // they are still writing P / dS: they find it finished when they come back for it.  Across items
        // too: the next item's K and V sit in the other buffer.
        if (it + 1 < steps) {
          if (!issue_sdp(g + 1, w, false)) { ok = false; break; }
        } else if (more) {
          if (!issue_sdp(g + 1, w + 1, true)) { ok = false; break; }
        }
        if (!mbar_wait_warp(pds_full, g & 1, abort_flag, status)) { ok = false; break; }
        ATT_TRACE(tr, 256, tslot);          // P, dS ready
        // a new item starts its dV / dK sums from zero: the previous item's must have been read out
        if (it == 0 && w > 0 && !mbar_wait_warp(dkv_free, (w - 1) & 1, abort_flag, status)) { ok = false; break; }
        tc_fence_after();
        if (elect_one()) {
#pragma unroll
          for (int k = 0; k < 8; ++k)       // dV += P^T dO_i   (K = query rows, 16 per step)
            umma_bf16_lohi(tm_dv, p_mn + k * MNSTEP, do_mn + k * MNSTEP, desc_hi, id_t, (it > 0 || k > 0));
#pragma unroll
          for (int k = 0; k < 8; ++k)       // dK += dS^T Q_i
            umma_bf16_lohi(tm_dk, ds_mn + k * MNSTEP, q_mn + k * MNSTEP, desc_hi, id_t, (it > 0 || k > 0));
          umma_commit(&q_empty[s]);         // Q_i and dO_i have their last readers queued: the stage reloads early
        }
        __syncwarp();
        // the previous step's dQ has been read out of TMEM (the row threads do that right after their hand-over)
        if (g > 0 && !mbar_wait_warp(dq_free, (g - 1) & 1, abort_flag, status)) { ok = false; break; }
        tc_fence_after();
        if (elect_one()) {
#pragma unroll
          for (int k = 0; k < 8; ++k)       // dQ_i = dS K_j     (K = kv rows)
            umma_bf16_lohi(tm_dq, ds_km + (k >> 2) * TILE16 + (k & 3) * KSTEP, k_mn + k * MNSTEP, desc_hi, id_q, k > 0);
          umma_commit(dq_full);
          if (it + 1 == steps) umma_commit(&kv_empty[kb]);
        }
        __syncwarp();
        ATT_TRACE(tr, 256, tslot);          // dV, dK, dQ issued
      }
      ++w;
    }
  } else if (warp == RED_WARP) {
    // ------------------------------------------------------------ dQ reducer
    // One TMA reduce-add per staged dQ tile into the fp32 dQ scratch.  Issuing a bulk reduction can hold the
    // issuing thread for most of a microsecond while earlier reductions drain into L2, so a thread of its own
    // does it: nothing on a row thread's path waits for global atomics.
    if (lane == 0) {
      uint32_t g = 0, w = 0;
      bool ok = true;
      for (int rr = 0; rr < rounds && ok; ++rr) {
        int idx;
        if (!next_item(rr, idx)) continue;
        const int j = idx / n_bh, bh = idx % n_bh;
        const int b = bh / nh, h = bh - b * nh;
        for (int i = j; i < nq; ++i, ++g) {
          if (!mbar_wait(dq_staged, g & 1, abort_flag, status)) { ok = false; break; }
          if constexpr (ONE) {
            asm volatile("cp.async.bulk.tensor.4d.global.shared::cta.tile.bulk_group [%0, {%1, %2, %3, %4}], [%5];"
                         ::"l"(&tmap_dkv), "r"(0), "r"(h), "r"(0), "r"(b), "r"(smem_u32(smem + L::DQ_OFF))
                         : "memory");
            for (int q = 0; q < 4 && colsum != nullptr; ++q) bulk_add(colsum + h * hs, smem + L::ONE_SUM_OFF + q * 256, hs * 4);
          } else
          for (int hh = 0; hh * 32 < hs; ++hh)          // 32 columns per head: the first staging half is the whole dQ tile
            asm volatile("cp.reduce.async.bulk.tensor.4d.global.shared::cta.add.tile.bulk_group [%0, {%1, %2, %3, %4}], [%5];"
                         ::"l"(&tmap_dq), "r"(hh * 32), "r"(h), "r"(i * ATT_BQ), "r"(b),
                           "r"(smem_u32(smem + L::DQ_OFF + hh * ATT_TILE_BYTES))
                         : "memory");
          asm volatile("cp.async.bulk.commit_group;" ::: "memory");
          asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory");
          mbar_arrive(dq_stage_free);
        }
        if (ok) {
          // dK and dV of the item: two [128 x 64] bf16 tiles staged in the P buffer, one bulk store each
          if (!mbar_wait(dkv_staged, w & 1, abort_flag, status)) break;
#pragma unroll
          for (int which = 0; which < 2; ++which)
            asm volatile("cp.async.bulk.tensor.4d.global.shared::cta.tile.bulk_group [%0, {%1, %2, %3, %4}], [%5];"
                         ::"l"(&tmap_dkv), "r"(0), "r"((which + 1) * nh + h), "r"(j * ATT_BK), "r"(b),
                           "r"(smem_u32(smem + L::P_OFF + which * ATT_TILE_BYTES))
                         : "memory");
          for (int q = 0; q < 8 && colsum != nullptr; ++q)
            bulk_add(colsum + ((q & 1) + 1) * d + h * hs, smem + L::SUM_OFF + q * 256, hs * 4);
          asm volatile("cp.async.bulk.commit_group;" ::: "memory");
          asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory");
          mbar_arrive(dkv_stored);
        }
        ++w;
      }
      asm volatile("cp.async.bulk.wait_group 0;" ::: "memory");     // reductions and stores complete before exit
    }
  } else {
    // ------------------------------------------------------------ row threads
    const int q4 = warp & 3, half = warp >> 2;     // TMEM lane quarter, column half
    const int r = q4 * 32 + lane;
    const uint32_t lane_addr = uint32_t(q4 * 32) << 16;
    uint8_t* sp = smem + L::P_OFF;
    uint8_t* sds = smem + L::DS_OFF;
    bool ok = true;
    if (threadIdx.x != 0) tr = nullptr;
    uint8_t* sdq = smem + L::DQ_OFF + half * ATT_TILE_BYTES;     // this thread's half: [128 rows][32 fp32]
    uint32_t g = 0, w = 0;
    float lse_next = 0.f, D_next = 0.f;
    pdl_wait();
    // dQ of global step gs: TMEM -> registers -> swizzled shared tile, which the reducer warp adds into the
    // fp32 dQ scratch.
    auto drain_dq = [&](uint32_t gs) -> bool {
      if (!mbar_wait(dq_full, gs & 1, abort_flag, status)) return false;
      tc_fence_after();
      ATT_TRACE(tr, 0, tslot);                // dQ product done
      uint32_t v[32];
      tmem_ld_32x32(tm_dq + lane_addr + half * 32, v);
      tmem_ld_wait();
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(dq_free);
      // the previous reduction must have finished reading the staging tile
      if (gs > 0 && !mbar_wait(dq_stage_free, (gs - 1) & 1, abort_flag, status)) return false;
      ATT_TRACE(tr, 0, tslot);                // the previous reduction has let go of the staging tile
      if constexpr (ONE) {          // one [128 x 64] bf16 tile
        if (colsum != nullptr) reinterpret_cast<float*>(smem + L::ONE_SUM_OFF)[q4 * 64 + half * 32 + lane] = column_sum(v);
#pragma unroll
        for (int c = 0; c < 4; ++c)
          *reinterpret_cast<uint4*>(smem + L::DQ_OFF + r * 128 + (((half * 4 + c) ^ (r & 7)) << 4)) = make_uint4(
              pack_bf16(__uint_as_float(v[8 * c]), __uint_as_float(v[8 * c + 1])),
              pack_bf16(__uint_as_float(v[8 * c + 2]), __uint_as_float(v[8 * c + 3])),
              pack_bf16(__uint_as_float(v[8 * c + 4]), __uint_as_float(v[8 * c + 5])),
              pack_bf16(__uint_as_float(v[8 * c + 6]), __uint_as_float(v[8 * c + 7])));
      } else {
#pragma unroll
        for (int c = 0; c < 8; ++c)
          *reinterpret_cast<uint4*>(sdq + r * 128 + ((c ^ (r & 7)) << 4)) = make_uint4(v[4 * c], v[4 * c + 1], v[4 * c + 2], v[4 * c + 3]);
      }
      fence_proxy_async();
      __syncwarp();
      if (lane == 0) mbar_arrive(dq_staged);
      ATT_TRACE(tr, 0, tslot);                // staged
      return true;
    };
    // this warp's 16 rows of D of an item (ONE)
    const int dot_row = q4 * 32 + half * 16;
    uint4* const o_mine = reinterpret_cast<uint4*>(smem + L::ONE_O_OFF) + warp * 96 + lane;
    uint4 o_last = make_uint4(0, 0, 0, 0);
    const auto dots_at = [&](int bh) {          // the first of the rows, or of the sequence where they lie behind it
      return ((long long)(bh / nh) * T + (dot_row < T ? dot_row : 0)) * d + (bh % nh) * hs;
    };
    const auto dots_to = [&](uint32_t item) { return reinterpret_cast<float*>(smem + L::ONE_D_OFF) + (item & 1) * 128 + dot_row; };
    const auto dots_done = [&] {
      __syncwarp();
      if (lane == 0) mbar_arrive(dots_full);
    };
    const auto dots_fetch = [&](int bh) {
      ItemDots<8>::fetch(out + dots_at(bh), d, T - dot_row, o_mine, o_last, lane);
    };
    const auto dots_finish = [&](uint32_t item) -> bool {
      const int s = item % L::QSTAGES;
      if (!mbar_wait(&q_full[s], (item / L::QSTAGES) & 1, abort_flag, status)) return false;
      const uint8_t* tile = smem + L::DO_OFF + s * ATT_TILE_BYTES;
      ItemDots<8>::finish(tile, dot_row, o_mine, o_last, dots_to(item), lane);
      dots_done();
      return true;
    };
    if (ONE) {                        // the CTA's first item, while its tiles are on their way
      int idx;
      next_item(0, idx);          // there is one: G <= total
      const long long at = dots_at(idx % n_bh);
      ItemDots<8>::first(out + at, dout + at, d, T - dot_row, dots_to(0), lane);
      dots_done();
    }
    for (int rr = 0; rr < rounds && ok; ++rr) {
      int idx;
      if (!next_item(rr, idx)) continue;
      const int j = idx / n_bh, bh = idx % n_bh;
      const int steps = nq - j;
      // where the next item's first step finds its row statistics (-1: this is the CTA's last item)
      int stat_after = -1, bh_after = -1;
      for (int r2 = rr + 1; r2 < rounds; ++r2) {
        int idx2;
        if (next_item(r2, idx2)) {
          // a row past the end of the sequence: its statistics are never used
          bh_after = idx2 % n_bh;
          stat_after = (idx2 / n_bh) * ATT_BQ + r < T ? bh_after * T + (idx2 / n_bh) * ATT_BQ + r : -1;
          break;
        }
      }
      for (int it = 0; it < steps && ok; ++it, ++g) {
        const int i = j + it;
        const int stat = bh * T + i * ATT_BQ + r;       // < 2^31: the launcher checks B * nh * T
        // row statistics: loaded for the CTA's first step, fetched one step ahead (across items too) after that
        // Rows past the end of the sequence (last tile of a length that is no multiple of 128), which the tiles hold
        // as zeros, have an infinite log-sum-exp: their P and dS come out as zeros and add nothing.
        const bool in_seq = i * ATT_BQ + r < T;
        if (g == 0 && in_seq) { lse_next = lse[stat]; if (!ONE) D_next = Dvec[stat]; }
        const float lse2 = in_seq ? lse_next * 1.4426950408889634f : INFINITY;
        float Dr = in_seq ? D_next : 0.f;
        if (ONE && bh_after >= 0) dots_fetch(bh_after);
        ATT_TRACE(tr, 0, tslot);              // step start
        if (!mbar_wait(sdp_full, g & 1, abort_flag, status)) { ok = false; break; }
        if constexpr (ONE) {          // a buffer is written again when every warp has handed over the item in between
          if (!mbar_wait(dots_full, g & 1, abort_flag, status)) { ok = false; break; }
          Dr = reinterpret_cast<const float*>(smem + L::ONE_D_OFF)[(g & 1) * 128 + r];
        }
        tc_fence_after();
        {
          const int sn = it + 1 < steps ? ((i + 1) * ATT_BQ + r < T ? stat + ATT_BQ : -1) : stat_after;
          if (sn >= 0) { lse_next = lse[sn]; if (!ONE) D_next = Dvec[sn]; }
        }
        ATT_TRACE(tr, 0, tslot);              // S, dP arrived
        // P and dS of this thread's 64 columns, in registers: the previous step's products may still be
        // reading the shared P / dS tiles
        uint32_t pk_p[2][16], pk_ds[2][16];
        {
          // all 64 columns of S and of dP leave TMEM in one go (a TMEM load takes a few hundred nanoseconds from
          // issue to data, whatever its width: four loads in a row would cost four such waits)
          uint32_t raw[4][2][16];
#pragma unroll
          for (int q = 0; q < 4; ++q) {
            tmem_ld_32x16(tm_s + lane_addr + half * 64 + q * 16, raw[q][0]);
            tmem_ld_32x16(tm_dp + lane_addr + half * 64 + q * 16, raw[q][1]);
          }
          tmem_ld_wait();
#pragma unroll
          for (int q = 0; q < 4; ++q) {
            const int c0 = half * 64 + q * 16;
            uint32_t* op = &pk_p[q >> 1][(q & 1) * 8];
            uint32_t* ods = &pk_ds[q >> 1][(q & 1) * 8];
            if (it == 0) bwd_row_chunk<true, 16>(raw[q][0], raw[q][1], op, ods, c0, r, scale_log2, lse2, Dr, scale);
            else         bwd_row_chunk<false, 16>(raw[q][0], raw[q][1], op, ods, c0, r, scale_log2, lse2, Dr, scale);
          }
        }
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(sdp_read);   // S and dP are in registers: the next pair may replace them
        ATT_TRACE(tr, 0, tslot);              // P, dS computed
        // the previous step's products must be done with P / dS before they are overwritten (the last step of
        // the item before was waited for when its dQ was taken out)
        if (it > 0 && !mbar_wait(dq_full, (g - 1) & 1, abort_flag, status)) { ok = false; break; }
        // ... and the bulk stores of the item before with the dK / dV tiles staged in the P buffer
        if (it == 0 && w > 0 && !mbar_wait(dkv_stored, (w - 1) & 1, abort_flag, status)) { ok = false; break; }
#pragma unroll
        for (int cc = 0; cc < 2; ++cc) {
#pragma unroll
          for (int c = 0; c < 32; c += 8) {
            const int q = c >> 1;
            *reinterpret_cast<uint4*>(sds + p_offset(r, half * 64 + cc * 32 + c)) =
                make_uint4(pk_ds[cc][q], pk_ds[cc][q + 1], pk_ds[cc][q + 2], pk_ds[cc][q + 3]);
          }
        }
#pragma unroll
        for (int cc = 0; cc < 2; ++cc) {
#pragma unroll
          for (int c = 0; c < 32; c += 8) {
            const int q = c >> 1;
            *reinterpret_cast<uint4*>(sp + p_offset(r, half * 64 + cc * 32 + c)) =
                make_uint4(pk_p[cc][q], pk_p[cc][q + 1], pk_p[cc][q + 2], pk_p[cc][q + 3]);
          }
        }
        ATT_TRACE(tr, 0, tslot);              // P, dS written
        fence_proxy_async();
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(pds_full);
        // the next item's D, under the products of this one
        if (ONE && bh_after >= 0 && !dots_finish(g + 1)) { ok = false; break; }
        // the previous step's dQ leaves after the hand-over, off the critical path (the next dQ product
        // waits for its read-out)
        if (it > 0 && !drain_dq(g - 1)) { ok = false; break; }
      }
      // the last step's dQ; its barrier also says that every dV / dK product of the item is done
      if (!ok || !drain_dq(g - 1)) { ok = false; break; }
      // dV and dK rows of this kv tile (TMEM lane = kv row)
      uint32_t vk[32], vv[32];
      tmem_ld_32x32(tm_dk + lane_addr + half * 32, vk);
      tmem_ld_32x32(tm_dv + lane_addr + half * 32, vv);
      tmem_ld_wait();
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(dkv_free);          // the next item's first products may overwrite the sums
      if (colsum != nullptr) {          // rows past the sequence are zeros
        float* sums = reinterpret_cast<float*>(smem + L::SUM_OFF) + q4 * 128 + half * 32 + lane;
        sums[0] = column_sum(vk);
        sums[64] = column_sum(vv);
      }
      // staged as two 128-byte-swizzled [128 x 64] bf16 tiles (dK, dV) in the P buffer, which nothing reads any more; the
      // reducer warp stores them with one bulk copy each
#pragma unroll
      for (int which = 0; which < 2; ++which) {
        const uint32_t* v = which == 0 ? vk : vv;
#pragma unroll
        for (int c = 0; c < 4; ++c)
          *reinterpret_cast<uint4*>(sp + which * ATT_TILE_BYTES + r * 128 + (((half * 4 + c) ^ (r & 7)) << 4)) = make_uint4(
              pack_bf16(__uint_as_float(v[8 * c]), __uint_as_float(v[8 * c + 1])),
              pack_bf16(__uint_as_float(v[8 * c + 2]), __uint_as_float(v[8 * c + 3])),
              pack_bf16(__uint_as_float(v[8 * c + 4]), __uint_as_float(v[8 * c + 5])),
              pack_bf16(__uint_as_float(v[8 * c + 6]), __uint_as_float(v[8 * c + 7])));
      }
      fence_proxy_async();
      __syncwarp();
      if (lane == 0) mbar_arrive(dkv_staged);
      ++w;
    }
  }

  tc_fence_before();
  __syncthreads();
  if (warp == MMA_WARP) {
    tc_fence_after();
    tmem_dealloc(tmem_base, 512);
  }
}

}  // namespace dsw

using namespace dsw;

static long long* g_att_trace = nullptr;

static int att_num_sms() {
  static int n = 0;
  if (n == 0) {
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess ||
        n <= 0)
      n = 148;
  }
  return n;
}
// Which forward kernel a call takes; the bits are the same.  us a launch, tcgen05 / short (attention_short.cuh), n heads of all
// sequences together.  Heads of 64: T = 24, n 4 to 296 5.8-7.0 / 2.7-2.9, 3000 41.5 / 10.6; T = 64, 4 5.9 / 3.5, 3000 41.7 /
// 23.1; T = 96, 4 5.9 / 4.4, 296 7.7 / 5.5, 1000 18.4 / 17.3; T = 128, 4 6.1 / 5.1, 296 7.8 / 6.8, 400 11.2 / 11.8, 1000 19.5 /
// 21.8 (296: one wave of two blocks per SM).  Heads of 32 at T = 128: 4 6.0 / 4.2, 296 7.8 / 5.2, 1000 19.4 / 15.6.
static bool attention_is_short(int T, int hs, int n_bh) {
  if (T > SHORT_MAX_T) return false;
  return hs == 32 || T <= 64 || n_bh <= 2 * att_num_sms() || (T <= 96 && n_bh <= 6 * att_num_sms());
}
// Which kernel a backward takes, and on how many blocks and warps if it is the one for short sequences; the bits are the same.
// us a launch, tcgen05 / short, n heads of all sequences together.  Heads of 64: T = 16, n 60 7.8 / 3.7, 768 32.8 / 6.0; T = 64, 60 8.0 /
// 5.3, 192 13.4 / 9.2, 768 33.0 / 21.3; T = 96, 192 13.5 / 13.1, 768 33.3 / 38.6; T = 128, 60 8.5 / 7.6, 148 9.2 / 9.6.  Where the two are
// close the rest of a pass decides, with weight gradients on the SMs beside it: forward and backward of 12 blocks, 1 x 128 tokens
// 1193 / 1203, 4 x 100 1464 / 1486, 12 x 192 2780 / 2842 (kernel alone, its three kernels against one, 20.3 / 17.8), 64 x 50 3681 / 3560,
// 64 x 16 2320 / 1996.  Heads of 32, half the products: T = 128, n 4 8.0 / 4.8, 800 32.8 / 24.7; T = 192, 4 12.6 / 6.7, 800 74.6 / 48.3; three
// blocks, 1 x 160 257 / 235, 64 x 190 1071 / 1026, 8 x 256 432 / 445.
// A second block for a head where it finds an SM of its own: T = 128, n 4 5.4 -> 4.8.
static ShortBwdPlan attention_bwd_plan(int T, int hs, int n_bh) {
  const int sms = att_num_sms(), blocks = (T + 15) / 16;
  if (T > (hs == 32 ? SHORT_BWD_MAX_T : 64)) return {0, 0, false};
  if (T > 128) return n_bh <= sms ? ShortBwdPlan{2, blocks, true} : ShortBwdPlan{1, (blocks + 1) / 2, true};
  if (n_bh > sms) return {1, T <= 32 ? 2 * blocks : blocks, true};
  if (T <= 64) return {1, 2 * blocks, false};
  return {2 * n_bh <= sms ? 2 : 1, blocks, false};
}
// Register (or clear, with nullptr) a device buffer of 512 int64 for the in-kernel timeline.
extern "C" int dsw_attention_set_trace(long long* buf) { g_att_trace = buf; return 0; }

// qkv: bf16 [B*T, 3*nh*hs]; out: bf16 [B*T, nh*hs]; lse: fp32 [B*nh*T].
// Requires hs == 64 or 32; T is any length.
extern "C" int dsw_attention_fwd(const void* qkv, void* out, float* lse, int B, int T, int nh, int hs, float scale,
                                 int* status, cudaStream_t st) {
  if ((hs != 64 && hs != 32) || T <= 0) return -10;
  const int d = nh * hs;
  if (attention_is_short(T, hs, B * nh)) {
    if (reinterpret_cast<uintptr_t>(qkv) & 15) return -10;          // 16-byte copies; a tensor map refuses it as well
    const float s2 = scale * 1.4426950408889634f;
    return hs == 64 ? attention_short<64>((const __nv_bfloat16*)qkv, (__nv_bfloat16*)out, lse, T, nh, B * nh, s2, st)
                    : attention_short<32>((const __nv_bfloat16*)qkv, (__nv_bfloat16*)out, lse, T, nh, B * nh, s2, st);
  }
  CUtensorMap tm;
  const int rc = cached_tmap(&tm, TMAP_BF16_4D, qkv, hs, 3LL * nh, T, 3LL * d, 64, 128, B);
  if (rc) return rc;
  static bool attr_set = false;
  if (!attr_set) {
    if (cudaFuncSetAttribute(attention_fwd_kernel<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, AttSmem::TOTAL) != cudaSuccess ||
        cudaFuncSetAttribute(attention_fwd_kernel<false>, cudaFuncAttributeMaxDynamicSharedMemorySize, AttSmem::TOTAL) != cudaSuccess)
      return -2;
    attr_set = true;
  }
  // persistent: two CTAs per SM walk the work items
  const int total = ((T + ATT_BQ - 1) / ATT_BQ) * B * nh;
  const int G = total < 2 * att_num_sms() ? total : 2 * att_num_sms();
  return launch(total <= att_num_sms() ? attention_fwd_kernel<true> : attention_fwd_kernel<false>, G, ATT_THREADS, AttSmem::TOTAL, st, 1,
                tm, (__nv_bfloat16*)out, lse, T, nh, B * nh, hs, scale * 1.4426950408889634f, status, g_att_trace) == cudaSuccess ? 0 : -3;
}

// qkv, out, dout as in the forward; lse from the forward.  dqkv: bf16 [B*T, 3*d] (all of it is written).
// dq_acc: fp32 scratch [B*T, d]; Dvec: fp32 scratch [B*nh*T].  Both may be overwritten.
// ordered: the kv tiles' contributions to dQ, which otherwise meet in whatever order their CTAs get there, are added tile
// by tile, one launch each.
static int attention_bwd(const void* qkv, const void* out, const void* dout, const float* lse, void* dqkv, float* dq_acc, float* Dvec,
                         int B, int T, int nh, int hs, float scale, bool ordered, int* status, cudaStream_t st) {
  if ((hs != 64 && hs != 32) || T <= 0 || (long long)B * nh * T >= (1LL << 31)) return -10;
  const int d = nh * hs;
  const long long rows = (long long)B * T;
  if (const ShortBwdPlan plan = attention_bwd_plan(T, hs, B * nh); plan.warps) {
    // 16-byte copies, and what the tensor maps of the other kernel refuse
    if ((reinterpret_cast<uintptr_t>(qkv) | reinterpret_cast<uintptr_t>(out) | reinterpret_cast<uintptr_t>(dout) |
         reinterpret_cast<uintptr_t>(dqkv) | reinterpret_cast<uintptr_t>(dq_acc)) & 15)
      return -10;
    const ShortBwdArgs a = {(const __nv_bfloat16*)qkv, (const __nv_bfloat16*)out, (const __nv_bfloat16*)dout, lse, (__nv_bfloat16*)dqkv,
                            tl_launch.colsum, T, nh, scale};
    tl_launch.colsum = nullptr;
    return hs == 64 ? attention_short_bwd<64>(a, plan, B * nh, st) : attention_short_bwd<32>(a, plan, B * nh, st);
  }
  CUtensorMap tq, tdo, tdq, tdkv;
  int rc = cached_tmap(&tq, TMAP_BF16_4D, qkv, hs, 3LL * nh, T, 3LL * d, 64, 128, B);
  if (!rc) rc = cached_tmap(&tdkv, TMAP_BF16_4D, dqkv, hs, 3LL * nh, T, 3LL * d, 64, 128, B);
  if (!rc) rc = cached_tmap(&tdo, TMAP_BF16_4D, dout, hs, nh, T, d, 64, 128, B);
  if (!rc) rc = cached_tmap(&tdq, TMAP_F32_4D, dq_acc, hs, nh, T, d, 32, 128, B);
  if (rc) return rc;
  static bool attr_set = false;
  if (!attr_set) {
    if (cudaFuncSetAttribute(attention_bwd_kernel<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, AttBwdSmem::TOTAL) != cudaSuccess ||
        cudaFuncSetAttribute(attention_bwd_kernel<false>, cudaFuncAttributeMaxDynamicSharedMemorySize, AttBwdSmem::TOTAL) != cudaSuccess)
      return -2;
    attr_set = true;
  }
  // persistent: one CTA per SM walks the work items
  const int tiles = (T + ATT_BK - 1) / ATT_BK, n_bh = B * nh;
  const auto grid = [](int items) { return items < att_num_sms() ? items : att_num_sms(); };
  float* const colsum = reinterpret_cast<uintptr_t>(tl_launch.colsum) & 15 ? nullptr : tl_launch.colsum;          // for bulk reductions
  if (colsum != nullptr) tl_launch.colsum = nullptr;
  if (T <= ATT_BK)
    return launch(attention_bwd_kernel<true>, grid(n_bh), ATT_BWD_THREADS, AttBwdSmem::TOTAL, st, 1, tq, tdo, tdq, tdkv,
                  (const __nv_bfloat16*)out, (const __nv_bfloat16*)dout, lse, Dvec, T, nh, n_bh, hs, 0, n_bh, scale, colsum, status,
                  g_att_trace) == cudaSuccess ? 0 : -3;
  // D = rowsum(dO * O) per head, and the dQ accumulator zeroed in the same pass
  {
    const long long want = (rows * 32 + 255) / 256;
    const int cap = att_num_sms() * 16;
    if (launch(attention_bwd_prep_kernel, (unsigned)(want < cap ? want : cap), 256, 0, st, 1, (const __nv_bfloat16*)out,
               (const __nv_bfloat16*)dout, Dvec, dq_acc, B, T, nh, hs) != cudaSuccess)
      return -3;
  }
  const int per_launch = ordered ? n_bh : tiles * n_bh;
  for (int item0 = 0; item0 < tiles * n_bh; item0 += per_launch)
    if (launch(attention_bwd_kernel<false>, grid(per_launch), ATT_BWD_THREADS, AttBwdSmem::TOTAL, st, 1, tq, tdo, tdq, tdkv,
               (const __nv_bfloat16*)out, (const __nv_bfloat16*)dout, lse, Dvec, T, nh, n_bh, hs, item0, per_launch, scale, colsum, status,
               g_att_trace) != cudaSuccess)
      return -3;
  const int width = d / 8 < 512 ? d / 8 : 512, per_step = 512 / width;
  const long long steps = (rows + per_step - 1) / per_step;
  return launch(attention_dq_convert_kernel, dim3(unsigned(steps < 296 ? steps : 296), (d + 8 * width - 1) / (8 * width)), width * per_step,
                colsum ? sizeof(float) * per_step * width * 8 : 0, st, 1, dq_acc, (__nv_bfloat16*)dqkv, rows, d, width, colsum) == cudaSuccess
             ? 0
             : -3;
}

extern "C" int dsw_attention_bwd(const void* qkv, const void* out, const void* dout, const float* lse, void* dqkv,
                                 float* dq_acc, float* Dvec, int B, int T, int nh, int hs, float scale, int* status,
                                 cudaStream_t st) {
  return attention_bwd(qkv, out, dout, lse, dqkv, dq_acc, Dvec, B, T, nh, hs, scale, false, status, st);
}
extern "C" int dsw_attention_bwd_ordered(const void* qkv, const void* out, const void* dout, const float* lse, void* dqkv,
                                         float* dq_acc, float* Dvec, int B, int T, int nh, int hs, float scale, int* status,
                                         cudaStream_t st) {
  return attention_bwd(qkv, out, dout, lse, dqkv, dq_acc, Dvec, B, T, nh, hs, scale, true, status, st);
}

extern "C" int dsw_load_attention() {
  cudaFuncAttributes a;
  int bad = 0;
  bad |= cudaFuncGetAttributes(&a, attention_fwd_kernel<true>) != cudaSuccess;
  bad |= load_attention_short();
  bad |= load_attention_short_bwd();
  bad |= cudaFuncGetAttributes(&a, attention_fwd_kernel<false>) != cudaSuccess;
  bad |= cudaFuncGetAttributes(&a, attention_bwd_kernel<false>) != cudaSuccess;
  bad |= cudaFuncGetAttributes(&a, attention_bwd_kernel<true>) != cudaSuccess;
  bad |= cudaFuncGetAttributes(&a, attention_bwd_prep_kernel) != cudaSuccess;
  bad |= cudaFuncGetAttributes(&a, attention_dq_convert_kernel) != cudaSuccess;
  return bad ? -1 : 0;
}
