// Device side of the tcgen05 GEMMs: epilogue, the one-CTA kernel and the CTA-pair kernel, as templates.
// Each kernel is a template on its epilogue class; gemm_one_cta.cu and gemm_pair.cu instantiate them
// (two translation units, so the kernels compile side by side) and gemm_tcgen05.cu holds the
// host entry point.
#pragma once
#include <cuda.h>
#include "ptx.cuh"

namespace dsw {

__device__ __forceinline__ long long gemm_gtimer() {
  long long t;
  asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
  return t;
}
// In-kernel timeline stamps exist only in the tracing build of the library (-DDSWARM_TRACE, used by
// benchmarks/timelines.py); the shipped kernels carry none of it.
#ifdef DSWARM_TRACE
#define GEMM_TRACE(buf, slot) do { if ((buf) != nullptr && (slot) < 256) (buf)[(slot)++] = gemm_gtimer(); } while (0)
#define GEMM_TRACE2(buf, slot) do { if ((buf) != nullptr && (slot) < 255) (buf)[(slot)++] = gemm_gtimer(); } while (0)
#else
#define GEMM_TRACE(buf, slot) do { } while (0)
#define GEMM_TRACE2(buf, slot) do { } while (0)
#endif

constexpr int BM = 128;
constexpr int BK = 64;          // one 128-byte swizzle row of bf16
constexpr int UMMA_K = 16;
constexpr int EPI_WARPS = 16;         // four per TMEM lane quarter, each takes a quarter of the tile's columns
constexpr int EPI_WARP0 = 4;          // warps 2 and 3 only keep the epilogue warps aligned with the TMEM lane quarters
constexpr int GEMM_THREADS = 32 * (EPI_WARP0 + EPI_WARPS);

enum EpiMode : int {
  EPI_STORE = 0,        // out = acc (+ bias)
  EPI_GELU = 1,         // out = gelu(acc + bias) ; aux_out (optional) = gelu'(acc + bias), what the backward multiplies by
  EPI_RESID = 2,        // out = acc + bias + resid (+ aux_in); aux_out (optional) = what rounding out to bf16 left over
  EPI_MUL = 3,          // out = acc * aux_in  (aux_in = the gelu' saved by EPI_GELU: the GELU backward)
  EPI_ATOMIC_F32 = 4,   // out_f32 += acc   (split-K safe)
  EPI_STORE_F32 = 5,    // out_f32 = acc; split of K number s stores split_stride * s elements further on
  // LM head without stored logits (dsw_head_lse / dsw_head_dlogits); acc = the logits of row and column
  EPI_LSE = 6,          // parts[column / 64][row] = log2 of the sum of 2^(acc log2 e) over 64 columns; tlogit[row] = acc at the target
  EPI_DLOGITS = 7,      // out = coef (softmax(acc) - onehot), lse2, target and coef from rows[row]
  EPI_RESID_LO = 8,     // EPI_RESID with aux_in or aux_out, on the kernels for many rows
  // EPI_GELU without aux_out, on the kernels for many rows: evaluation and sampling drop the derivative, whose arithmetic
  // and registers the class with aux_out carries all the same (32768 x 3072 from 768, CTA pairs: 144.8 -> 136.7 us)
  EPI_GELU_ONLY = 9,
  EPI_MUL_SUM = 10,     // EPI_MUL with colsum, whose code and registers a product without it does not carry
};

// What the second pass over the logits needs to know of a row: {log2-sum-exp2, factor (0: the row is masked), target as
// int bits, unused}.
typedef float4 HeadRow;
constexpr int LSE_COLS = 64;            // columns per partial log-sum-exp: what one epilogue warp drains of a 256-wide tile

struct GemmArgs {
  int M, N, K;
  int a_mn_major, b_mn_major;
  int mode;
  int split_k;
  void* out; long long ldo;
  const float* bias;
  const __nv_bfloat16* resid; long long ldr;
  __nv_bfloat16* aux_out; const __nv_bfloat16* aux_in; long long ldaux;
  int* status;
  const long long* targets; float* parts; float* tlogit;      // EPI_LSE
  const HeadRow* rows;                                         // EPI_DLOGITS
  long long split_stride;                                      // EPI_STORE_F32
  int group;            // row tiles per group of the tile order
  int b_static;         // B is older than the kernel before in the stream (weights): it may be loaded before pdl_wait()
  float* colsum;        // optional, EPI_MUL: += sums of the output's columns
  long long* trace;     // optional: CTA 0's MMA thread stores %globaltimer stamps per k-block (tuning aid)
};

// ------------------------------------------------------------------ epilogue
// Sixteen warps drain a finished accumulator: four per TMEM lane quarter (a warp may only read the
// 32 lanes of its quarter), each taking a quarter of the tile's columns.  With four epilogue warps
// per scheduler the latencies of one warp's TMEM load, shared-memory round trip and global loads
// are covered by the others; with two they were not, and the epilogue of a K = 768 tile took longer
// than the tile's main loop.
//
// A thread owns one accumulator row (that is how tcgen05.ld hands the data out), but a store in
// which every lane writes 16 bytes of a different row touches 32 cache lines per instruction.  So
// each warp passes its rows through a private 2 KB tile of shared memory, 32 rows x 64 bytes with
// the 16-byte chunks rotated by (row / 2) so that writes by row and reads by row group are both
// conflict-free, and writes it out with lane = (row within a group of 8, 16-byte chunk): every
// store, residual / aux load or fp32 reduction instruction then covers 8 rows x 64 contiguous bytes.
//
// The accumulator is drained in chunks of 32 columns (16 for fp32 outputs: 64 bytes per row either
// way).  Everything a chunk needs from global memory besides the accumulator (residual, saved GELU
// derivative) is requested before the wait for the accumulator, in one batch; the TMEM load of the
// next chunk is issued as soon as this chunk's registers have been converted, so it runs under the
// staging and the stores.
constexpr int EPI_STAGE_BYTES = 32 * 64;

// This thread's row: NW 32-bit words = NW / 4 consecutive 16-byte chunks starting at chunk 0.
__device__ __forceinline__ void stage_row64(uint8_t* stage, int lane, const uint32_t (&w)[16]) {
#pragma unroll
  for (int c = 0; c < 4; ++c)
    *reinterpret_cast<uint4*>(stage + lane * 64 + (((c + (lane >> 1)) & 3) << 4)) =
        make_uint4(w[4 * c], w[4 * c + 1], w[4 * c + 2], w[4 * c + 3]);
}
// Write-out order: iteration i, this lane handles row i*8 + (lane >> 2), 16-byte chunk lane & 3.
template <class F>
__device__ __forceinline__ void unstage_rows64(const uint8_t* stage, int lane, F&& emit) {
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const int rl = i * 8 + (lane >> 2), ch = lane & 3;
    const uint4 d = *reinterpret_cast<const uint4*>(stage + rl * 64 + (((ch + (rl >> 1)) & 3) << 4));
    emit(i, rl, ch, d);
  }
}

// What an epilogue keeps of its row and tile; loads are asked for before the wait for the accumulator.
template <int MODE>
struct RowInfo {
  __device__ __forceinline__ void load(const GemmArgs&, int, int) {}
};
template <>
struct RowInfo<EPI_ATOMIC_F32> {
  float* out;
  __device__ __forceinline__ void load(const GemmArgs& g, int, int ks) { out = reinterpret_cast<float*>(g.out) + ks * g.split_stride; }
};
template <>
struct RowInfo<EPI_LSE> {
  int target;
  __device__ __forceinline__ void load(const GemmArgs& g, int row, int) {
    const long long t = row < g.M ? g.targets[row] : 0;
    target = t < 0 || t >= g.N ? 0 : int(t);          // reported by head_rows_kernel where the row counts
  }
};
template <>
struct RowInfo<EPI_DLOGITS> {
  float lse2, coef;
  int target;
  __device__ __forceinline__ void load(const GemmArgs& g, int row, int) {
    const HeadRow r = row < g.M ? g.rows[row] : make_float4(0.f, 0.f, 0.f, 0.f);
    lse2 = r.x; coef = r.y; target = __float_as_int(r.z);
  }
};
constexpr float LOG2E = 1.4426950408889634f;

// NCOLS accumulator columns (a multiple of 32) starting at TMEM address t_addr, rows row_base..+31
// (one per lane), output columns col_base..+NCOLS-1.  `release` is called once, right after the last
// TMEM load has landed, so the MMA thread can refill the accumulator while the last chunk is written.
template <int MODE, int NCOLS, class Release>
__device__ __forceinline__ void epilogue_warp(const GemmArgs& g, uint32_t t_addr, int row_base, int lane, int col_base,
                                              uint8_t* stage, const RowInfo<MODE>& info, Release&& release) {
  if constexpr (MODE == EPI_LSE) {
    // Thread = row: maximum and sum of 2^(x - maximum) over the warp's 64 columns, straight from the fp32 accumulators.
    // Per column one special-function operation and two packed halves; nothing but 4 bytes per 64 columns leaves the SM.
    static_assert(NCOLS == LSE_COLS, "one partial result per warp and tile");
    constexpr int NCH = NCOLS / 32;
    uint32_t r[32];
    tmem_ld_32x32(t_addr, r);
    float m = -INFINITY, s = 0.f;
#pragma unroll
    for (int c = 0; c < NCH; ++c) {
      const int cb = col_base + c * 32;
      tmem_ld_wait();
      float v[32];
#pragma unroll
      for (int i = 0; i < 32; ++i) v[i] = __uint_as_float(r[i]);
      if (c + 1 < NCH) tmem_ld_32x32(t_addr + (c + 1) * 32, r);
      else release();
      if (cb >= g.N) continue;
      if (cb + 32 > g.N) {
#pragma unroll
        for (int i = 0; i < 32; ++i) v[i] = cb + i < g.N ? v[i] : -INFINITY;
      }
      if (unsigned(info.target - cb) < 32u && row_base + lane < g.M) {
        float t = 0.f;
#pragma unroll
        for (int i = 0; i < 32; ++i) t = cb + i == info.target ? v[i] : t;
        g.tlogit[row_base + lane] = t;
      }
      float mx[4] = {v[0], v[1], v[2], v[3]};
#pragma unroll
      for (int i = 4; i < 32; ++i) mx[i & 3] = fmaxf(mx[i & 3], v[i]);
      const float nm = fmaxf(m, fmaxf(fmaxf(mx[0], mx[1]), fmaxf(mx[2], mx[3])) * LOG2E);
      const float ref = nm == -INFINITY ? 0.f : nm;          // nothing but -inf so far: a sum of zeros
      s *= ex2_approx(m - ref);
      m = nm;
      f2 acc[2] = {f2_bcast(0.f), f2_bcast(0.f)};
      const f2 l2 = f2_bcast(LOG2E), neg = f2_bcast(-ref);
#pragma unroll
      for (int i = 0; i < 32; i += 2) {
        float x0, x1;
        f2_split(f2_fma(f2_make(v[i], v[i + 1]), l2, neg), x0, x1);
        acc[(i >> 1) & 1] = f2_add(acc[(i >> 1) & 1], f2_make(ex2_approx(x0), ex2_approx(x1)));
      }
      float a0, a1;
      f2_split(f2_add(acc[0], acc[1]), a0, a1);
      s += a0 + a1;
    }
    if (col_base < g.N && row_base + lane < g.M)
      g.parts[(long long)(col_base / LSE_COLS) * g.M + row_base + lane] = (m == -INFINITY ? 0.f : m) + log2f(s);
    return;
  } else
  if constexpr (MODE == EPI_ATOMIC_F32) {     // both fp32 outputs: accumulate (split-K safe) or plain store
    constexpr int NCH = NCOLS / 16;
    uint32_t r[16];
    tmem_ld_32x16(t_addr, r);
#pragma unroll
    for (int c = 0; c < NCH; ++c) {
      const int cb = col_base + c * 16;
      tmem_ld_wait();
      uint32_t w[16];
#pragma unroll
      for (int i = 0; i < 16; ++i) w[i] = r[i];
      if (c + 1 < NCH) tmem_ld_32x16(t_addr + (c + 1) * 16, r);
      else release();
      if (cb >= g.N) continue;
      __syncwarp();                                   // the previous chunk has been read out
      stage_row64(stage, lane, w);
      __syncwarp();
      unstage_rows64(stage, lane, [&](int, int rl, int ch, const uint4& d) {
        const int row = row_base + rl, col = cb + ch * 4;
        if (row < g.M && col < g.N) {
          float* o = info.out + (long long)row * g.ldo + col;
          if (g.mode == EPI_ATOMIC_F32)
            asm volatile("red.global.add.v4.f32 [%0], {%1, %2, %3, %4};" ::"l"(o), "f"(__uint_as_float(d.x)),
                         "f"(__uint_as_float(d.y)), "f"(__uint_as_float(d.z)), "f"(__uint_as_float(d.w))
                         : "memory");
          else
            *reinterpret_cast<uint4*>(o) = d;
        }
      });
    }
  } else if constexpr (MODE == EPI_RESID_LO) {
    // Residual stream of two bf16 arrays.  The accumulator passes the staging tile as fp32, 16 rows at a time, so that the
    // sum is rounded once, at its end, and its remainder once more: staged as bf16 like the plain residual's it lost the
    // bits that the low half is there to keep (sampling 8 x 777 tokens of GPT-2 small: error of the logits 4.4e-3 ->
    // 3.6e-3; 16384 x 768 from 3072 72.2 -> 73.2 us, 6216 x 768 from 768 some 1 us more).  Loads and stores cover 8 rows
    // of 64 bytes, as below; 16-column slices, whose 16 rows of 32 bytes cost the load/store unit twice the lines, took
    // 76.  The low half is asked for when its rows are staged: sooner, its registers spilled.
    constexpr int NCH = NCOLS / 32;
    const int my_ch = lane & 3, my_r = lane >> 2;
    uint32_t r[32];
    tmem_ld_32x32(t_addr, r);
#pragma unroll
    for (int c = 0; c < NCH; ++c) {
      const int cb = col_base + c * 32, col = cb + my_ch * 8;
      uint4 x[4];
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const int row = row_base + i * 8 + my_r;
        const bool in = row < g.M && col < g.N;
        x[i] = in ? *reinterpret_cast<const uint4*>(g.resid + (long long)row * g.ldr + col) : make_uint4(0, 0, 0, 0);
      }
      tmem_ld_wait();
#pragma unroll
      for (int half = 0; half < 2; ++half) {          // rows half * 16 .. + 15 as [16][128 bytes], chunks of 16 swizzled by row
        uint4 t[2];
#pragma unroll
        for (int j = 0; j < 2; ++j) {
          const int row = row_base + half * 16 + j * 8 + my_r;
          t[j] = row < g.M && col < g.N && g.aux_in != nullptr ? *reinterpret_cast<const uint4*>(g.aux_in + (long long)row * g.ldaux + col)
                                                               : make_uint4(0, 0, 0, 0);
        }
        __syncwarp();                                 // the rows before have been read out
        if ((lane >> 4) == half) {
#pragma unroll
          for (int i = 0; i < 8; ++i) {
            const float4 bb = (g.bias != nullptr && cb + 4 * i < g.N) ? __ldg(reinterpret_cast<const float4*>(g.bias + cb) + i)
                                                                     : make_float4(0.f, 0.f, 0.f, 0.f);
            *reinterpret_cast<float4*>(stage + (lane & 15) * 128 + ((i ^ (lane & 7)) << 4)) =
                make_float4(__uint_as_float(r[4 * i]) + bb.x, __uint_as_float(r[4 * i + 1]) + bb.y,
                            __uint_as_float(r[4 * i + 2]) + bb.z, __uint_as_float(r[4 * i + 3]) + bb.w);
          }
        }
        __syncwarp();
        if (half == 1) {
          if (c + 1 < NCH) tmem_ld_32x32(t_addr + (c + 1) * 32, r);
          else release();
        }
#pragma unroll
        for (int j = 0; j < 2; ++j) {
          const int i = half * 2 + j, rl = j * 8 + my_r, row = row_base + half * 16 + rl;
          float a[8];
#pragma unroll
          for (int h = 0; h < 2; ++h) {
            const float4 f = *reinterpret_cast<const float4*>(stage + rl * 128 + (((my_ch * 2 + h) ^ (rl & 7)) << 4));
            a[4 * h] = f.x; a[4 * h + 1] = f.y; a[4 * h + 2] = f.z; a[4 * h + 3] = f.w;
          }
          if (row >= g.M || col >= g.N) continue;
          if (!DSW_OK(col + 8 <= g.N && col + 8 <= g.ldo && rl >= 0 && rl < 16)) continue;
          const uint32_t xu[4] = {x[i].x, x[i].y, x[i].z, x[i].w}, tu[4] = {t[j].x, t[j].y, t[j].z, t[j].w};
          uint32_t hi[4], lo[4];
#pragma unroll
          for (int q = 0; q < 4; ++q) {
            const float2 e = unpack_bf16(xu[q]), f = unpack_bf16(tu[q]);
            const float s0 = a[2 * q] + (e.x + f.x), s1 = a[2 * q + 1] + (e.y + f.y);
            hi[q] = pack_bf16(s0, s1);
            const float2 h = unpack_bf16(hi[q]);
            lo[q] = pack_bf16(s0 - h.x, s1 - h.y);
          }
          *reinterpret_cast<uint4*>(reinterpret_cast<__nv_bfloat16*>(g.out) + (long long)row * g.ldo + col) =
              make_uint4(hi[0], hi[1], hi[2], hi[3]);
          if (g.aux_out != nullptr)
            *reinterpret_cast<uint4*>(g.aux_out + (long long)row * g.ldaux + col) = make_uint4(lo[0], lo[1], lo[2], lo[3]);
        }
      }
    }
  } else {
    constexpr int NCH = NCOLS / 32;
    constexpr bool MUL = MODE == EPI_MUL || MODE == EPI_MUL_SUM;
    constexpr bool EXTRA = MODE == EPI_RESID || MUL;
    const int my_ch = lane & 3, my_r = lane >> 2;
    uint32_t r[32];
    tmem_ld_32x32(t_addr, r);
#pragma unroll
    for (int c = 0; c < NCH; ++c) {
      const int cb = col_base + c * 32;
      const bool chunk_ok = cb < g.N;
      // ---- requests to global memory for this chunk, all at once, ahead of the accumulator
      uint4 x[EXTRA ? 4 : 1];
      if constexpr (EXTRA) {
        const __nv_bfloat16* src = MODE == EPI_RESID ? g.resid : g.aux_in;
        const long long ld = MODE == EPI_RESID ? g.ldr : g.ldaux;
        const int col = cb + my_ch * 8;
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          const int row = row_base + i * 8 + my_r;
          x[i] = (row < g.M && col < g.N) ? *reinterpret_cast<const uint4*>(src + (long long)row * ld + col)
                                          : make_uint4(0, 0, 0, 0);
        }
      }
      tmem_ld_wait();
      // bias (an L1 hit after the first tile row), add, round.  GELU: activation and derivative come out of
      // one evaluation of the fp32 sum; the derivative waits in registers until the activation chunk is out
      uint32_t w[16];
      uint32_t post[MODE == EPI_GELU ? 16 : 1];
      if constexpr (MODE == EPI_DLOGITS) {
        if (chunk_ok) {
          const f2 l2 = f2_bcast(LOG2E), neg = f2_bcast(-info.lse2), k2 = f2_bcast(info.coef);
          auto pair = [&](int i) {
            float x0, x1;
            f2_split(f2_fma(f2_make(__uint_as_float(r[2 * i]), __uint_as_float(r[2 * i + 1])), l2, neg), x0, x1);
            return f2_mul(f2_make(ex2_approx(x0), ex2_approx(x1)), k2);
          };
#pragma unroll
          for (int i = 0; i < 16; ++i) w[i] = pack_bf16_f2(pair(i));
          if (unsigned(info.target - cb) < 32u) {            // one chunk of the row
#pragma unroll
            for (int i = 0; i < 16; ++i)
              if (cb + 2 * i == (info.target & ~1)) {
                float p0, p1;
                f2_split(pair(i), p0, p1);
                if (info.target & 1) p1 -= info.coef; else p0 -= info.coef;
                w[i] = pack_bf16(p0, p1);
              }
          }
          if (info.coef == 0.f) {                              // a masked row: zeros, whatever its logits are
#pragma unroll
            for (int i = 0; i < 16; ++i) w[i] = 0;
          }
        }
      } else if (chunk_ok) {
#pragma unroll
        for (int i = 0; i < 8; ++i) {
          const float4 bb = (g.bias != nullptr && cb + 4 * i < g.N) ? __ldg(reinterpret_cast<const float4*>(g.bias + cb) + i)
                                                                   : make_float4(0.f, 0.f, 0.f, 0.f);
          const float v0 = __uint_as_float(r[4 * i]) + bb.x, v1 = __uint_as_float(r[4 * i + 1]) + bb.y;
          const float v2 = __uint_as_float(r[4 * i + 2]) + bb.z, v3 = __uint_as_float(r[4 * i + 3]) + bb.w;
          if constexpr (MODE == EPI_GELU || MODE == EPI_GELU_ONLY) {
            f2 ga, da, gb, db;
            gelu_pair(v0, v1, ga, da);
            gelu_pair(v2, v3, gb, db);
            w[2 * i] = pack_bf16_f2(ga);
            w[2 * i + 1] = pack_bf16_f2(gb);
            if constexpr (MODE == EPI_GELU) {
              post[2 * i] = pack_bf16_f2(da);
              post[2 * i + 1] = pack_bf16_f2(db);
            }
          } else {
            w[2 * i] = pack_bf16(v0, v1);
            w[2 * i + 1] = pack_bf16(v2, v3);
          }
        }
      }
      if (c + 1 < NCH) tmem_ld_32x32(t_addr + (c + 1) * 32, r);
      else release();
      if (!chunk_ok) continue;
      __syncwarp();                                   // the previous chunk has been read out
      stage_row64(stage, lane, w);
      __syncwarp();
      // sums of the output's columns (EPI_MUL_SUM): of this lane's rows, then over the warp's 32
      float cs[MODE == EPI_MUL_SUM ? 8 : 1];
      if constexpr (MODE == EPI_MUL_SUM) {
#pragma unroll
        for (int e = 0; e < 8; ++e) cs[e] = 0.f;
      }
      unstage_rows64(stage, lane, [&](int i, int rl, int ch, uint4 d) {
        const int row = row_base + rl, col = cb + ch * 8;
        if (row >= g.M || col >= g.N) return;
        if (!DSW_OK(col + 8 <= g.N && col + 8 <= g.ldo && rl >= 0 && rl < 32)) return;
        if constexpr (EXTRA) {
          uint32_t du[4] = {d.x, d.y, d.z, d.w};
          const uint32_t xu[4] = {x[i].x, x[i].y, x[i].z, x[i].w};
          // Both operands are bf16 by now, so one packed bf16 instruction does what unpacking, an fp32 product or sum and
          // packing did in seven, with the same single rounding (a product of two bf16 values is exact in fp32).
          if constexpr (MUL) {
#pragma unroll
            for (int q = 0; q < 4; ++q) du[q] = mul_bf16x2(du[q], xu[q]);
            if constexpr (MODE == EPI_MUL_SUM) {
#pragma unroll
              for (int q = 0; q < 4; ++q) {
                const float2 e = unpack_bf16(du[q]);
                cs[2 * q] += e.x;
                cs[2 * q + 1] += e.y;
              }
            }
          } else {
#pragma unroll
            for (int q = 0; q < 4; ++q) du[q] = add_bf16x2(du[q], xu[q]);
          }
          d = make_uint4(du[0], du[1], du[2], du[3]);
        }
        *reinterpret_cast<uint4*>(reinterpret_cast<__nv_bfloat16*>(g.out) + (long long)row * g.ldo + col) = d;
      });
      if constexpr (MODE == EPI_MUL_SUM) {
        // In place of a pass that reads the output once more (32768 x 3072: 40 us); here 150 -> 168 us with K = 768.
        // Over the eight lanes that hold the same columns: a lane ends with column lane / 4 of its eight.
        const float sum = fold_sums(cs);
        const int col = cb + my_ch * 8 + (lane >> 2);
        if (col < g.N) atomicAdd(g.colsum + col, sum);
      }
      if constexpr (MODE == EPI_GELU) {
        // Always so in this class, and asked all the same: ptxas makes a slower epilogue of the code without the branch (2128 x 4096
        // from 1024: 26.4 us, with it 24.6; 1024 rows 18.4 and 17.5).
        if (g.aux_out != nullptr) {
          __syncwarp();
          stage_row64(stage, lane, post);
          __syncwarp();
          unstage_rows64(stage, lane, [&](int, int rl, int ch, const uint4& d) {
            const int row = row_base + rl, col = cb + ch * 8;
            if (row < g.M && col < g.N) *reinterpret_cast<uint4*>(g.aux_out + (long long)row * g.ldaux + col) = d;
          });
        }
      }
    }
  }
}

// The residual / saved-derivative operand of a tile, asked into L2 one tile ahead: the epilogue's loads of it
// then cost an L2 round trip instead of a DRAM one, which otherwise sits exposed once per chunk.
// Same lane-to-address map as the loads in epilogue_warp; one request per 32-byte sector.
template <int MODE, int NCOLS>
__device__ __forceinline__ void prefetch_extra(const GemmArgs& g, int row_base, int lane, int col_base) {
  if constexpr (MODE == EPI_RESID || MODE == EPI_RESID_LO || MODE == EPI_MUL || MODE == EPI_MUL_SUM) {
    constexpr bool MUL = MODE == EPI_MUL || MODE == EPI_MUL_SUM;
    const __nv_bfloat16* src = MUL ? g.aux_in : g.resid;
    const long long ld = MUL ? g.ldaux : g.ldr;
    if (lane & 1) return;
#pragma unroll
    for (int c = 0; c < NCOLS / 32; ++c) {
      const int col = col_base + c * 32 + (lane & 3) * 8;
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const int row = row_base + i * 8 + (lane >> 2);
        if (row < g.M && col < g.N) {
          asm volatile("prefetch.global.L2 [%0];" ::"l"(src + (long long)row * ld + col));
          if (MODE == EPI_RESID_LO && g.aux_in != nullptr)
            asm volatile("prefetch.global.L2 [%0];" ::"l"(g.aux_in + (long long)row * g.ldaux + col));
        }
      }
    }
  }
}

// One tile's worth of epilogue for this warp.  MODE is the kernel's compile-time epilogue class: a kernel
// that switched on the mode at run time carried the registers of every epilogue at once and spilled.
template <int MODE, int NCOLS, class Release>
__device__ __forceinline__ void drain_tile(const GemmArgs& g, uint32_t t_addr, int row_base, int lane, int col_base,
                                           bool has_k, uint8_t* stage, const RowInfo<MODE>& info, Release&& release) {
  if (!has_k) { release(); return; }
  epilogue_warp<MODE, NCOLS>(g, t_addr, row_base, lane, col_base, stage, info, release);
}

// Tile `rem` of a slice of K: groups of g.group row tiles, all column tiles of a group before the next group.
__device__ __forceinline__ void tile_at(const GemmArgs& g, int rem, int tiles_m, int tiles_n, int& mt, int& nt) {
  const int per = g.group * tiles_n, grp = rem / per, r = rem - grp * per;
  const int first = grp * g.group, rows = min(g.group, tiles_m - first);
  nt = r / rows;
  mt = first + r - nt * rows;
}

template <int BN, int NSTAGE>
struct SmemLayout {
  static constexpr int A_BYTES = BM * BK * 2;
  static constexpr int B_BYTES = BN * BK * 2;
  static constexpr int STAGE_BYTES = A_BYTES + B_BYTES;
  static constexpr int EPI_OFFSET = NSTAGE * STAGE_BYTES;              // per-warp epilogue staging tiles
  static constexpr int BAR_OFFSET = EPI_OFFSET + EPI_WARPS * EPI_STAGE_BYTES;
  static constexpr int TOTAL = BAR_OFFSET + 256 + 1024;   // barriers + alignment slack
};

template <int BN, int NSTAGE, int MODE>
__global__ void __launch_bounds__(GEMM_THREADS, 1)
gemm_kernel(const __grid_constant__ CUtensorMap tmap_a, const __grid_constant__ CUtensorMap tmap_b, GemmArgs g) {
  using L = SmemLayout<BN, NSTAGE>;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint64_t* full_bar = reinterpret_cast<uint64_t*>(smem + L::BAR_OFFSET);
  uint64_t* empty_bar = full_bar + NSTAGE;
  uint64_t* acc_full = empty_bar + NSTAGE;      // [2]
  uint64_t* acc_empty = acc_full + 2;           // [2]
  uint32_t* tmem_holder = reinterpret_cast<uint32_t*>(acc_empty + 2);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_holder + 1);

  const int warp = threadIdx.x >> 5;
  const int lane = threadIdx.x & 31;

  const int tiles_m = (g.M + BM - 1) / BM;
  const int tiles_n = (g.N + BN - 1) / BN;
  const int kb_total = (g.K + BK - 1) / BK;
  const int splits = g.split_k > 1 ? g.split_k : 1;
  const int kb_per_split = (kb_total + splits - 1) / splits;
  const int num_tiles = tiles_m * tiles_n * splits;

  if (threadIdx.x == 0) {
    for (int s = 0; s < NSTAGE; ++s) { mbar_init(&full_bar[s], 1); mbar_init(&empty_bar[s], 1); }
    for (int b = 0; b < 2; ++b) { mbar_init(&acc_full[b], 1); mbar_init(&acc_empty[b], EPI_WARPS); }
    *abort_flag = 0;
    mbar_fence_init();
    fence_proxy_async();
  }
  if (warp == 1) {
    tmem_alloc(tmem_holder, 2 * BN);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_holder;

  if (warp == 0) {
    // ------------------------------------------------------------ producer (the whole warp, one lane issues)
    if (elect_one()) {
      tma_prefetch_desc(&tmap_a);
      tma_prefetch_desc(&tmap_b);
    }
    pdl_wait();
    uint32_t it = 0;
    bool ok = true;
    for (int tile = blockIdx.x; tile < num_tiles && ok; tile += gridDim.x) {
      const int ks = tile / (tiles_m * tiles_n);
      const int rem = tile - ks * tiles_m * tiles_n;
      int mt, nt;
      tile_at(g, rem, tiles_m, tiles_n, mt, nt);
      const int m0 = mt * BM, n0 = nt * BN;
      const int kb0 = ks * kb_per_split;
      const int kb1 = min(kb_total, kb0 + kb_per_split);
      for (int kb = kb0; kb < kb1; ++kb, ++it) {
        const int s = it % NSTAGE;
        const uint32_t ph = (it / NSTAGE) & 1;
        if (!mbar_wait_warp(&empty_bar[s], ph ^ 1, abort_flag, g.status)) { ok = false; break; }
        uint8_t* sa = smem + s * L::STAGE_BYTES;
        uint8_t* sb = sa + L::A_BYTES;
        const int k0 = kb * BK;
        if (elect_one()) {
          mbar_expect_tx(&full_bar[s], L::STAGE_BYTES);
          if (!g.a_mn_major) {
            tma_load_2d(sa, &tmap_a, &full_bar[s], k0, m0);
          } else {
#pragma unroll
            for (int c = 0; c < BM / 64; ++c) tma_load_2d(sa + c * 8192, &tmap_a, &full_bar[s], m0 + 64 * c, k0);
          }
          if (!g.b_mn_major) {
            tma_load_2d(sb, &tmap_b, &full_bar[s], k0, n0);
          } else {
#pragma unroll
            for (int c = 0; c < BN / 64; ++c) tma_load_2d(sb + c * 8192, &tmap_b, &full_bar[s], n0 + 64 * c, k0);
          }
        }
        __syncwarp();
      }
    }
    pdl_launch();
    if (!ok) {
      // give loads that are still in flight a bounded chance to land before the CTA exits
      for (int s = 0; s < NSTAGE; ++s) {
        for (int spin = 0; spin < 100000; ++spin)
          if (mbar_try_wait(&full_bar[s], 0) || mbar_try_wait(&full_bar[s], 1)) break;
      }
    }
  } else if (warp == 1) {
    // ------------------------------------------------------------ MMA issuer (the whole warp, one lane issues)
    const uint32_t idesc = make_idesc_bf16(BM, BN, g.a_mn_major, g.b_mn_major);
    const uint32_t desc_hi = smem_desc_hi(1024);
    const uint32_t a_lbo = g.a_mn_major ? 8192 : 16, b_lbo = g.b_mn_major ? 8192 : 16;
    const uint32_t a_step = g.a_mn_major ? (2048 >> 4) : (32 >> 4), b_step = g.b_mn_major ? (2048 >> 4) : (32 >> 4);
    uint32_t it = 0;
    uint32_t tcount = 0;
    bool ok = true;
    long long* tr = blockIdx.x == 0 && lane == 0 ? g.trace : nullptr;
    int tslot = 0;
    (void)tr; (void)tslot;
    for (int tile = blockIdx.x; tile < num_tiles && ok; tile += gridDim.x, ++tcount) {
      const int ks = tile / (tiles_m * tiles_n);
      const int kb0 = ks * kb_per_split;
      const int kb1 = min(kb_total, kb0 + kb_per_split);
      const int ab = tcount & 1;
      const uint32_t aph = (tcount >> 1) & 1;
      if (!mbar_wait_warp(&acc_empty[ab], aph ^ 1, abort_flag, g.status)) { ok = false; break; }
      tc_fence_after();
      const uint32_t d_tmem = tmem_base + ab * BN;
      for (int kb = kb0; kb < kb1; ++kb, ++it) {
        const int s = it % NSTAGE;
        const uint32_t ph = (it / NSTAGE) & 1;
        GEMM_TRACE(tr, tslot);
        if (!mbar_wait_warp(&full_bar[s], ph, abort_flag, g.status)) { ok = false; break; }
        GEMM_TRACE(tr, tslot);
        // no tcgen05 fence here: the operands were written by TMA (async proxy) and the mbarrier
        // wait orders them; a fence per k-block only delays the next MMAs behind the previous ones
        const uint32_t sa = smem_u32(smem + s * L::STAGE_BYTES);
        const uint32_t sb = sa + L::A_BYTES;
        // K-major: 16 elements = 32 bytes further along the swizzled row per MMA.
        // MN-major: 16 k-rows of 128 bytes further down.  Only the low descriptor word moves.
        const uint32_t a_lo = smem_desc_lo(sa, a_lbo), b_lo = smem_desc_lo(sb, b_lbo);
        if (elect_one()) {
#pragma unroll
          for (int k = 0; k < BK / UMMA_K; ++k)
            umma_bf16_lohi(d_tmem, a_lo + k * a_step, b_lo + k * b_step, desc_hi, idesc, kb > kb0 || k > 0);
          umma_commit(&empty_bar[s]);      // frees the smem stage when these MMAs retire
        }
        __syncwarp();
        GEMM_TRACE(tr, tslot);
        GEMM_TRACE(tr, tslot);
      }
      if (ok && elect_one()) umma_commit(&acc_full[ab]);  // accumulator complete
      __syncwarp();
    }
  } else if (warp >= EPI_WARP0) {
    // ------------------------------------------------------------ epilogue
    const int q = warp & 3;                 // TMEM lane quarter this warp may read
    const int part = (warp - EPI_WARP0) >> 2;   // which quarter of the tile's columns
    uint32_t tcount = 0;
    bool ok = true;
    auto prefetch_tile = [&](int tile) {
      if (tile >= num_tiles) return;
      const int rem = tile % (tiles_m * tiles_n);
      int mt, nt;
      tile_at(g, rem, tiles_m, tiles_n, mt, nt);
      prefetch_extra<MODE, BN / 4>(g, mt * BM + q * 32, lane, nt * BN + part * (BN / 4));
    };
    pdl_wait();
    prefetch_tile(blockIdx.x);
    for (int tile = blockIdx.x; tile < num_tiles && ok; tile += gridDim.x, ++tcount) {
      const int ks = tile / (tiles_m * tiles_n);
      const int rem = tile - ks * tiles_m * tiles_n;
      int mt, nt;
      tile_at(g, rem, tiles_m, tiles_n, mt, nt);
      const int m0 = mt * BM, n0 = nt * BN;
      const int ab = tcount & 1;
      const uint32_t aph = (tcount >> 1) & 1;
      const bool has_k = ks * kb_per_split < kb_total;
      prefetch_tile(tile + gridDim.x);
      RowInfo<MODE> info;
      info.load(g, m0 + q * 32 + lane, ks);
      if (!mbar_wait(&acc_full[ab], aph, abort_flag, g.status)) { ok = false; break; }
      tc_fence_after();
      const uint32_t t_addr = tmem_base + ab * BN + part * (BN / 4) + (uint32_t(q * 32) << 16);
      drain_tile<MODE, BN / 4>(g, t_addr, m0 + q * 32, lane, n0 + part * (BN / 4), has_k,
                         smem + L::EPI_OFFSET + (warp - EPI_WARP0) * EPI_STAGE_BYTES, info, [&] {
        tmem_ld_wait();
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(&acc_empty[ab]);
      });
    }
  }

  // ---------------------------------------------------------------- teardown
  tc_fence_before();
  __syncthreads();
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc(tmem_base, 2 * BN);
  }
}

// ------------------------------------------------------------------ CTA-pair variant
// 256 x BN output tile per cluster of two CTAs (tcgen05 cta_group::2).  Each CTA
// loads only its half of A (128 rows) and its half of B (128 columns) per k-block,
// 32 KB instead of the 48 KB a lone 128 x 256 CTA needs for the same FLOPs, which is
// what matters once the main loop is bound by L2-to-shared-memory traffic.  The
// leader CTA (cluster rank 0) issues the MMAs for both; each CTA drains its own
// 128 rows of the accumulator from its own TMEM.
//   full[s]      in the leader, 2 arrivals (one producer per CTA) + both CTAs' bytes
//   empty[s]     in each CTA, released by one multicast tcgen05.commit of the leader
//   acc_full[b]  in each CTA, same mechanism
//   acc_empty[b] in the leader, one arrival per epilogue warp of both CTAs
// KSUB k-blocks share one full/empty barrier pair (KSUB = 2: a stage is two 64-wide k-blocks, so the issuing
// thread pays one barrier wait and one commit per eight MMAs instead of per four).
// BN = 128 (64 columns of B per CTA) serves outputs too narrow, or with too few tiles, for 256: an SM takes in 24 KB per
// 128 x 128 x 64 products instead of the 32 KB of a lone 128 x 128 CTA, and that intake (some 120 bytes per ns) is what
// bounds a tile this small.
template <int BN>
struct PairSmem {
  static constexpr int STAGES = BN == 256 ? 6 : 8;      // k-blocks resident in shared memory
  static constexpr int A_BYTES = 128 * BK * 2;
  static constexpr int B_BYTES = BN / 2 * BK * 2;
  static constexpr int STAGE_BYTES = A_BYTES + B_BYTES;
  static constexpr int EPI_OFFSET = STAGES * STAGE_BYTES;
  static constexpr int BAR_OFFSET = EPI_OFFSET + EPI_WARPS * EPI_STAGE_BYTES;
  static constexpr int TOTAL = BAR_OFFSET + 256 + 1024;
};

constexpr int PAIR_KSUB = 2;           // k-blocks per barrier pair

template <int BN, int MODE>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(GEMM_THREADS, 1)
gemm_pair_kernel(const __grid_constant__ CUtensorMap tmap_a, const __grid_constant__ CUtensorMap tmap_b, GemmArgs g) {
  using L = PairSmem<BN>;
  constexpr int KSUB = PAIR_KSUB;
  constexpr int NSTAGE = L::STAGES / KSUB;            // barrier pairs; each covers KSUB k-blocks
  static_assert(L::STAGES % KSUB == 0, "stages must divide into groups");
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint64_t* full_bar = reinterpret_cast<uint64_t*>(smem + L::BAR_OFFSET);
  uint64_t* empty_bar = full_bar + NSTAGE;
  uint64_t* acc_full = empty_bar + NSTAGE;
  uint64_t* acc_empty = acc_full + 2;
  uint32_t* tmem_holder = reinterpret_cast<uint32_t*>(acc_empty + 2);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_holder + 1);

  const int warp = threadIdx.x >> 5;
  const int lane = threadIdx.x & 31;
  const uint32_t rank = cluster_ctarank();          // 0 = leader
  const int pair = blockIdx.x >> 1;
  const int num_pairs = gridDim.x >> 1;

  const int tiles_m = (g.M + 255) / 256;
  const int tiles_n = (g.N + BN - 1) / BN;
  const int kb_total = (g.K + BK - 1) / BK;
  const int splits = g.split_k > 1 ? g.split_k : 1;
  const int kb_per_split = (kb_total + splits - 1) / splits;
  const int num_tiles = tiles_m * tiles_n * splits;

  if (threadIdx.x == 0) {
    for (int s = 0; s < NSTAGE; ++s) { mbar_init(&full_bar[s], 2); mbar_init(&empty_bar[s], 1); }
    for (int b = 0; b < 2; ++b) { mbar_init(&acc_full[b], 1); mbar_init(&acc_empty[b], 2 * EPI_WARPS); }
    *abort_flag = 0;
    mbar_fence_init();
    fence_proxy_async();
  }
  if (warp == 1) {
    tmem_alloc_pair(tmem_holder, 2 * BN);
    tmem_relinquish_pair();
  }
  tc_fence_before();
  __syncthreads();
  cluster_sync_all();                 // both CTAs' barriers exist before anyone arrives remotely
  tc_fence_after();
  const uint32_t tmem_base = *tmem_holder;

  if (warp == 0) {
    // ------------------------------------------------------------ producer (one warp per CTA, one lane issues)
    if (elect_one()) {
      tma_prefetch_desc(&tmap_a);
      tma_prefetch_desc(&tmap_b);
    }
    pdl_wait();
    uint32_t it = 0;
    bool ok = true;
    for (int tile = pair; tile < num_tiles && ok; tile += num_pairs) {
      const int ks = tile / (tiles_m * tiles_n);
      const int rem = tile - ks * tiles_m * tiles_n;
      int mt, nt;
      tile_at(g, rem, tiles_m, tiles_n, mt, nt);
      const int m0 = mt * 256 + int(rank) * 128;         // this CTA's rows of A
      const int n0 = nt * BN + int(rank) * (BN / 2);     // this CTA's columns of B
      const int kb0 = ks * kb_per_split;
      const int kb1 = min(kb_total, kb0 + kb_per_split);
      for (int kb = kb0; kb < kb1; kb += KSUB, ++it) {
        const int s = it % NSTAGE;
        const uint32_t ph = (it / NSTAGE) & 1;
        const int nsub = min(KSUB, kb1 - kb);
        if (!mbar_wait_warp(&empty_bar[s], ph ^ 1, abort_flag, g.status)) { ok = false; break; }
        const uint32_t full_leader = map_to_cta(smem_u32(&full_bar[s]), 0);
        if (elect_one()) {
          mbar_expect_tx_cluster(full_leader, nsub * L::STAGE_BYTES);
#pragma unroll
          for (int sub = 0; sub < KSUB; ++sub) {
            if (sub >= nsub) break;
            uint8_t* sa = smem + (s * KSUB + sub) * L::STAGE_BYTES;
            uint8_t* sb = sa + L::A_BYTES;
            const int k0 = (kb + sub) * BK;
            if (!g.a_mn_major) {
              tma_load_2d_pair(sa, &tmap_a, full_leader, k0, m0);
            } else {
              tma_load_2d_pair(sa, &tmap_a, full_leader, m0, k0);
              tma_load_2d_pair(sa + 8192, &tmap_a, full_leader, m0 + 64, k0);
            }
            if (!g.b_mn_major) {
              tma_load_2d_pair(sb, &tmap_b, full_leader, k0, n0);
            } else {
              tma_load_2d_pair(sb, &tmap_b, full_leader, n0, k0);
              if constexpr (BN == 256) tma_load_2d_pair(sb + 8192, &tmap_b, full_leader, n0 + 64, k0);
            }
          }
        }
        __syncwarp();
      }
    }
    pdl_launch();
  } else if (warp == 1) {
    // ------------------------------------------------------------ MMA issuer (leader CTA only; the whole warp, one lane issues)
    if (rank == 0) {
      const uint32_t idesc = make_idesc_bf16(256, BN, g.a_mn_major, g.b_mn_major);
      const uint32_t desc_hi = smem_desc_hi(1024);
      const uint32_t a_lbo = g.a_mn_major ? 8192 : 16, b_lbo = g.b_mn_major ? 8192 : 16;
      const uint32_t a_step = g.a_mn_major ? (2048 >> 4) : (32 >> 4), b_step = g.b_mn_major ? (2048 >> 4) : (32 >> 4);
      uint32_t it = 0;
      uint32_t tcount = 0;
      bool ok = true;
      long long* tr = blockIdx.x == 0 && lane == 0 ? g.trace : nullptr;
      int tslot = 0;
      (void)tr; (void)tslot;
      for (int tile = pair; tile < num_tiles && ok; tile += num_pairs, ++tcount) {
        const int ks = tile / (tiles_m * tiles_n);
        const int kb0 = ks * kb_per_split;
        const int kb1 = min(kb_total, kb0 + kb_per_split);
        const int ab = tcount & 1;
        const uint32_t aph = (tcount >> 1) & 1;
        if (!mbar_wait_warp(&acc_empty[ab], aph ^ 1, abort_flag, g.status)) { ok = false; break; }
        tc_fence_after();
        const uint32_t d_tmem = tmem_base + ab * BN;
        for (int kb = kb0; kb < kb1; kb += KSUB, ++it) {
          const int s = it % NSTAGE;
          const uint32_t ph = (it / NSTAGE) & 1;
          const int nsub = min(KSUB, kb1 - kb);
          GEMM_TRACE(tr, tslot);
          if (!mbar_wait_warp(&full_bar[s], ph, abort_flag, g.status)) { ok = false; break; }
          GEMM_TRACE(tr, tslot);
          // no tcgen05 fence here: the operands were written by TMA (async proxy) and the mbarrier
          // wait orders them; a fence per k-block only delays the next MMAs behind the previous ones
          const uint32_t sa = smem_u32(smem + s * KSUB * L::STAGE_BYTES);
          const uint32_t a_lo = smem_desc_lo(sa, a_lbo), b_lo = smem_desc_lo(sa + L::A_BYTES, b_lbo);
          if (elect_one()) {
#pragma unroll
            for (int sub = 0; sub < KSUB; ++sub) {
              if (sub >= nsub) break;
              constexpr uint32_t SUB16 = L::STAGE_BYTES >> 4;
#pragma unroll
              for (int k = 0; k < BK / UMMA_K; ++k)
                umma_bf16_pair_lohi(d_tmem, a_lo + sub * SUB16 + k * a_step, b_lo + sub * SUB16 + k * b_step, desc_hi, idesc,
                                    kb > kb0 || sub > 0 || k > 0);
            }
            umma_commit_pair_all(smem_u32(&empty_bar[s]), 0x3);     // frees the stage in both CTAs
          }
          __syncwarp();
          GEMM_TRACE(tr, tslot);
          GEMM_TRACE(tr, tslot);
        }
        if (ok && elect_one()) umma_commit_pair_all(smem_u32(&acc_full[ab]), 0x3);
        __syncwarp();
      }
    }
  } else if (warp >= EPI_WARP0) {
    // ------------------------------------------------------------ epilogue (both CTAs, own 128 rows)
    const int q = warp & 3;
    const int part = (warp - EPI_WARP0) >> 2;
    uint32_t tcount = 0;
    bool ok = true;
    // tracing build: the first epilogue warp of CTA 0 stamps (waiting for the accumulator, got it, tile
    // written out) into the second half of the buffer
    long long* etr = (blockIdx.x == 0 && warp == EPI_WARP0 && lane == 0 && g.trace != nullptr) ? g.trace + 256 : nullptr;
    int eslot = 0;
    (void)etr; (void)eslot;
    auto prefetch_tile = [&](int tile) {
      if (tile >= num_tiles) return;
      const int rem = tile % (tiles_m * tiles_n);
      int mt, nt;
      tile_at(g, rem, tiles_m, tiles_n, mt, nt);
      prefetch_extra<MODE, BN / 4>(g, mt * 256 + int(rank) * 128 + q * 32, lane, nt * BN + part * (BN / 4));
    };
    pdl_wait();
    prefetch_tile(pair);
    for (int tile = pair; tile < num_tiles && ok; tile += num_pairs, ++tcount) {
      const int ks = tile / (tiles_m * tiles_n);
      const int rem = tile - ks * tiles_m * tiles_n;
      int mt, nt;
      tile_at(g, rem, tiles_m, tiles_n, mt, nt);
      const int m0 = mt * 256 + int(rank) * 128, n0 = nt * BN;
      const int ab = tcount & 1;
      const uint32_t aph = (tcount >> 1) & 1;
      const bool has_k = ks * kb_per_split < kb_total;
      prefetch_tile(tile + num_pairs);
      RowInfo<MODE> info;
      info.load(g, m0 + q * 32 + lane, ks);
      GEMM_TRACE2(etr, eslot);
      if (!mbar_wait(&acc_full[ab], aph, abort_flag, g.status)) { ok = false; break; }
      GEMM_TRACE2(etr, eslot);
      tc_fence_after();
      const uint32_t t_addr = tmem_base + ab * BN + part * (BN / 4) + (uint32_t(q * 32) << 16);
      drain_tile<MODE, BN / 4>(g, t_addr, m0 + q * 32, lane, n0 + part * (BN / 4), has_k,
                         smem + L::EPI_OFFSET + (warp - EPI_WARP0) * EPI_STAGE_BYTES, info, [&] {
        tmem_ld_wait();
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive_cluster(map_to_cta(smem_u32(&acc_empty[ab]), 0));
      });
      GEMM_TRACE2(etr, eslot);
    }
  }

  // ---------------------------------------------------------------- teardown
  tc_fence_before();
  __syncthreads();
  cluster_sync_all();                 // the peer may still be arriving on this CTA's barriers until here
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc_pair(tmem_base, 2 * BN);
  }
}


// Epilogue classes the kernels are instantiated for; both fp32 outputs share one.
inline int epi_class(const GemmArgs& g) {
  if (g.mode == EPI_STORE_F32) return EPI_ATOMIC_F32;
  if (g.mode == EPI_GELU && g.aux_out == nullptr) return EPI_GELU_ONLY;
  if (g.mode == EPI_MUL && g.colsum != nullptr) return EPI_MUL_SUM;
  return g.mode == EPI_RESID && (g.aux_in != nullptr || g.aux_out != nullptr) ? EPI_RESID_LO : g.mode;
}

// Defined in gemm_one_cta.cu / gemm_pair.cu.  bn = 128 or 256 for the one-CTA kernel.
int launch_one_cta(int bn, const CUtensorMap& ta, const CUtensorMap& tb, const GemmArgs& g, int num_sms, int max_ctas,
                   cudaStream_t st);
// bn = 256 or 128
int launch_pair(int bn, const CUtensorMap& ta, const CUtensorMap& tb, const GemmArgs& g, int num_sms, int max_ctas,
                cudaStream_t st);
int load_one_cta_kernels();
int load_pair_kernels();

}  // namespace dsw
