// Instantiations and launcher of the split-K cluster GEMM kernel for few rows (gemm_split.cuh).
#include "gemm_narrow.cuh"
#include "dswarm.h"
#include "launch.h"

namespace dsw {

namespace {
constexpr int kMaxDevices = 64;

template <int BN, int MODE>
int launch_one(const CUtensorMap& ta, const CUtensorMap& tb, const GemmArgs& g, cudaStream_t st) {
  using L = SplitSmem<BN>;
  static bool attr_set[kMaxDevices] = {false};          // the attribute is per device
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= kMaxDevices) return -2;
  if (!attr_set[dev]) {
    if (cudaFuncSetAttribute(gemm_split_kernel<BN, MODE>, cudaFuncAttributeMaxDynamicSharedMemorySize, L::TOTAL) != cudaSuccess)
      return -2;
    attr_set[dev] = true;
  }
  const int tiles = ((g.M + BM - 1) / BM) * ((g.N + BN - 1) / BN);
  return launch(gemm_split_kernel<BN, MODE>, tiles * g.split_k, SPLIT_THREADS, L::TOTAL, st, g.split_k, ta, tb, g) ==
                 cudaSuccess
             ? 0
             : -3;
}

template <int BN>
int launch_bn(const CUtensorMap& ta, const CUtensorMap& tb, const GemmArgs& g, cudaStream_t st) {
  switch (g.mode) {
    case EPI_STORE: return launch_one<BN, EPI_STORE>(ta, tb, g, st);
    case EPI_GELU: return launch_one<BN, EPI_GELU>(ta, tb, g, st);
    case EPI_RESID: return launch_one<BN, EPI_RESID>(ta, tb, g, st);
    case EPI_MUL: return g.colsum ? launch_one<BN, EPI_MUL_SUM>(ta, tb, g, st) : launch_one<BN, EPI_MUL>(ta, tb, g, st);
    default: return -13;
  }
}

template <int BN>
int load_bn() {
  cudaFuncAttributes a;
  int bad = 0;
  bad |= cudaFuncGetAttributes(&a, gemm_split_kernel<BN, EPI_STORE>) != cudaSuccess;
  bad |= cudaFuncGetAttributes(&a, gemm_split_kernel<BN, EPI_GELU>) != cudaSuccess;
  bad |= cudaFuncGetAttributes(&a, gemm_split_kernel<BN, EPI_RESID>) != cudaSuccess;
  bad |= cudaFuncGetAttributes(&a, gemm_split_kernel<BN, EPI_MUL>) != cudaSuccess;
  bad |= cudaFuncGetAttributes(&a, gemm_split_kernel<BN, EPI_MUL_SUM>) != cudaSuccess;
  return bad;
}
}  // namespace

int launch_split(int bn, const CUtensorMap& ta, const CUtensorMap& tb, const GemmArgs& g, cudaStream_t st) {
  const int s = g.split_k, kb = (g.K + BK - 1) / BK;
  if (s < 1 || s > 8 || (s & (s - 1)) || s > kb || bn / s < 8 || g.a_mn_major || (bn == 32 && g.b_mn_major)) return -12;
  if (bn == 32) return launch_bn<32>(ta, tb, g, st);
  if (bn == 64) return launch_bn<64>(ta, tb, g, st);
  return launch_bn<128>(ta, tb, g, st);
}

namespace {
template <int MODE, bool MN, bool LN>
int launch_narrow_one(const GemmArgs& g, const NarrowArgs& n, cudaStream_t st) {
  static bool attr_set[kMaxDevices] = {false};
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= kMaxDevices) return -2;
  if (!attr_set[dev]) {
    if (cudaFuncSetAttribute(gemm_narrow_kernel<MODE, MN, LN>, cudaFuncAttributeMaxDynamicSharedMemorySize, narrow_smem_bytes(NARROW_MAX_K, 8)) !=
        cudaSuccess)
      return -2;
    attr_set[dev] = true;
  }
  const dim3 grid((g.M + NARROW_ROWS - 1) / NARROW_ROWS, (g.N + NARROW_COLS - 1) / NARROW_COLS);
  return launch(gemm_narrow_kernel<MODE, MN, LN>, grid, NARROW_THREADS, narrow_smem_bytes(g.K, g.split_k), st, 1, g, n) == cudaSuccess ? 0 : -3;
}
template <bool MN>
int launch_narrow_mn(const GemmArgs& g, const NarrowArgs& n, cudaStream_t st) {
  switch (g.mode) {
    case EPI_STORE: return launch_narrow_one<EPI_STORE, MN, false>(g, n, st);
    case EPI_GELU: return launch_narrow_one<EPI_GELU, MN, false>(g, n, st);
    case EPI_RESID: return launch_narrow_one<EPI_RESID, MN, false>(g, n, st);
    case EPI_MUL: return launch_narrow_one<EPI_MUL, MN, false>(g, n, st);
    default: return -13;
  }
}
template <bool MN>
int load_narrow() {
  cudaFuncAttributes a;
  return cudaFuncGetAttributes(&a, gemm_narrow_kernel<EPI_STORE, MN, false>) != cudaSuccess ||
         cudaFuncGetAttributes(&a, gemm_narrow_kernel<EPI_GELU, MN, false>) != cudaSuccess ||
         cudaFuncGetAttributes(&a, gemm_narrow_kernel<EPI_RESID, MN, false>) != cudaSuccess ||
         cudaFuncGetAttributes(&a, gemm_narrow_kernel<EPI_MUL, MN, false>) != cudaSuccess ||
         cudaFuncGetAttributes(&a, gemm_narrow_kernel<EPI_STORE, false, true>) != cudaSuccess ||
         cudaFuncGetAttributes(&a, gemm_narrow_kernel<EPI_GELU, false, true>) != cudaSuccess;
}
}  // namespace

int launch_narrow(const GemmArgs& g, const NarrowArgs& n, bool layernorm, cudaStream_t st) {
  if (layernorm) return g.mode == EPI_GELU ? launch_narrow_one<EPI_GELU, false, true>(g, n, st) : launch_narrow_one<EPI_STORE, false, true>(g, n, st);
  return g.b_mn_major ? launch_narrow_mn<true>(g, n, st) : launch_narrow_mn<false>(g, n, st);
}

int load_split_kernels() { return load_narrow<false>() || load_narrow<true>() ? -1 : (load_bn<32>() | load_bn<64>() | load_bn<128>()) ? -1 : 0; }

}  // namespace dsw
