// Instantiations and launcher of the CTA-pair tcgen05 GEMM kernel (gemm_kernels.cuh): 256 x 256 and
// 256 x 128 tiles on two CTAs of a cluster (cta_group::2), one instantiation per width and epilogue class.
#include "gemm_kernels.cuh"
#include "dswarm.h"
#include "launch.h"

namespace dsw {

namespace {
constexpr int kMaxDevices = 64;

template <int BN, int MODE>
int launch_pair_mode(const CUtensorMap& ta, const CUtensorMap& tb, const GemmArgs& g, int num_sms, int max_ctas,
                     cudaStream_t st) {
  static bool attr_set[kMaxDevices] = {false};          // the attribute is per device
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= kMaxDevices) return -2;
  if (!attr_set[dev]) {
    if (cudaFuncSetAttribute(gemm_pair_kernel<BN, MODE>, cudaFuncAttributeMaxDynamicSharedMemorySize, PairSmem<BN>::TOTAL) !=
        cudaSuccess)
      return -2;
    attr_set[dev] = true;
  }
  const int tiles = ((g.M + 255) / 256) * ((g.N + BN - 1) / BN) * (g.split_k > 1 ? g.split_k : 1);
  int pairs = num_sms / 2;
  if (max_ctas > 0 && pairs > max_ctas / 2) pairs = max_ctas / 2 > 0 ? max_ctas / 2 : 1;
  if (pairs > tiles) pairs = tiles;
  return launch(gemm_pair_kernel<BN, MODE>, 2 * pairs, GEMM_THREADS, PairSmem<BN>::TOTAL, st, 1, ta, tb, g) == cudaSuccess ? 0 : -3;
}

template <int BN>
int launch_bn(const CUtensorMap& ta, const CUtensorMap& tb, const GemmArgs& g, int num_sms, int max_ctas, cudaStream_t st) {
  switch (epi_class(g)) {
    case EPI_GELU: return launch_pair_mode<BN, EPI_GELU>(ta, tb, g, num_sms, max_ctas, st);
    case EPI_GELU_ONLY: return launch_pair_mode<BN, EPI_GELU_ONLY>(ta, tb, g, num_sms, max_ctas, st);
    case EPI_RESID: return launch_pair_mode<BN, EPI_RESID>(ta, tb, g, num_sms, max_ctas, st);
    case EPI_RESID_LO: return launch_pair_mode<BN, EPI_RESID_LO>(ta, tb, g, num_sms, max_ctas, st);
    case EPI_MUL: return launch_pair_mode<BN, EPI_MUL>(ta, tb, g, num_sms, max_ctas, st);
    case EPI_MUL_SUM: return launch_pair_mode<BN, EPI_MUL_SUM>(ta, tb, g, num_sms, max_ctas, st);
    case EPI_ATOMIC_F32: return launch_pair_mode<BN, EPI_ATOMIC_F32>(ta, tb, g, num_sms, max_ctas, st);
    case EPI_STORE: return launch_pair_mode<BN, EPI_STORE>(ta, tb, g, num_sms, max_ctas, st);
    default: break;
  }
  if constexpr (BN == 256) {          // the LM head's epilogues
    if (g.mode == EPI_LSE) return launch_pair_mode<BN, EPI_LSE>(ta, tb, g, num_sms, max_ctas, st);
    if (g.mode == EPI_DLOGITS) return launch_pair_mode<BN, EPI_DLOGITS>(ta, tb, g, num_sms, max_ctas, st);
  }
  return -13;
}

template <int BN>
int load_bn() {
  cudaFuncAttributes a;
  int bad = 0;
  bad |= cudaFuncGetAttributes(&a, gemm_pair_kernel<BN, EPI_STORE>) != cudaSuccess;
  bad |= cudaFuncGetAttributes(&a, gemm_pair_kernel<BN, EPI_GELU>) != cudaSuccess;
  bad |= cudaFuncGetAttributes(&a, gemm_pair_kernel<BN, EPI_GELU_ONLY>) != cudaSuccess;
  bad |= cudaFuncGetAttributes(&a, gemm_pair_kernel<BN, EPI_RESID>) != cudaSuccess;
  bad |= cudaFuncGetAttributes(&a, gemm_pair_kernel<BN, EPI_RESID_LO>) != cudaSuccess;
  bad |= cudaFuncGetAttributes(&a, gemm_pair_kernel<BN, EPI_MUL>) != cudaSuccess;
  bad |= cudaFuncGetAttributes(&a, gemm_pair_kernel<BN, EPI_MUL_SUM>) != cudaSuccess;
  bad |= cudaFuncGetAttributes(&a, gemm_pair_kernel<BN, EPI_ATOMIC_F32>) != cudaSuccess;
  if constexpr (BN == 256) {
    bad |= cudaFuncGetAttributes(&a, gemm_pair_kernel<BN, EPI_LSE>) != cudaSuccess;
    bad |= cudaFuncGetAttributes(&a, gemm_pair_kernel<BN, EPI_DLOGITS>) != cudaSuccess;
  }
  return bad;
}
}  // namespace

int launch_pair(int bn, const CUtensorMap& ta, const CUtensorMap& tb, const GemmArgs& g, int num_sms, int max_ctas,
                cudaStream_t st) {
  return bn == 256 ? launch_bn<256>(ta, tb, g, num_sms, max_ctas, st) : launch_bn<128>(ta, tb, g, num_sms, max_ctas, st);
}

}  // namespace dsw
DSW_BOUNDS_TU(dsw_bounds_gemm_pair)
namespace dsw {

int load_pair_kernels() { return (load_bn<256>() | load_bn<128>()) ? -1 : 0; }

}  // namespace dsw
