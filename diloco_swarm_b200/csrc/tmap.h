// Tensor maps for the TMA loads and stores of the GEMM and attention kernels (gemm_tcgen05.cu).
#pragma once
#include <cuda.h>

namespace dsw {

enum { TMAP_BF16_2D = 0, TMAP_F32_2D = 1, TMAP_BF16_3D = 2, TMAP_F32_3D = 3 };

// Encoded map from a per-thread table of recent ones.  2-D kinds: `inner` contiguous elements, `outer` rows of `ld`
// elements (ncol = 1).  3-D kinds: a [outer, ncol * inner] matrix seen as (inner, ncol, outer).
int cached_tmap(CUtensorMap* tm, int kind, const void* ptr, long long inner, long long ncol, long long outer, long long ld,
                int box_inner, int box_outer);

}  // namespace dsw
