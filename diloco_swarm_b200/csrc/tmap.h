// Tensor maps for the TMA loads and stores of the GEMM and attention kernels (gemm_tcgen05.cu).
#pragma once
#include <cuda.h>

namespace dsw {

enum { TMAP_BF16_2D = 0, TMAP_BF16_4D = 1, TMAP_F32_4D = 2 };

// Encoded map from a per-thread table of recent ones.  2-D: `inner` contiguous elements, `outer` rows of `ld` elements
// (ncol = batch = 1).  4-D: a [batch, outer, ncol * inner] array seen as (inner, ncol, outer, batch).
int cached_tmap(CUtensorMap* tm, int kind, const void* ptr, long long inner, long long ncol, long long outer, long long ld,
                int box_inner, int box_outer, long long batch = 1);

}  // namespace dsw
