// Gradient of the linear cross-entropy with respect to its logits, from the fp32 logits that the forward product stored.
#pragma once
#include "gemm_sm100.cuh"

namespace opk {

constexpr int kLceGradChunks = 8;      // 32-column blocks per warp: 512 contiguous bytes of every row of the result

// One warp per 32 rows x 256 columns, one row per thread, the arithmetic of EPI_LCE_BWD on the values it would have formed: the
// result has the same bits. Bound by memory (4 bytes read, 2 written per logit); the product that it replaces reads and
// multiplies the hidden states and the head again: 2048 x 128256 logits 280 us (5.6 TB/s) against 709 us for 2048 columns of the
// hidden states and 1,498 us for 4096; storing the logits adds 50 to 110 us to the forward product. Even with the product at 768
// columns (see lce_keeps_logits in ops/gemm.py).
__global__ void __launch_bounds__(256, 2) lce_grad_kernel(const GemmParams p) {
  __shared__ __align__(16) uint8_t scratch[8][kEpiScratch];
  pdl_trigger();
  const int warp = threadIdx.x >> 5;
  const int n_cb = (p.N + 31) >> 5, groups = (n_cb + kLceGradChunks - 1) / kLceGradChunks;
  const long long item = (long long)blockIdx.x * 8 + warp;
  const int rb = (int)(item / groups), g = (int)(item - (long long)rb * groups);
  const int row0 = rb * 32;
  if (row0 >= p.M) return;               // the same in all lanes
  EpiState e = epi_begin<EPI_LCE_GRAD>(p, scratch[warp], row0, 0);
  const int c_begin = g * kLceGradChunks, c_end = min(n_cb, c_begin + kLceGradChunks);
  const float4* z = z_block(p.z, p.N, row0, c_begin * 32);
  float4 next[8];
#pragma unroll
  for (int q = 0; q < 8; ++q) next[q] = __ldcs(z + 32 * q);
#pragma unroll 1
  for (int c = c_begin; c < c_end; ++c) {
    float v[32];
#pragma unroll
    for (int q = 0; q < 8; ++q) { v[4 * q] = next[q].x; v[4 * q + 1] = next[q].y; v[4 * q + 2] = next[q].z; v[4 * q + 3] = next[q].w; }
    z += 256;
    if (c + 1 < c_end) {                 // the next block is in flight while this one is computed
#pragma unroll
      for (int q = 0; q < 8; ++q) next[q] = __ldcs(z + 32 * q);
    }
    epi_chunk<EPI_LCE_GRAD>(p, e, v, c * 32);
  }
}

}  // namespace opk
