// Keys of the rounded-key layouts' thresholds.
#pragma once
#include "walk_quant.cuh"

namespace tb {

// Fills the key field of every split node from its exact threshold (run once at upload,
// so that thresholds and row values are quantised by the very same device arithmetic).
// wide = 1: the 15-bit keys and feature codes of the wide-row layout (quant_pack.h);
// 0: the same keys with the deep-tree layout's codes, `code_unit` per feature (deep_pack.h).
// Pass-through nodes keep their key 0.
__global__ void tb_quant_fill_keys(uint32_t *node_plane, const float *exact_plane, const float *lo,
                                   const float *scale, unsigned long long n, int num_features, int wide, uint32_t code_unit) {
  const unsigned long long i = (unsigned long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const uint32_t node = node_plane[i];
  if (wide) {
    const uint32_t code = node >> 16, f = (code >> 6) * 2u + (code & 1u);
    if (f < (uint32_t)num_features) node_plane[i] = (code << 16) | quant_threshold_key15_dev(exact_plane[i], lo[f], scale[f]);
  } else {
    const uint32_t code = node >> 16, f = code / code_unit;
    if (node & 0xffffu) node_plane[i] = (code << 16) | quant_threshold_key15_dev(exact_plane[i], lo[f], scale[f]);
  }
}

} // namespace tb
