// The kernels behind a walk whose trees were split: what the chunks' partial sums become.
#pragma once
#include "walk_kernels.cuh"

namespace tb {

// Second pass: sums the partials of all tree chunks for a row (fixed order, no
// atomics), adds the initial value and applies the transformation / class argmax.
// Reference: the per-column serial sum plus initial value of
// src/reduction/LowerReduceOps.cpp:921-1003.
__global__ void tb_finalize_kernel(const float *__restrict__ partial, int chunks, long long n_rows, int W,
                                   int num_classes, float initial_value, int transform, void *out,
                                   int out_kind) {
  const long long row = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (row >= n_rows) return;
  if (num_classes == 0) {
    float s = 0.f;
    for (int c = 0; c < chunks; ++c) s += partial[(long long)c * n_rows + row];
    reinterpret_cast<float *>(out)[row] = apply_transform(initial_value + s, transform);
  } else {
    const int arg = argmax_last(W, [&](int k) {
      float s = 0.f;
      for (int c = 0; c < chunks; ++c) s += partial[((long long)c * n_rows + row) * W + k];
      return initial_value + s;
    });
    if (out_kind == 1) reinterpret_cast<int8_t *>(out)[row] = (int8_t)arg;
    else reinterpret_cast<float *>(out)[row] = (float)arg;
  }
}

// Sums tree-chunk partials into one partial per row (tree-sharded use: the result is
// what crosses the NVLink reduction).
__global__ void tb_sum_partials_kernel(const float *__restrict__ partial, int chunks, long long total,
                                       float *__restrict__ dst) {
  const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= total) return;
  float s = 0.f;
  for (int c = 0; c < chunks; ++c) s += partial[(long long)c * total + i];
  dst[i] = s;
}

} // namespace tb
