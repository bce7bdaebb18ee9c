// A row's BF16 copy, shared by the pack kernel and the refresh's row pass (the
// same float operations with and without contraction).
#pragma once

#include <cuda_bf16.h>

#include "common.cuh"
#include "kernels.hpp"

namespace kb2::dev {

using launch::Bf16Store;

// scale = max |a_ij| (1 for a zero row), stored value = bf16(a_ij / scale), alone
// or with the column's offset from the row in the low half of a word.
__device__ __forceinline__ void bf16_store_row(int i, const float* vals, const Bf16Store& out) {
  const int begin = out.rows[i], end = out.rows[i + 1];
  float most = 0.0f;
  row_values(vals, begin, end, [&](int, float v) { most = fmaxf(most, fabsf(v)); });
  const float s = most > 0.0f ? most : 1.0f;
  out.scale[i] = s;
  const float inv = 1.0f / s;
  constexpr int kBatch = 8;
  for (int j = begin; j < end; j += kBatch) {
    float v[kBatch];
    int c[kBatch];
#pragma unroll
    for (int k = 0; k < kBatch; ++k) {
      v[k] = j + k < end ? vals[j + k] : 0.0f;
      c[k] = out.packed != nullptr && j + k < end ? out.cols[j + k] : 0;
    }
#pragma unroll
    for (int k = 0; k < kBatch; ++k) {
      if (j + k >= end) continue;
      const unsigned short word = __bfloat16_as_ushort(__float2bfloat16_rn(v[k] * inv));
      if (out.packed != nullptr)
        out.packed[j + k] =
            static_cast<unsigned>(word) << 16 | (static_cast<unsigned>(c[k] - i) & 0xffffu);
      else
        out.v16[j + k] = word;
    }
  }
}

}  // namespace kb2::dev
