// tc_layout.cuh -- layout of the tensor-core blocks' B operand.
#pragma once

#include <cstdint>

namespace kb {

// Byte offset of fp16 element (row, kk) of a K-major image with `rows` rows
// under the 128-byte swizzle.
__host__ __device__ __forceinline__ uint32_t sw128_offset_h(int row, int kk, int rows) {
  const int kb = kk >> 6;             // 64 fp16 per 128-byte atom row
  const int chunk = (kk & 63) >> 3;   // 16-byte chunk in the row
  return (uint32_t)(kb * rows * 128 + row * 128 + ((chunk ^ (row & 7)) << 4) + ((kk & 7) << 1));
}

}  // namespace kb
