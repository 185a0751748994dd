// Plan-time rules of FP32 contractions that run as products of their operands'
// three-way bf16 splits (TC_F32X6). Plain C++ without CUDA.
#pragma once
#include <cstdint>

namespace tccg {

// K padded to whole k-blocks of 32.
inline int64_t f32_split_k(int64_t K) { return (K + 31) / 32 * 32; }

// Whether every index of the packed operands is representable: rows and K as
// 32-bit values, and the packed columns (hi | mid | lo: 96 per k-block) as TMA
// coordinates, which are signed 32-bit. Past that the last k-blocks would be
// read at negative coordinates, as zeros.
inline bool f32_split_fits(int64_t M, int64_t N, int64_t K) {
  const int64_t lim = int64_t(1) << 30;
  return M < lim && N < lim && K < lim && 3 * f32_split_k(K) <= INT32_MAX;
}

}  // namespace tccg
