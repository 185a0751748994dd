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

// Whether an automatic plan may take the split's workspace: 6 bytes per operand
// element, where the FFMA forms need 4 or none, so a call that fills the GPU could
// fit with those only. Operands, C and workspace together stay within half of
// the 180 GB.
inline bool f32_split_memory(int64_t M, int64_t N, int64_t K) {
  const double k = (double)f32_split_k(K);
  return 10.0 * ((double)M + (double)N) * k + 4.0 * (double)M * (double)N <= 90e9;
}

// k-blocks of 32 per accumulation chunk of an automatic plan, 0 = FFMA, by the
// chains of FP32 adds of the FFMA form: `splits` k slices of `chain` each. Tensor
// memory truncates each of a chunk's 2 sums per k-block, so the split's error
// goes with the chunk and FFMA's with the chain; on operands of one sign the
// truncations add up. RMS error over |A| |B| of six 384 x 320 results, 1e-8,
// FFMA | chunks of 4, 2, 1:
//   chain         128               256                384               768               1536
//   uniform(0,1)  16 | 15 8.2 5.9   22 | 15 8.2 6.3    29 | 15 8.3 6.9   42 | 15 8.0 5.6   59 | 15 8.1 5.8
//   exponential   16 | 19 10  6.6   23 | 19 10  7.1    29 | 19 10  7.6   42 | 19 9.9 6.5   59 | 19 10  6.6
//   lognormal(1)  17 | 16 8.2 5.7   24 | 16 8.3 6.3    28 | 16 8.4 6.7   39 | 16 8.1 5.7   54 | 16 8.2 5.7
//   lognormal(2)  18 | 44 21  12    24 | 45 22  13     30 | 46 23  13    42 | 47 23  13    60 | 48 24  14
//   e^-20u        16 | 46 25  14    26 | 44 24  14     34 | 44 24  15    60 | 43 23  14    107| 42 23  14
//   e^-58u                         8.3| 17 11  8.1    9.9| 17 11  8.7    14 | 16 10 7.8     21 | 15 9.9 7.7
//   normal        2.8| 1.7 1.0 .85  2.7| .9 .6 .6      2.6| .7 .5 .5     2.6| .5 .4 .3     2.6| .3 .3 .2
// Below 256 FFMA stays: 14 against 16 is no distance. 4096 x 4096 x 1024 takes
// 210 us by chunks of 4, 231 of 2, 263 of 1 (FFMA 658).
// Slices add up with independent errors, so they count as chains of chain /
// splits, and their plans run chunks of 1 at least: 384 x 320 x 4096 in 32
// slices, normwise, 1e-8, FFMA | chunks of 2, 1: normal 23 | 11 11, uniform 8.3 |
// 8.9 6.8, exponential 8.4 | 11 7.6, lognormal(1) 9.4 | 9.4 7.3; operands over
// many magnitudes are even or a little behind: lognormal(2) 15 | 32 19,
// e^-20u 13 | 23 14.
inline int f32_split_chunk(int64_t chain, int64_t splits) {
  const int64_t c = chain / splits;
  return c >= 1536 ? 4 : c >= 768 ? 3 : c >= 512 ? 2 : c >= 256 || splits > 1 ? 1 : 0;
}

}  // namespace tccg
