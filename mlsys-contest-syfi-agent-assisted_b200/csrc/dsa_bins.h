// The indexer's order of scores and its bins of score values, as plain functions that also compile without CUDA
// (tests check them on the host).
#pragma once
#include <math.h>
#include <stdint.h>
#include <string.h>

#ifdef __CUDACC__
#define SYFI_HD __host__ __device__ __forceinline__
#else
#define SYFI_HD inline
#endif

namespace syfi {

constexpr int kBins = 4096;        // value bins of one sequence: a score's bin is linear in the score

// larger float <-> larger key (NaN aside); key 0 is below every score
SYFI_HD uint32_t score_key(float s) {
  uint32_t u;
  memcpy(&u, &s, 4);
  return (u & 0x80000000u) ? ~u : (u | 0x80000000u);
}

SYFI_HD float key_score(uint32_t key) {   // inverse of score_key
  const uint32_t u = (key & 0x80000000u) ? (key ^ 0x80000000u) : ~key;
  float s;
  memcpy(&s, &u, 4);
  return s;
}

// Always a valid bin: a score outside the range that `lowest` and `scale` describe (the score of a position that was
// never scored, see the score kernel) falls into the first or the last one, NaN into the first.  Every step is
// monotone, rounding included, so a larger score never has a smaller bin.
SYFI_HD int score_bin(float s, float lowest, float scale) {
  return static_cast<int>(fminf(fmaxf((s - lowest) * scale, 0.0f), static_cast<float>(kBins - 1)));
}

}  // namespace syfi
