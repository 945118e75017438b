// Shared pieces of the packed 16-bit banded Smith-Waterman kernels.  A strip's
// 16 rows are 8 pairs of 16-bit lanes: pair p holds row p at column c (low half)
// and row p + 8 at column c - 1 (high half).
#pragma once
#include <cstdint>

#include "common.cuh"

namespace drg {
namespace sw {

constexpr int kRows = 16;          // rows per strip
constexpr int kPairs = kRows / 2;  // s16x2 pairs
constexpr uint32_t kNeg2 = 0xC000C000u;  // (-16384, -16384)

__device__ __forceinline__ uint32_t prmt(uint32_t a, uint32_t b, uint32_t sel) {
  uint32_t r;
  asm("prmt.b32 %0, %1, %2, %3;" : "=r"(r) : "r"(a), "r"(b), "r"(sel));
  return r;
}
__device__ __forceinline__ uint32_t add2(uint32_t a, uint32_t b) {
  uint32_t r;
  asm("add.s16x2 %0, %1, %2;" : "=r"(r) : "r"(a), "r"(b));
  return r;
}
__device__ __forceinline__ uint32_t max2(uint32_t a, uint32_t b) {
  uint32_t r;
  asm("max.s16x2 %0, %1, %2;" : "=r"(r) : "r"(a), "r"(b));
  return r;
}
// x << n, 0 from n = 32 on.
__device__ __forceinline__ uint32_t shl_clamp(uint32_t x, int n) {
  uint32_t r;
  asm("shl.b32 %0, %1, %2;" : "=r"(r) : "r"(x), "r"(n));
  return r;
}
// Sign-extending byte pick: low half = byte b of lo, high half = byte b of hi.
__device__ __forceinline__ constexpr uint32_t pick_sel(int b) {
  return (uint32_t)(b) | ((uint32_t)(8 | b) << 4) | ((uint32_t)(4 + b) << 8) | ((uint32_t)(8 | (4 + b)) << 12);
}

// Residue of subject index j, or the sentinel off the sequence.
template <typename Lane>
__device__ __forceinline__ uint32_t subject_residue(const Lane& L, int j) {
  return ((unsigned)j < (unsigned)L.m) ? (uint32_t)__ldg(L.s + j) : (uint32_t)kSentinel;
}

__device__ __forceinline__ int lo16(uint32_t x) { return (int)(int16_t)(x & 0xFFFFu); }
__device__ __forceinline__ int hi16(uint32_t x) { return (int)(int16_t)(x >> 16); }

}  // namespace sw
}  // namespace drg
