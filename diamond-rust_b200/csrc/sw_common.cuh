// Shared pieces of the packed 16-bit banded Smith-Waterman kernels: the
// s16x2 helpers, the per-thread register state of one 16-row strip and the
// per-lane subject view.  A strip's 16 rows are 8 pairs of 16-bit lanes: pair
// p holds row p at column c (low half) and row p + 8 at column c - 1 (high
// half).
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

// Columns that a residue is loaded ahead of its use (2, 3, 6 and 8 measured
// beside 4: 17.92, 18.10, 17.82 and 17.81 ms against 17.82 for the 1,000-query
// sensitive search).
constexpr int kQueue = 4;

struct Lane {
  const uint8_t* s;  // subject letters
  int m;             // subject length
  int jbase;         // absolute column of relative column 0 in this strip
  uint32_t queue[kQueue];  // prefetched residues of the next columns
};

// Residue of subject index j, or the sentinel off the sequence.
__device__ __forceinline__ uint32_t subject_residue(const Lane& L, int j) {
  return ((unsigned)j < (unsigned)L.m) ? (uint32_t)__ldg(L.s + j) : (uint32_t)kSentinel;
}
// The residue of column c (subject index jbase + c - 1) from the prefetch
// queue, issuing the load of column c + kQueue.
__device__ __forceinline__ uint32_t next_residue(Lane& L, int c) {
  const uint32_t ahead = subject_residue(L, L.jbase + c + kQueue - 1);
  const uint32_t res = L.queue[0];
#pragma unroll
  for (int i = 0; i + 1 < kQueue; ++i) L.queue[i] = L.queue[i + 1];
  L.queue[kQueue - 1] = ahead;
  return res;
}

__device__ __forceinline__ int lo16(uint32_t x) { return (int)(int16_t)(x & 0xFFFFu); }
__device__ __forceinline__ int hi16(uint32_t x) { return (int)(int16_t)(x >> 16); }

}  // namespace sw
}  // namespace drg
