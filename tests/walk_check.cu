// The traceback walk's check of where it starts: a best cell outside the
// matrix or the band gives a record of score -1 (an internal error to the host),
// one on its edge an alignment.  Every buffer holds what a walk without the check would read.
#include "sw_sys.cu"

#include <cstdio>

namespace drg {
void count_launch() {}
uint64_t kernel_launch_count() { return 0; }
void launch_sw_band(SwBandArgs, int, cudaStream_t) {}

struct Start {
  int bi, bj, single, score;  // score: the expected record's
};

__global__ void k_walks(SysArgs a, const Start* starts, int m) {
  __shared__ int8_t mat[kResidues * 32];
  stage_scores(mat, a.scores625);
  const Start s = starts[blockIdx.x];
  walk_warp(a, blockIdx.x, a.bands[0], m, CellOut{7, s.bi, s.bj}, mat, s.single != 0,
            [](int, int) -> uint32_t { return 0u; });
}
}  // namespace drg

using namespace drg;

int main() {
  constexpr int kN = 20, kM = 12, kPad = 64;  // band: diagonals -3 to 4
  const Start starts[] = {{10, 9, 0, 7},  {20, 16, 0, -1}, {20, 12, 1, 7}, {20, 12, 0, -1}, {21, 12, 1, -1},
                          {0, 3, 0, -1},  {3, 0, 0, -1},   {14, 13, 0, -1}, {13, 9, 0, 7},  {14, 9, 0, -1},
                          {6, 9, 0, 7},   {5, 9, 0, -1},   {1, 1, 0, 7},    {16, 12, 0, 7}, {-5, 1, 0, -1}};
  constexpr int kStarts = sizeof(starts) / sizeof(starts[0]);
  char* base = nullptr;  // one block of managed memory for all
  DRG_CUDA(cudaMallocManaged(&base, 1 << 20));
  char* at = base;
  auto take = [&](size_t bytes) {
    char* p = at;
    at += (bytes + 255) / 256 * 256;
    return p;
  };
  SysArgs a{};
  uint8_t* letters = (uint8_t*)take(2 * kPad + 64);
  for (int i = 0; i < 2 * kPad + 64; ++i) letters[i] = 0;
  Band* b = (Band*)take(sizeof(Band));
  *b = Band{};
  b->n = kN;
  b->d0 = -3;
  b->d1 = 4;
  uint64_t* off = (uint64_t*)take(2 * 8);
  off[0] = 0;
  off[1] = kM;
  uint64_t* ops_off = (uint64_t*)take(kStarts * 8);
  for (int k = 0; k < kStarts; ++k) ops_off[k] = (uint64_t)k * (kN + kM);
  Start* ds = (Start*)take(sizeof(starts));
  for (int k = 0; k < kStarts; ++k) ds[k] = starts[k];
  a.bands = b;
  a.q_letters = a.s_letters = letters + kPad;
  a.q_offsets = a.s_offsets = off;
  a.ops_off = ops_off;
  a.ops = (uint32_t*)take((size_t)kStarts * (kN + kM) * 4);
  a.out = (ExactOut*)take(kStarts * sizeof(ExactOut));
  a.oc = 12;
  a.ge = 1;
  for (int i = 0; i < 625; ++i) a.scores625[i] = 1;
  k_walks<<<kStarts, 32>>>(a, ds, kM);
  DRG_CUDA(cudaGetLastError());
  DRG_CUDA(cudaDeviceSynchronize());
  for (int k = 0; k < kStarts; ++k) {
    const ExactOut& r = a.out[k];
    const bool found = starts[k].score > 0;
    if (r.score != starts[k].score || (r.n_ops > 0) != found || (found && (int)r.q_end != starts[k].bi)) {
      std::printf("start %d: score %d, %u ops\n", k, r.score, r.n_ops);
      return 1;
    }
  }
  std::printf("ok\n");
  return 0;
}
