// Banded affine Smith-Waterman (gapped.rs:67-203) with the lanes of a warp on
// one band: the bands of the score pass wider than the lane kernel's 511
// columns (sw_sys.cu).
//
// Intra-band, systolic: lane l runs strip 32b + l of the band (16
// DP rows, the same s16x2 pair layout and column recurrence as the packed
// inter-band kernel) in block b of 32 strips.  Strip k + 1 at relative column
// c needs the (H, E') of strip k's last row at strip k's relative column c +
// 16, which strip k produces at its step c + 17.  So lane l runs its step c at
// warp time T = c + 18 l and takes that word from lane l - 1's output of time
// T - 1 with one shuffle; the D operand is the word of the step before.  Lane
// 0 of block b + 1 reads lane 31's words of block b from shared memory.
//
// Few bands are this wide (1,600 of 42,000 in the search of 13 queries at the
// highest sensitivity), so the chain of a step bounds them: eight pairs of two
// DPX operations.  Everything else is kept off it.  Cells outside the band are
// dead through an addend on their diagonal and open cost instead of masks on
// what they give (as in the lane kernel, sw_sys.cu): -16384 for pair p in the columns
// where it was for pair 0 p columns earlier, one new value per column.  A lane
// runs dead columns before its strip starts and after it ends, without a
// branch.  Letters are loaded four columns ahead, profile words lie one lane
// to a bank.  (Masks on H, E and F of each pair, a branch per step and the
// letter loaded when used: 3,000 -> 1,590 us for
// those bands.)
//
// Scores equal the packed inter-band kernel's and hence the reference's.
#include "kernels.h"
#include "smem_limit.h"
#include "sw_common.cuh"

namespace drg {

namespace {

using namespace sw;

constexpr int kLag = kRows + 2;   // steps between consecutive lanes
constexpr int kProfWords = 26 * 4 * 32;  // profile of a warp's strips: [residue][rows 4w..4w+3][lane]
constexpr int kBandWarps = 4;

// Columns that a residue is loaded ahead of its use.
constexpr int kQueue = 4;

struct Lane {
  const uint8_t* s;  // subject letters
  int m;             // subject length
  int jbase;         // absolute column of relative column 0 in this strip
  uint32_t queue[kQueue];  // prefetched residues of the next columns
};

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

// State of a lane's strip; M[p]: what the cells of pair p add at this column.
struct BandRegs {
  uint32_t H[kPairs], F[kPairs], M[kPairs];
  uint32_t E7, htop_old, mx0, mx1;
  uint32_t hi[2];  // profile words of rows 8 to 15 at the last column
};

// One column step of a strip; rw is the (H, E') word of the row above at this
// column and M[0] is set.  Returns the word of row 15 at the last column.
__device__ __forceinline__ uint32_t band_step(BandRegs& R, const uint32_t* __restrict__ prof, uint32_t res,
                                              uint32_t rw, uint32_t noc2, uint32_t nge2) {
  const uint32_t* row = prof + res * 128;
  const uint32_t lo[2] = {row[0], row[32]}, hi[2] = {R.hi[0], R.hi[1]};
  R.hi[0] = row[64];
  R.hi[1] = row[96];
  const uint32_t h_top = prmt(rw, R.H[kPairs - 1], 0x5410);
  uint32_t h_up = h_top;
  uint32_t e_up = prmt(rw, R.E7, 0x5432);
  uint32_t hd = R.htop_old;
#pragma unroll
  for (int p = 0; p < kPairs; ++p) {
    const uint32_t sc = prmt(lo[p >> 2], hi[p >> 2], pick_sel(p & 3));
    const uint32_t no = add2(noc2, R.M[p]);
    const uint32_t e = __viaddmax_s16x2(e_up, nge2, h_up);
    const uint32_t h =
        __viaddmax_s16x2(e, no, __viaddmax_s16x2_relu(R.F[p], no, add2(hd, add2(sc, R.M[p]))));
    hd = R.H[p];
    R.H[p] = h;
    R.F[p] = __viaddmax_s16x2(R.F[p], nge2, h);
    h_up = h;
    e_up = e;
  }
  R.mx0 = __vimax3_s16x2(R.mx0, R.H[0], R.H[1]);
  R.mx1 = __vimax3_s16x2(R.mx1, R.H[2], R.H[3]);
  R.mx0 = __vimax3_s16x2(R.mx0, R.H[4], R.H[5]);
  R.mx1 = __vimax3_s16x2(R.mx1, R.H[6], R.H[7]);
  R.E7 = e_up;
  R.htop_old = h_top;
  return prmt(R.H[kPairs - 1], add2(R.E7, R.M[kPairs - 1]), 0x7632);  // E' dead with its row
}

__global__ void __launch_bounds__(kBandWarps * 32) k_sw_band(SwBandArgs a) {
  extern __shared__ __align__(16) uint8_t smem[];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  int8_t* mat = reinterpret_cast<int8_t*>(smem);
  for (int i = threadIdx.x; i < 625; i += blockDim.x) mat[i] = a.scores625[i];
  __syncthreads();
  const uint64_t t = a.lo + (uint64_t)blockIdx.x * kBandWarps + warp;
  if (t >= a.hi) return;  // warp-uniform
  uint32_t* prof = reinterpret_cast<uint32_t*>(smem + 640) + warp * kProfWords + lane;
  uint32_t* xbuf =
      reinterpret_cast<uint32_t*>(smem + 640) + kBandWarps * kProfWords + (size_t)warp * 2 * a.xbuf_words;
  const SwBandJob job = a.jobs[t];
  const Band band = a.bands[job.band];
  const int W = band.d1 - band.d0 + 1;
  const int steps = W + kRows;  // column steps of one strip
  const uint8_t* q = a.q_letters + a.q_offsets[band.target] + band.q0;
  const int n = (int)band.n;
  Lane L;
  L.s = a.s_letters + a.s_offsets[band.subject];
  L.m = (int)(a.s_offsets[band.subject + 1] - a.s_offsets[band.subject]);
  const uint32_t noc2 = (uint32_t)(uint16_t)(-(a.gap_open + a.gap_extend)) * 0x10001u;
  const uint32_t nge2 = (uint32_t)(uint16_t)(-a.gap_extend) * 0x10001u;
  int best = 0, best_i = 0;
  const int n_strips = (int)job.n_strips;
  for (int b0 = 0, blk = 0; b0 < n_strips; b0 += 32, ++blk) {
    const int cnt = min(32, n_strips - b0);
    const bool feeds_next = b0 + 32 < n_strips;
    const int i0 = (int)job.row_first + kRows * (b0 + lane);
    // this lane's strip profile (rows past the query: the sentinel's score)
    {
      uint32_t qr[kRows];
#pragma unroll
      for (int r = 0; r < kRows; ++r) {
        const int i = i0 + r;
        qr[r] = lane >= cnt || i > n ? 255u : (uint32_t)min((uint32_t)q[i - 1], 24u);
      }
      for (int res = 0; res < 26; ++res) {
#pragma unroll
        for (int r4 = 0; r4 < 4; ++r4) {
          uint32_t w = 0;
#pragma unroll
          for (int k = 0; k < 4; ++k) {
            const uint32_t r = qr[r4 * 4 + k];
            const int v = (res == 25 || r == 255u) ? kSentinelScore : mat[r * 25 + res];
            w |= ((uint32_t)(uint8_t)(int8_t)v) << (8 * k);
          }
          prof[(res * 4 + r4) * 32] = w;
        }
      }
    }
    __syncwarp();
    const uint32_t* xin = xbuf + (size_t)((blk + 1) & 1) * a.xbuf_words;  // lane 31's words of the last block
    uint32_t* xout = xbuf + (size_t)(blk & 1) * a.xbuf_words;
    L.jbase = i0 - band.d1;
    BandRegs R;
#pragma unroll
    for (int p = 0; p < kPairs; ++p) {
      R.H[p] = R.F[p] = 0;
      R.M[p] = kNeg2;
    }
    R.E7 = 0;
    R.mx0 = R.mx1 = 0;
    R.htop_old = lane == 0 && blk > 0 ? xin[kRows] & 0xFFFFu : 0u;  // H of the row above at column -1
    // columns inside the band: [0, width) of pair 0's low half, 9 later of its
    // high half; none without a strip
    const unsigned width = lane < cnt ? (unsigned)W : 0u;
    int c = -kLag * lane;
    {
      const uint32_t* row = prof + subject_residue(L, L.jbase + c - 2) * 128;
      R.hi[0] = row[64];
      R.hi[1] = row[96];
    }
#pragma unroll
    for (int i = 0; i < kQueue; ++i) L.queue[i] = subject_residue(L, L.jbase + c - 1 + i);
    uint32_t out = 0;
    const int t_end = steps + kLag * (cnt - 1);
#pragma unroll 2
    for (int T = 0; T < t_end; ++T) {
      uint32_t rw = __shfl_up_sync(0xFFFFFFFFu, out, 1);
      if (lane == 0) rw = blk > 0 && c + kRows + 1 < steps ? xin[c + kRows + 1] : 0u;  // row 0 of the reference: dead
#pragma unroll
      for (int p = kPairs - 1; p > 0; --p) R.M[p] = R.M[p - 1];
      R.M[0] = ((unsigned)c < width ? 0u : kNeg2 & 0xFFFFu) | ((unsigned)(c - 9) < width ? 0u : kNeg2 & 0xFFFF0000u);
      out = band_step(R, prof, next_residue(L, c), rw, noc2, nge2);
      if (feeds_next && lane == 31 && (unsigned)c < (unsigned)steps) xout[c] = out;
      ++c;
    }
    const uint32_t mx = max2(R.mx0, R.mx1);
    const int v = max(lo16(mx), hi16(mx));
    if (v > best) {
      best = v;
      best_i = i0 + kRows - 1;  // a bound of the best's row
    }
    __syncwarp();
  }
  // first row-major maximum over the lanes: highest score, then lowest row
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    const int ob = __shfl_xor_sync(0xFFFFFFFFu, best, o);
    const int oi = __shfl_xor_sync(0xFFFFFFFFu, best_i, o);
    if (ob > best || (ob == best && ob > 0 && oi < best_i)) {
      best = ob;
      best_i = oi;
    }
  }
  best_i = best == 0 ? 0 : min(best_i, n);
  if (lane != 0) return;
  a.score[job.band] = best;
  if (a.best_row) a.best_row[job.band] = best_i;
}

}  // namespace

size_t sw_band_smem(int max_width) {
  const size_t xwords = (size_t)(max_width + kRows + 2) & ~(size_t)1;
  return 640 + (size_t)kBandWarps * kProfWords * 4 + (size_t)kBandWarps * 2 * xwords * 4;
}

void launch_sw_band(SwBandArgs a, int max_width, cudaStream_t st) {
  if (a.hi <= a.lo) return;
  a.xbuf_words = (uint32_t)(((size_t)(max_width + kRows + 2)) & ~(size_t)1);
  const size_t smem = sw_band_smem(max_width);
  allow_smem((const void*)k_sw_band, sw_band_smem(kSwMaxWidth));
  const int blocks = ceil_div((long long)(a.hi - a.lo), kBandWarps);
  count_launch();
  k_sw_band<<<blocks, kBandWarps * 32, smem, st>>>(a);
  DRG_CUDA(cudaGetLastError());
}

}  // namespace drg
