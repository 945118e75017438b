// Banded affine Smith-Waterman (gapped.rs:67-203) for many bands that share a
// query window (or a subject, transposed): the score pass of the E-value gate.
//
// Mapping (inter-task): one thread = one band; one half warp = up to 16 bands
// of the same query window, which share its profile in shared memory; a warp
// runs two such tasks of nearly equal strips, widths and corners (they are
// sorted so), of any two queries.  A warp runs the union of its bands' rows
// and columns: with 32 bands of one window per warp, 64 bands of a query (the
// 20,000-query search) are two warps whose lanes each need half of it, 1.91
// computed cells per cell of a band; 16 make it 1.65 (15.9 -> 13.1 ms), and
// the 1,000-query sensitive search, 40 warps a query, 1.39 -> 1.33 (12.9 ->
// 12.3 ms).  8 make the former 1.44, but at 12.3 ms, and the latter slower
// (12.4 ms): the profiles cost twice as much, and class 0 has to end at 134
// columns for three blocks to fit an SM.
// The band is swept in strips of 16 DP rows.  Inside a strip, relative column
// c covers absolute subject column j = i0 - d1 + c, and row r of the strip is
// in the band for r <= c <= r + W - 1.  The 16 rows are held as 8 pairs of
// signed 16-bit lanes (DPX s16x2 instructions): pair p holds row p at column c
// in its low half and row p + 8 at column c - 1 in its high half.  With that
// one-column skew every dependency of a pair is already computed.  The gap
// scores are kept with the cost of a gap's first letter added back (oc):
//   E'(i,j) = E + oc = max(E'(i-1,j) - ge, H(i-1,j))   this step, pair above
//   F'(i,j) = F + oc = max(F'(i,j-1) - ge, H(i,j-1))   previous step, same pair
//   H       = max(0, H(i-1,j-1) + S, max(E', F') - oc)
// Row 8's "pair above" is row 7, taken from the previous step; row 0's is the
// previous strip's last row, kept in a per-thread ring in shared memory.  The
// ring holds W + 1 words (H | E' << 16): a strip reads the previous strip's
// word for column c and then overwrites the slot of column c - 1, which is the
// word the next strip needs at its column c - 17.
//
// In this form all of H, E' and F' are at least 0, no H - oc is kept, and a
// cell outside the band or the matrix is plain 0 (E' = 0 is E = -oc, which
// raises nothing).  A pair update is four operations of the ALU pipe, at two
// cycles a warp each, and three adds of the FMA pipe, which runs beside:
//   sc = the pair's two scores (one byte permute)
//   E' = max(E' - ge, H of the pair above)            (viaddmax)
//   H  = max(Hdiag + sc, E' - oc, F' - oc, 0)         (three adds, vimax3.relu)
//   F' = max(F' - ge, H)                              (viaddmax, for the next column)
// Near a strip's ends a cell outside the band is dead by an addend of -16384 on
// its diagonal and open cost, as in the lane kernel (sw_sys.cu, which says why
// the H that it may keep beside scores above 16384 changes none).
//
// ALU bound: that pipe is busy 86.5 % of the time, at 3.35 operations per computed
// cell (ncu, 200 queries).  The recurrence above is 2.25 of them; the edges'
// addends, the letters, the byte picks of a column and the ring are the rest.
// Before, neither more warps nor fewer operations changed anything: with the
// first and last 16 steps of a strip unrolled, each with its masks, the code
// of an SM's twelve warps did not stay in its instruction cache.
// Now two loops of four steps make up a strip, edges and middle.  A loop holds
// whole groups of four columns because a load in flight that is moved from
// register to register waits, so letters come four at a time as words, a group
// ahead (loaded singly into a rotating queue, with loops of 1, 2, 3 and 4
// steps: 23.0, 18.4, 17.6 and 17.0 ms for the 1,000-query sensitive search;
// unrolled edges 16.8; now 15.25, and 13.8 -> 12.6 ms for 250 very-sensitive
// queries).
//
// Exactness: values equal the reference's int32 DP while the band's best is
// below 31744 = 0x7C00 (bands that could reach it are not given to this
// kernel).
// Cells with j < 0, j > m or rows past the query read a sentinel residue
// scoring -64; they can neither raise the maximum above the true band maximum
// nor feed an in-band cell.  Rows past m + d1 are not computed: the reference
// keeps one cell per such row, clamped to column m, whose H is at most
// max(largest matrix score, band best - open), so a packed best above the
// matrix's largest score is the reference's; smaller results are recomputed
// exactly.
//
// The traceback of the HSPs that pass the gate runs in sw_sys.cu.
#include "kernels.h"
#include "smem_limit.h"
#include "sw_common.cuh"

namespace drg {

namespace {

using namespace sw;

constexpr int kParts = 32 / kSwPart;  // tasks per warp
constexpr int kProfHigh = 26 * 8;     // profile bytes of rows 8 to 15, after those of rows 0 to 7
constexpr int kProfBytes = 2 * kProfHigh;

// The column letters of one lane, a group of four columns at a time: taken
// from the two aligned words that hold them (the second is the next group's
// first), fetched a group ahead.  Every letter buffer starts on a word
// boundary and has slack behind its end.
struct Letters {
  const uint8_t* s;  // column letters
  int m;             // how many
  int jbase;         // absolute column of relative column 0 in this strip
  uint32_t w0, w1;  // aligned words: of the next group's first letter, and the one after
  uint32_t shift;   // bits of w0 before the group's first letter
  int j;            // subject index of the next group's first column
};

// The aligned word of letters [t, t + 4), s + t on a word boundary; not read
// where no letter of it is the sequence's.
__device__ __forceinline__ uint32_t letter_word(const Letters& L, int t) {
  return (unsigned)t + 3u < (unsigned)L.m + 3u ? __ldg(reinterpret_cast<const uint32_t*>(L.s + t)) : 0u;
}
// Before column c (a multiple of 4) of a strip.
__device__ __forceinline__ void letters_at(Letters& L, int c) {
  L.j = L.jbase + c - 1;
  const int off = (int)((reinterpret_cast<uintptr_t>(L.s) + (intptr_t)L.j) & 3);
  L.shift = 8 * off;
  L.w0 = letter_word(L, L.j - off);
  L.w1 = letter_word(L, L.j - off + 4);
}
// The next four columns' residues, the sentinel off the sequence.
__device__ __forceinline__ uint32_t next_letters(Letters& L) {
  const uint32_t w = __funnelshift_r(L.w0, L.w1, L.shift);
  L.w0 = L.w1;
  L.w1 = letter_word(L, L.j + 8 - (int)(L.shift >> 3));
  const uint32_t below = shl_clamp(0xFFFFFFFFu, 8 * __vimin_s32_relu(-L.j, 4));      // letters from index 0 on
  const uint32_t past = shl_clamp(0xFFFFFFFFu, 8 * __vimin_s32_relu(L.m - L.j, 4));  // letters from index m on
  const uint32_t in = below & ~past;
  L.j += 4;
  return (w & in) | (0x01010101u * kSentinel & ~in);
}

// Registers of one lane's 16-row strip in the score pass.
struct SRegs {
  uint32_t H[kPairs], F[kPairs];
  uint32_t E7;        // E' of pair 7 at the previous step
  uint32_t htop_old;  // H above pair 0 at the previous step (its D operand)
  const uint8_t* prow_prev;  // profile row of the previous column's residue
  uint32_t mx0, mx1;  // maximum H of the strip so far, folded over rows
};

// The residue of a group's column k.
__device__ __forceinline__ uint32_t residue(uint32_t r4, int k) { return prmt(r4, 0u, 0x4440u + k); }

// One column step.  res is the column's residue, rw the (H, E') word of the row above row 0 at column c;
// wp receives row 15's word of column c - 1.  EDGE: near a strip's first and
// last columns, where M[p] holds what pair p's cells outside the band add.
template <bool EDGE>
__device__ __forceinline__ void sw_step(SRegs& R, uint32_t res, const uint8_t* __restrict__ prof, uint32_t rw,
                                        uint32_t* __restrict__ wp, uint32_t noc2, uint32_t nge2,
                                        const uint32_t (&M)[kPairs]) {
  const uint8_t* prow = prof + res * 8;
  const uint2 lo8 = *reinterpret_cast<const uint2*>(prow);
  const uint2 hi8 = *reinterpret_cast<const uint2*>(R.prow_prev + kProfHigh);
  R.prow_prev = prow;
  const uint32_t h_top = prmt(rw, R.H[kPairs - 1], 0x5410);
  uint32_t h_up = h_top;
  uint32_t e_up = prmt(rw, R.E7, 0x5432);
  uint32_t hd = R.htop_old;
#pragma unroll
  for (int p = 0; p < kPairs; ++p) {
    uint32_t sc = prmt(p < 4 ? lo8.x : lo8.y, p < 4 ? hi8.x : hi8.y, pick_sel(p & 3));
    uint32_t no = noc2;
    if (EDGE) {
      sc = add2(sc, M[p]);
      no = add2(no, M[p]);
    }
    const uint32_t f = R.F[p];
    const uint32_t e = __viaddmax_s16x2(e_up, nge2, h_up);
    // (at the edges the FMA pipe has two adds more: one of these goes back)
    const uint32_t h = EDGE ? __viaddmax_s16x2(e, no, __viaddmax_s16x2_relu(f, no, add2(hd, sc)))
                            : __vimax3_s16x2_relu(add2(hd, sc), add2(f, no), add2(e, no));
    hd = R.H[p];
    R.H[p] = h;
    R.F[p] = __viaddmax_s16x2(f, nge2, h);
    h_up = h;
    e_up = e;
  }
  // the strip's maximum, two accumulators of four pairs each
  R.mx0 = __vimax3_s16x2(R.mx0, R.H[0], R.H[1]);
  R.mx1 = __vimax3_s16x2(R.mx1, R.H[4], R.H[5]);
  R.mx0 = __vimax3_s16x2(R.mx0, R.H[2], R.H[3]);
  R.mx1 = __vimax3_s16x2(R.mx1, R.H[6], R.H[7]);
  R.E7 = e_up;
  // (H, E') of row 15 at column c - 1; E' dead with its row
  *wp = prmt(R.H[kPairs - 1], EDGE ? add2(R.E7, M[kPairs - 1]) : R.E7, 0x7632);
  R.htop_old = h_top;
}

// Words of a lane's ring: at least W + 1, a whole number of groups.  (A strip
// may run up to three columns past W + 16, to the end of a group; then the
// ring has a word more for each but two, which keeps the words that it writes
// there off those that the next strip reads.)
__host__ __device__ constexpr int ring_words(int W) { return (W + 4) & ~3; }

// Score pass: scores[band] = the band's best H, best_row[band] = the last row
// of the first strip that holds it (an upper bound of the reference's best_i,
// which is all the traceback pass needs).
// Shared memory holds three blocks per SM in the 4- and 2-warp classes.
template <int WARPS>
__global__ void __launch_bounds__(WARPS * 32, WARPS >= 2 ? 3 : 1) k_sw(SwScoreArgs a) {
  extern __shared__ __align__(16) uint8_t smem[];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int part = lane / kSwPart, at = lane % kSwPart;
  const uint64_t task_id = a.task_lo + ((uint64_t)blockIdx.x * WARPS + warp) * kParts;
  constexpr int stride = WARPS * 32;
  int8_t* mat = reinterpret_cast<int8_t*>(smem);  // 25 x 25 scores
  uint8_t* prof = smem + 640 + (warp * kParts + part) * kProfBytes;  // strip profile
  uint32_t* ring = reinterpret_cast<uint32_t*>(smem + 640 + WARPS * kParts * kProfBytes) + threadIdx.x;
  for (int i = threadIdx.x; i < 625; i += blockDim.x) mat[i] = a.scores625[i];
  __syncthreads();
  if (task_id >= a.task_hi) return;
  // a part past the launch's last task repeats the warp's first, to no effect
  const bool idle = task_id + part >= a.task_hi;
  const SwTask task = a.tasks[task_id + (idle ? 0 : part)];
  const int W = (int)__reduce_max_sync(0xFFFFFFFFu, task.width);     // widest band of the warp
  const int Wmin = (int)__reduce_min_sync(0xFFFFFFFFu, task.w_min);  // narrowest
  const uint32_t n_strips = __reduce_max_sync(0xFFFFFFFFu, task.n_strips);
  const int buf = ring_words(W);
  const bool active = !idle && at < (int)task.count;
  const uint32_t bidx = a.order[task.first + (at < (int)task.count ? at : 0)];
  const Band band = a.bands[bidx];
  const int Wl = band.d1 - band.d0 + 1;  // this lane's width
  // Rows are the query window and columns the subject, or (a transposed
  // task, whose lanes share the subject) rows the subject and columns the
  // window with the diagonals negated: the same cells, so the same best.
  const bool tr = task.transposed != 0;
  const uint8_t* qw = a.q_letters + a.q_offsets[band.target] + band.q0;
  const uint8_t* sj = a.s_letters + a.s_offsets[band.subject];
  const int m_s = (int)(a.s_offsets[band.subject + 1] - a.s_offsets[band.subject]);
  const uint8_t* q = tr ? sj : qw;  // row letters
  const int n = tr ? m_s : (int)band.n;
  const int d1 = tr ? -band.d0 : band.d1;
  Letters L;
  L.s = tr ? qw : sj;  // column letters
  L.m = tr ? (int)band.n : m_s;
  const uint32_t noc2 = (uint32_t)(uint16_t)(-(a.gap_open + a.gap_extend)) * 0x10001u;
  const uint32_t nge2 = (uint32_t)(uint16_t)(-a.gap_extend) * 0x10001u;
  // a dead cell's word is 0 (H = 0, E' = 0); the row above the first strip, row
  // 0 of the reference, is dead
  for (int g = 0; g < buf; ++g) ring[g * stride] = 0;
  uint32_t* const ring_end = ring + buf * stride;
  int base = 0;  // ring slot of relative column 0 of the current strip
  SRegs R;
  int best = 0, best_i = 0;
  uint64_t steps_done = 0;  // column steps run (all strips)
  for (uint32_t k = 0; k < n_strips; ++k) {
    const int i0 = (int)task.row_first + (int)(k * kRows);
    // strip profile of each part: the score of row i0 + r against column
    // residue res at prof[8 res + r] (r < 8), prof[kProfHigh + 8 res + r - 8];
    // a lane writes one row (rows at..at + kSwPart step)
    __syncwarp();
    for (int r = at; r < kRows; r += kSwPart) {
      const int i = i0 + r;
      const bool in = i <= n;
      const int row = in ? (int)min((uint32_t)q[i - 1], 24u) : 0;
      const int8_t* sc = mat + (tr ? row : row * 25);
      const int step = tr ? 25 : 1;
      uint8_t* out = prof + (r < 8 ? r : kProfHigh + r - 8);
#pragma unroll 5
      for (int res = 0; res < 25; ++res) out[res * 8] = (uint8_t)(in ? sc[res * step] : (int8_t)kSentinelScore);
      out[25 * 8] = (uint8_t)(int8_t)kSentinelScore;
    }
    __syncwarp();
    L.jbase = i0 - d1;
    // column c_begin - 1 of the strip: dead cells
#pragma unroll
    for (int p = 0; p < kPairs; ++p) R.H[p] = R.F[p] = 0;
    R.mx0 = R.mx1 = 0;
    R.E7 = 0;
    // Steps whose cells all lie off the matrix for every lane of the warp are
    // skipped: at step c a lane's cells sit at subject columns jbase + c (rows
    // 0-7) and jbase + c - 1 (rows 8-15), all j <= 0 for c <= -jbase and all
    // j > m for c >= m + 2 - jbase.  Such cells are H = 0 on the left and can
    // never exceed an in-matrix value on the right, so only the ring words a
    // later strip reads need care (below).
    const int lead = __reduce_min_sync(0xFFFFFFFFu, max(0, 1 - L.jbase));
    const int trail = __reduce_max_sync(0xFFFFFFFFu, L.m + 2 - L.jbase);
    // (whole groups of columns, and the whole prologue or none of it)
    const int c_begin = lead >= kRows ? min(lead, Wmin) & ~3 : 0;
    const int c_end = (max(c_begin, min(W + kRows, max(trail, kRows))) + 3) & ~3;
    steps_done += (uint64_t)(c_end - c_begin);
    // rp: the ring word of column c; wp: the slot before, which takes the word
    // of column c - 1 once that is read.  base, the ring and c are multiples of
    // 4 here, so only the end of a group meets the wrap of the ring.
    int slot = base + c_begin;
    slot = slot >= buf ? slot - buf : slot;
    uint32_t* rp = ring + slot * stride;
    uint32_t* wp = slot == 0 ? ring_end - stride : rp - stride;
    // H of column c_begin - 1 of the row above; row 7 not yet computed: 0
    R.htop_old = *wp & 0xFFFFu;
    R.prow_prev = prof + subject_residue(L, L.jbase + c_begin - 2) * 8;  // column c_begin - 1
    letters_at(L, c_begin);
    // The steps with an edge of the band among a strip's rows, the first 16 and
    // those from the narrowest band's width on, are one loop, entered before and
    // after the steps between.  Pair p is at the edge p columns after pair 0, so
    // a step computes one new addend and moves the others on.
    uint32_t M[kPairs];
#pragma unroll
    for (int p = 0; p < kPairs; ++p) M[p] = kNeg2;
    const int mid_end = min(Wmin & ~3, c_end);
    int c = c_begin;
#pragma unroll 1
    for (int stop = c_begin == 0 ? kRows : c_begin;; stop = c_end) {
#pragma unroll 1
      for (; c < stop; c += 4) {
        const uint32_t res = next_letters(L);
#pragma unroll
        for (int k = 0; k < 4; ++k) {
#pragma unroll
          for (int p = kPairs - 1; p > 0; --p) M[p] = M[p - 1];
          const bool in = c + k < Wl;
          M[0] = (in ? 0u : kNeg2 & 0xFFFFu) | ((unsigned)(c + k - 9) < (unsigned)Wl ? 0u : kNeg2 & 0xFFFF0000u);
          sw_step<true>(R, residue(res, k), prof, in ? rp[k * stride] : 0u, k == 0 ? wp : rp + (k - 1) * stride, noc2,
                        nge2, M);
        }
        wp = rp + 3 * stride;
        rp = rp + 4 * stride == ring_end ? ring : rp + 4 * stride;
      }
      if (c == c_end) break;
#pragma unroll 1
      for (; c < mid_end; c += 4) {
        const uint32_t res = next_letters(L);
#pragma unroll
        for (int k = 0; k < 4; ++k)
          sw_step<false>(R, residue(res, k), prof, rp[k * stride], k == 0 ? wp : rp + (k - 1) * stride, noc2, nge2, M);
        wp = rp + 3 * stride;
        rp = rp + 4 * stride == ring_end ? ring : rp + 4 * stride;
      }
#pragma unroll
      for (int p = 0; p < kPairs; ++p) M[p] = 0;
    }
    // Ring words the next strip may read that this strip did not write: the
    // next strip's column x reads this strip's column x + 16.  Skipped columns
    // on the left hold dead cells, and so do those past the early stop, where
    // the next strip computes only off-matrix cells.
    for (int x = kRows - 1; x <= c_begin - 2; ++x) {
      int ls = base + x;
      ls = ls >= buf ? ls - buf : ls;
      ring[ls * stride] = 0;
    }
    if (c_end < W + kRows) {
      const int x_hi = min(W + kRows - 1, max(c_end - 1, 2 * kRows - 1));
      for (int x = c_end - 1; x <= x_hi; ++x) {
        int ls = base + x;
        ls = ls >= buf ? ls - buf : ls;
        ls = ls >= buf ? ls - buf : ls;
        ring[ls * stride] = 0;
      }
    }
    // this lane's column Wl + 15 is the next strip's column Wl - 1: outside
    // the band on the right.
    {
      int ls = base + Wl + kRows - 1;
      ls = ls >= buf ? ls - buf : ls;
      ls = ls >= buf ? ls - buf : ls;
      ring[ls * stride] = 0;
    }
    base += kRows;
    if (base >= buf) base -= buf;
    // strictly greater: the first strip holding the maximum keeps it
    const uint32_t m2 = max2(R.mx0, R.mx1);
    const int v = max(lo16(m2), hi16(m2));
    if (v > best) {
      best = v;
      best_i = i0 + kRows - 1;
    }
  }
  if (a.cells_eval) {
    const int lanes = __popc(__ballot_sync(0xFFFFFFFFu, active));
    if (lane == 0) {
      atomicAdd(a.cells_eval, (unsigned long long)(steps_done * kRows * lanes));
      atomicAdd(a.cells_eval + 2, (unsigned long long)(steps_done * kRows * 32));  // idle lanes included
    }
  }
  if (!active) return;
  a.score[bidx] = best;
  // transposed: the best cell's subject row i' <= best_i sits on query row
  // i' + d (d in [d0, d1]), so best_i + d1 bounds the reference's best row
  if (tr && best_i > 0) best_i = min((int)band.n, best_i + band.d1);
  if (a.best_row) a.best_row[bidx] = best_i;
}

template <int WARPS>
constexpr size_t class_smem(int max_width) {
  return 640 + WARPS * kParts * kProfBytes + (size_t)WARPS * 32 * ring_words(max_width) * 4;
}

template <int WARPS>
void launch_class(const SwScoreArgs& a, int max_width, cudaStream_t st) {
  if (a.task_hi <= a.task_lo) return;
  const int threads = WARPS * 32;
  const size_t smem = class_smem<WARPS>(max_width);
  // (classes 2 and 3 are the same kernel)
  allow_smem((const void*)k_sw<WARPS>, WARPS == 1 ? class_smem<1>(kSwC3) : smem);
  const int blocks = ceil_div((long long)(a.task_hi - a.task_lo), WARPS * kParts);
  count_launch();
  k_sw<WARPS><<<blocks, threads, smem, st>>>(a);
  DRG_CUDA(cudaGetLastError());
}

}  // namespace

void launch_sw_class(const SwScoreArgs& a, int cls, cudaStream_t st) {
  switch (cls) {
    case 0: launch_class<4>(a, kSwClassMax[0], st); break;
    case 1: launch_class<2>(a, kSwClassMax[1], st); break;
    case 2: launch_class<1>(a, kSwClassMax[2], st); break;
    default: launch_class<1>(a, kSwClassMax[3], st); break;
  }
}

}  // namespace drg
