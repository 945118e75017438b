// Banded affine Smith-Waterman, systolic: the traceback of the HSPs that
// survive the E-value gate and the exact score of the bands that the packed
// 16-bit kernels do not settle, in 32-bit lanes (gapped.rs:67-280); and, two
// bands per warp in 16-bit halves (k_sys_pair), the bands of the score pass
// that do not fill a warp of the packed kernel or would outlast it.
//
// What bounds these bands is the dependency chain of one band, not the chip:
// there are few of them (4,000 of 1.4M bands of a search of 1,000 queries) and
// some are long.  So a band is spread over the lanes of a warp with as few
// rows per lane as the band's width lets the lanes hold: a lane runs R rows
// (4, or 8 for wider bands) of one column per step, and the chain of a step
// is R cells and one shuffle.  In 32-bit lanes a cell needs no saturation
// rule, no minimum width and no exact re-run.
//
// Rotating kernel (k_sys_rot, W <= 151 with R = 4, W <= 271 with R = 8):
// strip s (rows rs + R s ...) runs on lane s mod 32 and starts at step
// (R + 1) s, one step behind the strip above it, whose last row's (H, E) it
// takes by a shuffle.  Relative column c = T - (R + 1) s of a strip covers
// subject column j = i0 - d1 + c, and row r is in the band for
// r <= c <= r + W - 1.  A cell outside is dead by an addend (kNegI) on all that
// flows into it, so its H is 0 and its E and F are near -inf.  Row r is
// outside in the column that row 0 was r columns earlier, so a lane computes
// one addend per column and keeps the last R + 1; its columns before the first
// are dead as well, which is the left edge of its rows and leaves the state
// that a strip starts from.
// Cells off the matrix need no mask: residues and rows there score -64, their
// H stays below the H it came from, and nothing flows from them to a matrix
// cell.  A strip's profile (R scores per residue, one word per lane and
// residue: conflict-free) is built by the whole warp one turn before it
// starts, from letters loaded 32 strips ahead.
//
// Block kernel (k_sys_block, any width): 8 warps, each running strips of 32
// lanes x 4 rows (128 rows) at absolute columns, lane l one column behind
// lane l - 1.  The warps advance in phases of 32 columns between block
// barriers; the strip below runs two phases behind the one above and reads
// its last row from a shared ring (from global memory where the strips wrap
// around the block), so no warp ever waits on a flag.
//
// Rows past m + d1 keep one cell in the reference, clamped to column m
// (gapped.rs:86-92): its diagonal is 0 and its E comes from cells above, so
// it can hold the best only with the score of its own pair.  Those rows are
// looked at only when the best of the others is at most the matrix's largest
// score, and their alignment is that one pair.
//
// In trace mode each step stores one word per lane, 32 consecutive words per
// step, with a nibble per row: whether a gap beat the diagonal, whether F beat
// E, and whether E and F extend a gap (gapped.rs:120-200).  Each is the sign
// of a difference, pushed into the word by one funnel shift.  Whether H is 0
// is not stored: the walk (gapped.rs:205-279) knows H along its way.  It takes
// up to 32 cells at a time: lane k reads the cell k steps back along the
// diagonal (or the gap), a scan of the pairs' scores gives H there, and a
// ballot finds where the run ends.  A band's best cell is the largest of one
// integer per column made of H, row and column.  A cell costs some nine ALU
// operations (27 with compares and selects for the masks, a stored choice of
// four and a maximum and column per row).
//
// Measured on one B200 (first figure: the form this replaces, 16 rows per
// lane in 16-bit pairs with a lane walking alone, and one thread per band
// where that form did not apply; second: with masks and choices):
//   traceback of 4 bands of a 497-aa query        415 -> 133 -> 106 us
//   of 26,597 bands (20,000 queries)             7394 -> 2250 -> 1440 us
//   of 4,182 bands (1,000 queries, sensitive)    1283 -> 530 -> 385 us, routes side by side
//   13 bands up to 2,000 x 4,000, scores    1,206,000 -> 1,140 -> 950 us
#include "kernels.h"
#include "smem_limit.h"
#include "sw_common.cuh"

namespace drg {

namespace {

constexpr int kNegI = -(1 << 29);
constexpr int kResidues = 26;  // 25 letters and the sentinel
constexpr int kRotWarpsPerBlock = 4;
constexpr int kBlkWarps = 8;
constexpr int kBlkR = 4;
constexpr int kBlkRows = 32 * kBlkR;  // rows of a strip of the block kernel
constexpr unsigned kAll = 0xFFFFFFFFu;

struct CellOut {
  int best, bi, bj;
};

__device__ __forceinline__ int score_byte(uint32_t w, int r) {  // sign-extended byte r
  int v;
  const uint32_t sel = (uint32_t)r | (8u | (uint32_t)r) << 4 | (8u | (uint32_t)r) << 8 | (8u | (uint32_t)r) << 12;
  asm("prmt.b32 %0, %1, %1, %2;" : "=r"(v) : "r"(w), "r"(sel));
  return v;
}

// mat[q * 32 + res]: scores by letter, the sentinel for q or res = 25.
__device__ __forceinline__ void stage_scores(int8_t* mat, const int8_t* scores625) {
  for (int i = threadIdx.x; i < kResidues * 32; i += blockDim.x) {
    const int q = i >> 5, r = i & 31;
    mat[i] = q < 25 && r < 25 ? scores625[q * 25 + r] : (int8_t)kSentinelScore;
  }
  __syncthreads();
}

// Adds the sign bit of x below the bits of v: one funnel shift.
__device__ __forceinline__ uint32_t push_sign(uint32_t v, int x) { return __funnelshift_l((uint32_t)x, v, 1); }

// R rows of one column.  up = (hu, eu): the row above row 0 at this column;
// hd: that row's H one column before.  dead(r): 0, or kNegI where row r is
// outside the band: its H is then 0, its E and F near -inf.  In trace mode
// returns a nibble per row, row 0's highest: f_ext << 3 | e_ext << 2 | (F > E)
// << 1 | (max(E, F) > D).
template <int R, bool TR, typename Dead>
__device__ __forceinline__ uint32_t column(int (&hl)[R], int (&f)[R], int hd, int& hu, int& eu, const uint32_t* w,
                                           int oc, int ge, Dead dead) {
  uint32_t nib = 0;
#pragma unroll
  for (int r = 0; r < R; ++r) {
    const int z = dead(r);
    const int te = eu + z - ge, to = hu + z - oc;
    const int tf = f[r] + z - ge, tfo = hl[r] + z - oc;
    const int e = max(te, to), fn = max(tf, tfo), g = max(e, fn);
    const int d = hd + score_byte(w[r >> 2], r & 3) + z;
    const int h = __vimax_s32_relu(d, g);
    if (TR) {
      nib = push_sign(nib, tfo - tf);
      nib = push_sign(nib, to - te);
      nib = push_sign(nib, e - fn);
      nib = push_sign(nib, d - g);
    }
    hd = hl[r];
    hl[r] = h;
    f[r] = fn;
    hu = h;
    eu = e;
  }
  return nib;
}

// The first row-major maximum over the warp: highest score, then lowest row
// (each row's column is its first).
__device__ __forceinline__ CellOut warp_best(CellOut b) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    const int s = __shfl_xor_sync(kAll, b.best, o), i = __shfl_xor_sync(kAll, b.bi, o),
              j = __shfl_xor_sync(kAll, b.bj, o);
    if (s > b.best || (s == b.best && i < b.bi)) {
      b.best = s;
      b.bi = i;
      b.bj = j;
    }
  }
  return b;
}

// Rows past m + d1 (see the head of the file): the first row with the largest
// score of its own pair, when that beats `b`.
__device__ __forceinline__ CellOut clamped_rows(CellOut b, const uint8_t* q, const uint8_t* s, int n, int m, int d1,
                                                const int8_t* mat) {
  const int lane = threadIdx.x & 31;
  const int64_t v0 = (int64_t)m + d1 + 1;
  CellOut v{0, 0x7FFFFFFF, m};
  const uint32_t sm = min((uint32_t)s[m - 1], 24u);
  for (int64_t i = (v0 > 1 ? v0 : 1) + lane; i <= n; i += 32) {
    const int sc = mat[min((uint32_t)q[i - 1], 24u) * 32 + sm];
    if (sc > v.best) {
      v.best = sc;
      v.bi = (int)i;
    }
  }
  v = warp_best(v);
  return v.best > b.best ? v : b;
}

// A record without an alignment: score 0, or -1, which the host reports as an
// internal error.
__device__ __forceinline__ void write_none(const SysArgs& a, uint32_t band, int score = 0) {
  ExactOut R;
  R.score = score;
  R.q_begin = R.q_end = R.s_begin = R.s_end = 0;
  R.identities = R.positives = R.mismatches = R.gap_openings = R.gaps = R.length = 0;
  R.n_ops = 0;
  R.cells = 0;
  a.out[band] = R;
}

// The walk of one band by a whole warp.  cell(i, j) is the nibble of a cell of
// the band with i >= 1 and j >= 1.  It ends where H is 0, and H is known along
// it: a pair's score less after a diagonal step, a gap's cost more after a gap.
// A best cell outside the matrix or the band (single: of a row past m + d1,
// which has one cell) cannot be, and is reported.
template <typename Cell>
__device__ __forceinline__ void walk_warp(const SysArgs& a, uint32_t band, const Band& b, int m, const CellOut& best,
                                          const int8_t* mat, bool single, Cell cell) {
  const int lane = threadIdx.x & 31;
  const uint8_t* q = a.q_letters + a.q_offsets[b.target] + b.q0;
  const uint8_t* s = a.s_letters + a.s_offsets[b.subject];
  const int n = (int)b.n;
  const int64_t d_best = (int64_t)best.bi - best.bj;
  if (best.bi < 1 || best.bi > n || best.bj < 1 || best.bj > m || (!single && (d_best < b.d0 || d_best > b.d1))) {
    if (lane == 0) write_none(a, band, -1);
    return;
  }
  uint32_t* ops = a.ops + a.ops_off[band];
  const uint32_t cap = (uint32_t)n + (uint32_t)m;  // op slots of the band
  int i = best.bi, j = best.bj;
  uint32_t nops = 0, length = 0, gaps = 0, openings = 0, matches = 0;
  uint32_t ident = 0, pos = 0;  // per lane, summed at the end
  uint32_t cur_op = 3, cur_cnt = 0;
  bool in_gap = false;
  int h = best.best;  // H of (i, j) in state 0
  // runs are found last to first: they fill the band's slots from the end
  auto emit = [&](uint32_t op, uint32_t cnt) {
    if (op == cur_op) {
      cur_cnt += cnt;
      return;
    }
    if (cur_cnt) {
      ++nops;
      if (lane == 0) ops[cap - nops] = (cur_cnt << 2) | cur_op;
    }
    cur_op = op;
    cur_cnt = cnt;
  };
  int state = 0;
  while (i > 0 && j > 0) {
    const int di = state == 2 ? 0 : lane, dj = state == 1 ? 0 : lane;
    const int ci = i - di, cj = j - dj;
    const int64_t d = (int64_t)ci - cj;
    const bool ok = single ? lane == 0 : ci > 0 && cj > 0 && d >= b.d0 && d <= b.d1;
    const uint32_t nb = !ok || single ? 0u : cell(ci, cj);
    if (__shfl_sync(kAll, (int)ok, 0) == 0) break;  // outside the row's range (gapped.rs:216)
    if (state == 0) {
      const uint32_t x = ok ? q[ci - 1] : 0u, y = ok ? s[cj - 1] : 0u;
      const int sc = mat[min(x, 24u) * 32 + min(y, 24u)];
      int sum = ok ? sc : 0;  // of this cell's pair and those before it
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const int v = __shfl_up_sync(kAll, sum, o);
        if (lane >= o) sum += v;
      }
      // a run ends before a cell whose H is 0 or came from a gap
      const uint32_t stop = __ballot_sync(kAll, !ok || (nb & 1u) != 0 || h - (sum - sc) <= 0);
      const uint32_t run = stop ? (uint32_t)__ffs(stop) - 1u : 32u;
      if (run == 0) {
        if (h <= 0) break;
        state = (__shfl_sync(kAll, nb, 0) & 2u) ? 2 : 1;
        continue;
      }
      if ((uint32_t)lane < run) {
        ident += x == y;
        pos += sc > 0;
      }
      emit(0, run);
      matches += run;
      length += run;
      in_gap = false;
      h -= __shfl_sync(kAll, sum, (int)run - 1);
      i -= (int)run;
      j -= (int)run;
      if (single) break;  // a row past m + d1 holds one cell
    } else {
      // an op per cell up to the first whose extension bit is clear
      const uint32_t bit = state == 1 ? 4u : 8u;
      const uint32_t open = __ballot_sync(kAll, (nb & bit) == 0u);
      const uint32_t bad = __ballot_sync(kAll, !ok);
      uint32_t run = open ? (uint32_t)__ffs(open) : 32u;
      if (bad) run = min(run, (uint32_t)__ffs(bad) - 1u);
      emit(state == 1 ? 1u : 2u, run);
      length += run;
      gaps += run;
      if (!in_gap) ++openings;
      in_gap = true;
      h += (int)run * a.ge + (open ? a.oc - a.ge : 0);
      if (state == 1) i -= (int)run;
      else j -= (int)run;
      if (open) state = 0;
    }
  }
  emit(3, 0);  // the last run
  ident = __reduce_add_sync(kAll, ident);
  pos = __reduce_add_sync(kAll, pos);
  __syncwarp();
  if (nops < cap) {
    for (uint32_t k0 = 0; k0 < nops; k0 += 32) {  // ascending, every chunk read before it is written over
      const uint32_t k = k0 + lane;
      const uint32_t v = k < nops ? ops[cap - nops + k] : 0u;
      __syncwarp();
      if (k < nops) ops[k] = v;
      __syncwarp();
    }
  }
  if (lane == 0) {
    ExactOut R;
    R.score = best.best;
    R.q_begin = (uint32_t)i;
    R.q_end = (uint32_t)best.bi;
    R.s_begin = (uint32_t)j;
    R.s_end = (uint32_t)best.bj;
    R.identities = ident;
    R.positives = pos;
    R.mismatches = matches - ident;
    R.gap_openings = openings;
    R.gaps = gaps;
    R.length = length;
    R.n_ops = nops;
    R.cells = 0;
    a.out[band] = R;
  }
}

// Job t's trace.
__device__ __forceinline__ uint8_t* sys_trace(const SysArgs& a, uint64_t t) {
  return a.trace + (a.jobs[t].trace_off - a.trace_base);
}

template <int R>
struct TraceWord {
  typedef uint16_t T;  // 4 rows
};
template <>
struct TraceWord<8> {
  typedef uint32_t T;
};

// ---- rotating strips: one warp per band ---------------------------------------
template <int R, bool TR>
__global__ void __launch_bounds__(kRotWarpsPerBlock * 32) k_sys_rot(SysArgs a) {
  constexpr int kLag = R + 1, kWords = R / 4;
  typedef typename TraceWord<R>::T Word;
  __shared__ int8_t mat[kResidues * 32];
  __shared__ uint32_t prof_all[kRotWarpsPerBlock][kWords][kResidues * 32];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  stage_scores(mat, a.scores625);
  uint32_t(*prof)[kResidues * 32] = prof_all[warp];
  const uint64_t n_jobs = a.d_count ? (uint64_t)*a.d_count : a.hi;
  const uint64_t step_jobs = (uint64_t)gridDim.x * kRotWarpsPerBlock;
  for (uint64_t t = a.lo + (uint64_t)blockIdx.x * kRotWarpsPerBlock + warp; t < n_jobs; t += step_jobs) {
    const uint32_t band = TR ? a.jobs[t].band : a.list[t];
    const Band b = a.bands[band];
    const uint8_t* q = a.q_letters + a.q_offsets[b.target] + b.q0;
    const uint8_t* sl = a.s_letters + a.s_offsets[b.subject];
    const int m = (int)(a.s_offsets[b.subject + 1] - a.s_offsets[b.subject]);
    const int n = (int)b.n;
    const SysGeom g = sys_geom(b, m, TR);
    const int W = g.d1 - g.d0 + 1;
    const int S = g.rows > 0 ? (g.rows + R - 1) / R : 0;
    const int turns = sys_rot_turns(S, W, R);
    Word* tr = TR ? reinterpret_cast<Word*>(sys_trace(a, t)) + lane : nullptr;
    int hl[R], f[R];
    int out[kLag];  // per column of the last R + 1: kNegI where the strip's first row is outside its band
    // the strip's maximum; in trace mode with its place, the first row-major
    // one the largest: (H * R + R - 1 - row) * 512 + 511 - column
    uint32_t top = 0;
#pragma unroll
    for (int r = 0; r < R; ++r) {
      hl[r] = 0;
      f[r] = kNegI;
    }
#pragma unroll
    for (int u = 0; u < kLag; ++u) out[u] = kNegI;
    CellOut best{0, 0x7FFFFFFF, 0};
    int s = lane;                    // this lane's strip
    int c = -kLag * lane;            // its column at the coming step
    unsigned width = s < S ? W : 0;  // columns [0, width) are in its first row's band
    int p = g.rs - g.d1 - 1 - lane;  // subject index of that column
    auto letter = [&](int x) -> uint32_t {
      return (unsigned)x < (unsigned)m ? min((uint32_t)__ldg(sl + x), 24u) : (uint32_t)kSentinel;
    };
    // the R query letters of strip k (32 strips at a time, lane x holds k0 + x)
    auto load_rows = [&](int k, uint32_t (&v)[kWords]) {
#pragma unroll
      for (int w = 0; w < kWords; ++w) {
        uint32_t x = 0;
#pragma unroll
        for (int r = 0; r < 4; ++r) {
          const int64_t i = (int64_t)g.rs + (int64_t)R * k + 4 * w + r;
          x |= (k < S && i <= n ? min((uint32_t)__ldg(q + i - 1), 24u) : (uint32_t)kSentinel) << (8 * r);
        }
        v[w] = x;
      }
    };
    uint32_t qv[kWords], qn[kWords];
    load_rows(lane, qv);
    load_rows(32 + lane, qn);
    auto build = [&](int k) {  // the profile of strip k, for lane k mod 32
#pragma unroll
      for (int w = 0; w < kWords; ++w) {
        const uint32_t ql = __shfl_sync(kAll, qv[w], k & 31);
        uint32_t x = 0;
#pragma unroll
        for (int r = 0; r < 4; ++r)
          x |= (uint32_t)(uint8_t)mat[((ql >> (8 * r)) & 0xFFu) * 32 + lane] << (8 * r);
        if (lane < kResidues) prof[w][lane * 32 + (k & 31)] = x;
      }
    };
    // fold the finished strip's maximum into the lane's best
    auto fold = [&]() {
      const int h = (int)(TR ? top / (512 * R) : top);
      if (h > best.best) {
        const int row = TR ? R - 1 - (int)(top / 512 % R) : R - 1;  // score mode: a bound of the best's row
        best.best = h;
        best.bi = g.rs + R * s + row;
        best.bj = g.rs + R * s - g.d1 + 511 - (int)(top % 512);
      }
      top = 0;
    };
    __syncwarp();
    if (S > 0) build(0);
    __syncwarp();
    uint32_t l0 = letter(p), l1 = letter(p + 1);  // letters of this step's and the next step's columns
    uint32_t wn[kWords];
#pragma unroll
    for (int w = 0; w < kWords; ++w) wn[w] = prof[w][l0 * 32 + lane];
    int hup = 0, h_out = 0, e_out = kNegI;
    const int src = (lane + 31) & 31;
    for (int k = 0; k < turns; ++k) {
      // strip k starts now on lane k mod 32; strip k + 1 gets its lane and profile
      if (((k + 1) & 31) == 0) {
#pragma unroll
        for (int w = 0; w < kWords; ++w) qv[w] = qn[w];
        load_rows(k + 33 + lane, qn);
      }
      if (k + 1 < S) build(k + 1);
      if (k >= 31 && lane == ((k + 1) & 31)) {
        fold();
        s += 32;
        c -= 32 * kLag;
        p -= 32;
        if (s >= S) width = 0;
      }
      // (the R + 1 dead columns before a strip leave H = 0 and F near -inf)
      if (lane == (k & 31)) top = 0;
      __syncwarp();
#pragma unroll
      for (int u = 0; u < kLag; ++u) {
        // (strip 0 has lane 31 above it, which is dead until its first strip)
        int hu = __shfl_sync(kAll, h_out, src), eu = __shfl_sync(kAll, e_out, src);
        out[u] = (unsigned)c < width ? 0 : kNegI;
        uint32_t w[kWords];
#pragma unroll
        for (int x = 0; x < kWords; ++x) {
          w[x] = wn[x];
          wn[x] = prof[x][l1 * 32 + lane];
        }
        l1 = letter(p + 2);
        const int hd = hup;
        hup = hu;
        const uint32_t nib = column<R, TR>(hl, f, hd, hu, eu, w, a.oc, a.ge,
                                           [&](int r) { return out[(u - r + kLag) % kLag]; });
        h_out = hu;
        e_out = eu;
        if (TR) {
          *tr = (Word)nib;
          tr += 32;
          uint32_t t = 0;
#pragma unroll
          for (int r = 0; r < R; r += 2)
            t = __vimax3_u32(t, (uint32_t)hl[r] * R + (R - 1 - r), (uint32_t)hl[r + 1] * R + (R - 2 - r));
          top = max(top, t * 512u + (uint32_t)(511 - c));
        } else {
#pragma unroll
          for (int r = 0; r < R; r += 2) top = __vimax3_u32(top, (uint32_t)hl[r], (uint32_t)hl[r + 1]);
        }
        ++c;
        ++p;
      }
    }
    if (s < S) fold();
    best = warp_best(best);
    bool single = false;
    if (best.best < a.exact_below && n > 0 && m > 0) {
      const CellOut v = clamped_rows(best, q, sl, n, m, b.d1, mat);
      single = v.best > best.best;
      best = v;
    }
    if (!TR) {
      if (lane == 0) {
        a.score[band] = best.best;
        if (a.best_row) a.best_row[band] = best.best > 0 ? min(best.bi, n) : 0;
      }
    } else if (best.best == 0) {
      if (lane == 0) write_none(a, band);
    } else {
      __syncwarp();
      const Word* base = reinterpret_cast<const Word*>(sys_trace(a, t));
      walk_warp(a, band, b, m, best, mat, single, [&](int i, int j) -> uint32_t {
        const int ii = i - g.rs, sk = ii / R, r = ii % R;
        const int cc = j - (g.rs + R * sk - g.d1);
        return ((uint32_t)base[(int64_t)(cc + kLag * sk) * 32 + (sk & 31)] >> (4 * (R - 1 - r))) & 15u;
      });
    }
    __syncwarp();
  }
}

// ---- rotating strips, two bands per warp (score pass) ----------------------------
// The same strips with a band in each 16-bit half: lane and step of a strip
// depend on its number only, so two bands run in step, each with its own
// letters, profile and right edge.  Jobs are sorted by route and length, so
// that a pair's bands end together.  For bands whose best stays below 2^15
// (the packed kernels' bound).
// E and F are kept with the open cost added back (E' = max(E' - ge, H) above,
// F' = max(F' - ge, H) to the left, H = max(0, D, E' - oc, F' - oc): all at
// least 0).  Outside the band no cell is masked after it is computed: an
// addend of -16384 on D and on the open cost makes its H 0 below 16384 + oc.
// Scores go up to 31743, so a cell beside the band may keep an H of up to some
// 15300.  That changes no score: a path that turns outside the band pays 16384
// for it, again for each further cell there that it aligns or turns at and for
// each strip that its E' leaves (e_out), and comes back at most R rows below
// where it left, which a path inside reaches for some R mismatches.  Row r is
// outside in the column that row 0 was r columns earlier, so a lane computes
// one addend per column and keeps the last R + 1; a strip starts with all of
// them dead, which is its left edge; and the E' that a strip hands down is dead
// with its last row.  A cell is five ALU operations, half a three-input
// maximum and three adds on the FMA pipe, which runs beside (ten ALU
// operations with masks on E and H and selects for the left edge: 22 bands of
// a 497-aa query 141 -> 129 us, the widest route of 1,000 queries very
// sensitive 4,620 -> 3,100 us, of 13 queries ultra-sensitive 2,160 -> 1,600
// us).
// All 32 lanes run whatever the width, so a band takes the fewest rows per lane
// that hold it: 4, 6, 8, 12 or 16, the widths up to 151, 211, 271, 391 and 511
// (with 4, 8 and 16 alone: 26.3 ms for 1,000 queries very sensitive, whose
// wide bands are mostly 250 to 350 columns; 25.7 with all five).  24 and 32
// rows, up to 991 columns, were slower than a warp per band (sw_band.cu): a
// step is then too long a chain (13 queries, ultra-sensitive: 6.9 against 6.6
// ms).
using sw::add2;
using sw::pick_sel;
using sw::prmt;

constexpr uint32_t kDead2 = 0xC000C000u;  // (-16384, -16384)

template <int R>
constexpr size_t pair_smem() {
  return (size_t)kRotWarpsPerBlock * 2 * ((R + 3) / 4) * kResidues * 32 * sizeof(uint32_t);
}

template <int R>
__global__ void __launch_bounds__(kRotWarpsPerBlock * 32) k_sys_pair(SwBandArgs a) {
  constexpr int kLag = R + 1, kWords = (R + 3) / 4;
  extern __shared__ __align__(16) uint32_t pair_prof[];
  __shared__ int8_t mat[kResidues * 32];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  stage_scores(mat, a.scores625);
  const uint64_t t0 = a.lo + 2 * ((uint64_t)blockIdx.x * kRotWarpsPerBlock + warp);
  if (t0 >= a.hi) return;  // warp-uniform
  uint32_t* prof = pair_prof + (size_t)warp * 2 * kWords * kResidues * 32;  // [half][word][residue][lane]
  // per half: geometry and letters (an odd last job runs twice, written once)
  SysGeom g[2];
  uint32_t band[2];
  const uint8_t *q[2], *sl[2];
  int n[2], m[2], W[2], S[2];
  int turns = 0;
#pragma unroll
  for (int x = 0; x < 2; ++x) {
    band[x] = a.jobs[t0 + x < a.hi ? t0 + x : t0].band;
    const Band b = a.bands[band[x]];
    q[x] = a.q_letters + a.q_offsets[b.target] + b.q0;
    sl[x] = a.s_letters + a.s_offsets[b.subject];
    m[x] = (int)(a.s_offsets[b.subject + 1] - a.s_offsets[b.subject]);
    n[x] = (int)b.n;
    g[x] = sys_geom(b, m[x], false);
    W[x] = g[x].d1 - g[x].d0 + 1;
    S[x] = g[x].rows > 0 ? (g[x].rows + R - 1) / R : 0;
    turns = max(turns, sys_rot_turns(S[x], W[x], R));
  }
  const uint32_t noc2 = (uint32_t)(uint16_t)(-(a.gap_open + a.gap_extend)) * 0x10001u;
  const uint32_t nge2 = (uint32_t)(uint16_t)(-a.gap_extend) * 0x10001u;
  uint32_t hl[R], f[R];  // H of the last column, F' of this one
  uint32_t out[kLag];    // per column of the last R + 1: kDead2 where a strip's first row is outside its band
  uint32_t top = 0;
#pragma unroll
  for (int r = 0; r < R; ++r) {
    hl[r] = 0;
    f[r] = 0;
  }
#pragma unroll
  for (int u = 0; u < kLag; ++u) out[u] = kDead2;
  int best[2] = {0, 0}, bi[2] = {0x7FFFFFFF, 0x7FFFFFFF};
  int s = lane;
  // per half: column past the right end of the first row's band, c - (W - 1);
  // kPast (dead throughout) of a lane without a strip, or before its strip
  // starts: what it passes on then reaches the strip of 32 before
  constexpr uint32_t kPast = 0x3FFF;
  uint32_t cw2 = kPast | kPast << 16;
  int p[2] = {g[0].rs - g[0].d1 - 1 - lane, g[1].rs - g[1].d1 - 1 - lane};
  auto letter = [&](int x, int at) -> uint32_t {
    return (unsigned)at < (unsigned)m[x] ? (uint32_t)__ldg(sl[x] + at) : (uint32_t)kSentinel;
  };
  auto load_rows = [&](int x, int k, uint32_t (&v)[kWords]) {
#pragma unroll
    for (int w = 0; w < kWords; ++w) {
      uint32_t y = 0;
#pragma unroll
      for (int r = 0; r < 4; ++r) {
        const int64_t i = (int64_t)g[x].rs + (int64_t)R * k + 4 * w + r;
        y |= (k < S[x] && i <= n[x] ? min((uint32_t)__ldg(q[x] + i - 1), 24u) : (uint32_t)kSentinel) << (8 * r);
      }
      v[w] = y;
    }
  };
  uint32_t qv[2][kWords], qn[2][kWords];
#pragma unroll
  for (int x = 0; x < 2; ++x) {
    load_rows(x, lane, qv[x]);
    load_rows(x, 32 + lane, qn[x]);
  }
  auto build = [&](int k) {
#pragma unroll
    for (int x = 0; x < 2; ++x) {
#pragma unroll
      for (int w = 0; w < kWords; ++w) {
        const uint32_t ql = __shfl_sync(kAll, qv[x][w], k & 31);
        uint32_t y = 0;
#pragma unroll
        for (int r = 0; r < 4; ++r) y |= (uint32_t)(uint8_t)mat[((ql >> (8 * r)) & 0xFFu) * 32 + lane] << (8 * r);
        if (lane < kResidues) prof[((x * kWords + w) * kResidues + lane) * 32 + (k & 31)] = y;
      }
    }
  };
  auto fold = [&]() {
    const int t2[2] = {(int)(top & 0xFFFFu), (int)(top >> 16)};
#pragma unroll
    for (int x = 0; x < 2; ++x) {
      if (t2[x] > best[x]) {
        best[x] = t2[x];
        bi[x] = g[x].rs + R * s + R - 1;  // a bound of the best's row
      }
    }
    top = 0;
  };
  __syncwarp();
  build(0);
  __syncwarp();
  uint32_t l1[2], wn[2][kWords];
#pragma unroll
  for (int x = 0; x < 2; ++x) {
    const uint32_t l0 = letter(x, p[x]);
    l1[x] = letter(x, p[x] + 1);
#pragma unroll
    for (int w = 0; w < kWords; ++w) wn[x][w] = prof[((x * kWords + w) * kResidues + l0) * 32 + lane];
  }
  uint32_t hup = 0, h_out = 0, e_out = 0;
  const int src = (lane + 31) & 31;
  for (int k = 0; k < turns; ++k) {
    if (((k + 1) & 31) == 0) {
#pragma unroll
      for (int x = 0; x < 2; ++x) {
#pragma unroll
        for (int w = 0; w < kWords; ++w) qv[x][w] = qn[x][w];
        load_rows(x, k + 33 + lane, qn[x]);
      }
    }
    if (k + 1 < max(S[0], S[1])) build(k + 1);
    if (k >= 31 && lane == ((k + 1) & 31)) {
      fold();
      s += 32;
      p[0] -= 32;
      p[1] -= 32;
      cw2 = kPast | kPast << 16;
    }
    const bool starts = lane == (k & 31);
    if (starts) {
      top = 0;
      cw2 = (s < S[0] ? (uint32_t)(uint16_t)(1 - W[0]) : kPast) | (s < S[1] ? (uint32_t)(uint16_t)(1 - W[1]) : kPast) << 16;
#pragma unroll
      for (int r = 0; r < R; ++r) {
        hl[r] = 0;
        f[r] = 0;
      }
    }
    __syncwarp();
#pragma unroll
    for (int u = 0; u < kLag; ++u) {
      // cw > 0: right of the first row's band
      out[u] = ~prmt(add2(cw2, 0xFFFFFFFFu), 0u, 0xBB99u) & kDead2;
      // (strip 0 has lane 31 above it, which is dead until its first strip)
      uint32_t hu = __shfl_sync(kAll, h_out, src), eu = __shfl_sync(kAll, e_out, src);
      uint32_t w[2][kWords];
#pragma unroll
      for (int x = 0; x < 2; ++x) {
#pragma unroll
        for (int y = 0; y < kWords; ++y) {
          w[x][y] = wn[x][y];
          wn[x][y] = prof[((x * kWords + y) * kResidues + l1[x]) * 32 + lane];
        }
        l1[x] = letter(x, p[x] + 2);
      }
      uint32_t hd = hup;
      hup = hu;
      uint32_t h_even = 0;
#pragma unroll
      for (int r = 0; r < R; ++r) {
        const uint32_t sc = prmt(w[0][r >> 2], w[1][r >> 2], pick_sel(r & 3));
        const uint32_t dead = out[(u - r + kLag) % kLag];
        const uint32_t no = add2(noc2, dead);
        const uint32_t e = __viaddmax_s16x2(eu, nge2, hu);
        const uint32_t h = __viaddmax_s16x2(e, no, __viaddmax_s16x2_relu(f[r], no, add2(hd, add2(sc, dead))));
        hd = hl[r];
        hl[r] = h;
        f[r] = __viaddmax_s16x2(f[r], nge2, h);
        hu = h;
        eu = e;
        if (r & 1) top = __vimax3_s16x2(top, h_even, h);
        h_even = h;
      }
      h_out = hu;
      e_out = add2(eu, out[(u + 2) % kLag]);  // of row R - 1
      cw2 = add2(cw2, 0x00010001u);
      ++p[0];
      ++p[1];
    }
  }
  fold();
#pragma unroll
  for (int x = 0; x < 2; ++x) {
    const CellOut b = warp_best(CellOut{best[x], bi[x], 0});
    if (lane == 0 && t0 + x < a.hi) {
      a.score[band[x]] = b.best;
      if (a.best_row) a.best_row[band[x]] = b.best > 0 ? min(b.bi, n[x]) : 0;
    }
  }
}

// ---- any width: one block per band ----------------------------------------------
template <bool TR>
__global__ void __launch_bounds__(kBlkWarps * 32) k_sys_block(SysArgs a) {
  constexpr int R = kBlkR;
  __shared__ int8_t mat[kResidues * 32];
  __shared__ uint32_t prof_all[kBlkWarps][kResidues * 32];
  __shared__ int2 ring[kBlkWarps][128];  // last row of a warp's strip, columns modulo 128
  __shared__ int2 above[kBlkWarps][32];  // the row above lane 0, this phase's columns
  __shared__ CellOut bests[kBlkWarps];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  stage_scores(mat, a.scores625);
  uint32_t* prof = prof_all[warp];
  int2* wrap = a.wrap + (uint64_t)blockIdx.x * a.wrap_words;  // the last warp's last row, by column
  const uint64_t n_jobs = a.d_count ? (uint64_t)*a.d_count : a.hi;
  for (uint64_t t = a.lo + blockIdx.x; t < n_jobs; t += gridDim.x) {
    const uint32_t band = TR ? a.jobs[t].band : a.list[t];
    const Band b = a.bands[band];
    const uint8_t* q = a.q_letters + a.q_offsets[b.target] + b.q0;
    const uint8_t* sl = a.s_letters + a.s_offsets[b.subject];
    const int m = (int)(a.s_offsets[b.subject + 1] - a.s_offsets[b.subject]);
    const int n = (int)b.n;
    const SysGeom g = sys_geom(b, m, TR);
    const int W = g.d1 - g.d0 + 1;
    const int S = g.rows > 0 ? (g.rows + kBlkRows - 1) / kBlkRows : 0;
    const SysBlockPlan plan = sys_block_plan(g, m);
    uint16_t* tr = TR ? reinterpret_cast<uint16_t*>(sys_trace(a, t)) : nullptr;
    int hl[R], f[R], rowmax[R], rowcol[R];
    int out[R] = {};  // of the last R columns: kNegI where the lane's first row is outside its band
    CellOut best{0, 0x7FFFFFFF, 0};
    int hup = 0, h_out = 0, e_out = kNegI;
    int s = warp, turn = 0;  // this warp's strip
    auto fold = [&](int i0) {
#pragma unroll
      for (int r = 0; r < R; ++r) {
        if (rowmax[r] > best.best) {
          best.best = rowmax[r];
          best.bi = i0 + r;
          best.bj = rowcol[r];
        }
      }
    };
    const int p_first = S > 0 ? plan.b0(g, 0) : 0;
    const int p_last = S > 0 ? 2 * ((S - 1) % kBlkWarps) + (S - 1) / kBlkWarps * plan.stride + plan.b1(g, m, S - 1) : -1;
    for (int ph = p_first; ph <= p_last; ++ph) {
      if (s < S) {
        const int B = ph - (2 * warp + turn * plan.stride);
        const int i0 = g.rs + kBlkRows * s;
        const int il = i0 + R * lane;  // this lane's first row
        const int b0 = plan.b0(g, s), b1 = plan.b1(g, m, s);
        if (B == b0) {  // the strip starts: profile and state
          uint32_t ql[R];
#pragma unroll
          for (int r = 0; r < R; ++r) ql[r] = (int64_t)il + r <= n ? min((uint32_t)__ldg(q + il + r - 1), 24u) : 25u;
          for (int res = 0; res < kResidues; ++res) {
            uint32_t x = 0;
#pragma unroll
            for (int r = 0; r < R; ++r) x |= (uint32_t)(uint8_t)mat[ql[r] * 32 + res] << (8 * r);
            prof[res * 32 + lane] = x;
          }
#pragma unroll
          for (int r = 0; r < R; ++r) {
            hl[r] = 0;
            f[r] = kNegI;
            rowmax[r] = rowcol[r] = 0;
            out[r] = (unsigned)(32 * B - lane - (il - g.d1) - (R - r)) < (unsigned)W ? 0 : kNegI;
          }
          hup = 0;
          h_out = 0;
          e_out = kNegI;
        }
        if (B >= b0 && B <= b1) {
          {  // the row above: columns [lo, hi] of row i0 - 1, else nothing flows in
            const int j = 32 * B + lane;
            const int lo = max(1, i0 - 1 - g.d1), hi = min(m, i0 - 1 - g.d0);
            int2 v = make_int2(0, kNegI);
            if (s > 0 && j >= lo && j <= hi) v = warp > 0 ? ring[warp - 1][j & 127] : wrap[j];
            above[warp][lane] = v;
          }
          __syncwarp();
          int j = 32 * B - lane;           // this lane's column
          int c = j - (il - g.d1);         // relative to its first row's band
          uint32_t l0 = (unsigned)(j - 1) < (unsigned)m ? min((uint32_t)__ldg(sl + j - 1), 24u) : (uint32_t)kSentinel;
          uint16_t* trp = TR ? tr + ((uint64_t)(s * (int64_t)plan.nb + (B - b0)) * 32) * 32 + lane : nullptr;
#pragma unroll 4
          for (int x = 0; x < 32; ++x) {
            int hu = __shfl_up_sync(kAll, h_out, 1), eu = __shfl_up_sync(kAll, e_out, 1);
            const int2 av = above[warp][x];
            if (lane == 0) {
              hu = av.x;
              eu = av.y;
            }
            const uint32_t w = prof[l0 * 32 + lane];
            l0 = (unsigned)j < (unsigned)m ? min((uint32_t)__ldg(sl + j), 24u) : (uint32_t)kSentinel;
            const int hd = hup;
            hup = hu;
            out[x % R] = (unsigned)c < (unsigned)W ? 0 : kNegI;
            const uint32_t nib = column<R, TR>(hl, f, hd, hu, eu, &w, a.oc, a.ge,
                                               [&](int r) { return out[(x - r + R) % R]; });
            h_out = hu;
            e_out = eu;
#pragma unroll
            for (int r = 0; r < R; ++r) {
              if (hl[r] > rowmax[r]) {
                rowmax[r] = hl[r];
                rowcol[r] = j;
              }
            }
            if (TR) {
              *trp = (uint16_t)nib;
              trp += 32;
            }
            if (lane == 31 && j >= 1 && j <= m) {
              if (warp < kBlkWarps - 1) ring[warp][j & 127] = make_int2(h_out, e_out);
              else wrap[j] = make_int2(h_out, e_out);
            }
            ++j;
            ++c;
          }
          if (B == b1) {
            fold(il);
            s += kBlkWarps;
            ++turn;
          }
        }
      }
      __syncthreads();
    }
    best = warp_best(best);
    if (lane == 0) bests[warp] = best;
    __syncthreads();
    if (warp == 0) {
      best = lane < kBlkWarps ? bests[lane] : CellOut{0, 0x7FFFFFFF, 0};
      best = warp_best(best);
      bool single = false;
      if (best.best < a.exact_below && n > 0 && m > 0) {
        const CellOut v = clamped_rows(best, q, sl, n, m, b.d1, mat);
        single = v.best > best.best;
        best = v;
      }
      if (!TR) {
        if (lane == 0) {
          a.score[band] = best.best;
          if (a.best_row) a.best_row[band] = best.best > 0 ? best.bi : 0;
        }
      } else if (best.best == 0) {
        if (lane == 0) write_none(a, band);
      } else {
        walk_warp(a, band, b, m, best, mat, single, [&](int i, int j) -> uint32_t {
          const int ii = i - g.rs, sk = ii / kBlkRows, ln = (ii / R) & 31, r = ii % R;
          const int j0 = j + ln;  // lane 0's column when lane ln was at j
          const int64_t at = (int64_t)sk * plan.nb + ((j0 >> 5) - plan.b0(g, sk));
          return ((uint32_t)tr[(at * 32 + (j0 & 31)) * 32 + ln] >> (4 * (R - 1 - r))) & 15u;
        });
      }
    }
    __syncthreads();  // bests, rings and the wrap row are free for the next band
  }
}

// Blocks for n bands of the block kernel: each has a wrap row.
unsigned block_grid(const SysArgs& a, uint64_t n) { return (unsigned)(n < a.wrap_blocks ? n : a.wrap_blocks); }

}  // namespace

// Bands that the packed score kernels did not settle (k_sys_lists): one warp
// each up to 151 wide, one block each above.  The counts stay on the device:
// the grids are at most one wave.
void launch_sys_score(SysArgs a, int route, uint64_t n_max, cudaStream_t st) {
  if (n_max == 0) return;
  count_launch();
  if (route == 0) {
    const uint64_t blocks = (n_max + kRotWarpsPerBlock - 1) / kRotWarpsPerBlock;
    k_sys_rot<4, false><<<(unsigned)(blocks < 148 * 8 ? blocks : 148 * 8), kRotWarpsPerBlock * 32, 0, st>>>(a);
  } else {
    k_sys_block<false><<<block_grid(a, n_max), kBlkWarps * 32, 0, st>>>(a);
  }
  DRG_CUDA(cudaGetLastError());
}

template <int R>
static void launch_pair(const SwBandArgs& a, cudaStream_t st) {
  allow_smem((const void*)k_sys_pair<R>, pair_smem<R>());
  const uint64_t warps = (a.hi - a.lo + 1) / 2;
  count_launch();
  k_sys_pair<R><<<(unsigned)((warps + kRotWarpsPerBlock - 1) / kRotWarpsPerBlock), kRotWarpsPerBlock * 32,
                  pair_smem<R>(), st>>>(a);
  DRG_CUDA(cudaGetLastError());
}

void launch_sw_band_route(const SwBandArgs& a, int route, int max_width, cudaStream_t st) {
  if (a.hi <= a.lo) return;
  switch (route) {
    case 0: launch_pair<pair_rows(0)>(a, st); break;
    case 1: launch_pair<pair_rows(1)>(a, st); break;
    case 2: launch_pair<pair_rows(2)>(a, st); break;
    case 3: launch_pair<pair_rows(3)>(a, st); break;
    case 4: launch_pair<pair_rows(4)>(a, st); break;
    default: launch_sw_band(a, max_width, st); break;
  }
}

void launch_sys_trace(SysArgs a, int route, cudaStream_t st) {
  if (a.hi <= a.lo) return;
  const uint64_t n = a.hi - a.lo;
  const uint64_t blocks = (n + kRotWarpsPerBlock - 1) / kRotWarpsPerBlock;
  count_launch();
  switch (route) {
    case 0: k_sys_rot<4, true><<<(unsigned)blocks, kRotWarpsPerBlock * 32, 0, st>>>(a); break;
    case 1: k_sys_rot<8, true><<<(unsigned)blocks, kRotWarpsPerBlock * 32, 0, st>>>(a); break;
    default: k_sys_block<true><<<block_grid(a, n), kBlkWarps * 32, 0, st>>>(a); break;
  }
  DRG_CUDA(cudaGetLastError());
}

}  // namespace drg
