// blastx front end on the device: six-frame translation, short-ORF masking
// and the drop of frames without a real residue (translate.rs:54-137,
// workflow.rs:112-127).
//
// Layout: reads are the FASTA records' upper-cased bytes back to back with
// u64 offsets.  One warp per (read, frame) translates its frame into a
// scratch buffer at an offset fixed by the frame's length alone
// ((L - offset) / 3 codons), masks the stop-free stretches shorter than the
// read's minimum ORF length in place, and flags the frame when a letter
// below X survives.  The kept frames are then compacted, in (read, frame)
// order, into the target batch layout the search takes.
#include <algorithm>

#include "kernels.h"

namespace drg {

namespace {

constexpr int kFrameWarps = 8;          // warps per block, one frame each at a time
constexpr uint8_t kXLetterDev = 23;     // alphabet.rs X_LETTER
constexpr uint8_t kStopLetterDev = 24;  // alphabet.rs STOP_LETTER

// translate.rs:15-23: T/U 0, C 1, A 2, G 3, anything else 4 (lower case too)
__device__ __forceinline__ uint32_t base_of(uint8_t b) {
  switch (b) {
    case 'T': case 't': case 'U': case 'u': return 0;
    case 'C': case 'c': return 1;
    case 'A': case 'a': return 2;
    case 'G': case 'g': return 3;
    default: return 4;
  }
}
// translate.rs:25-45: complement of the upper-case IUPAC codes; other bytes
// (S, W, N, lower case, ...) stay as they are
__device__ __forceinline__ uint8_t complement_of(uint8_t b) {
  switch (b) {
    case 'A': return 'T';
    case 'T': return 'A';
    case 'C': return 'G';
    case 'G': return 'C';
    case 'U': return 'A';
    case 'R': return 'Y';
    case 'Y': return 'R';
    case 'K': return 'M';
    case 'M': return 'K';
    case 'B': return 'V';
    case 'V': return 'B';
    case 'D': return 'H';
    case 'H': return 'D';
    default: return b;
  }
}

// The standard genetic code (TCAG order) as letter codes, built per block
// from the one-letter table: alphabet index of each codon's amino acid.
__device__ __forceinline__ void stage_codons(uint8_t* codon) {
  const char* code = "FFLLSSSSYY**CC*WLLLLPPPPHHQQRRRRIIIMTTTTNNKKSSRRVVVVAAAADDEEGGGG";
  const char* alphabet = "ARNDCQEGHILKMFPSTWYVBJZX*";
  for (int i = threadIdx.x; i < 64; i += blockDim.x) {
    uint8_t v = kXLetterDev;
    for (int k = 0; k < 25; ++k)
      if (alphabet[k] == code[i]) v = (uint8_t)k;
    codon[i] = v;
  }
  __syncthreads();
}

// translate.rs:124-137 min_orf_len, or the caller's value when >= 0
__device__ __forceinline__ uint64_t min_orf_of(uint64_t dna_len, int64_t user) {
  if (user >= 0) return (uint64_t)user;
  return dna_len < 30 ? 1 : (dna_len < 100 ? 20 : 40);
}

__global__ void k_frame_lengths(const uint64_t* __restrict__ nt_off, uint64_t n_reads, uint64_t* __restrict__ len) {
  const uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x;
  if (i > 6 * n_reads) return;
  if (i == 6 * n_reads) {
    len[i] = 0;  // the scan's total slot
    return;
  }
  const uint64_t L = nt_off[i / 6 + 1] - nt_off[i / 6];
  const uint64_t o = (i % 6) % 3;
  len[i] = L >= o ? (L - o) / 3 : 0;
}

// What base_of gives for each byte, and for each byte's complement.
__device__ __forceinline__ void stage_bases(uint8_t (&base)[2][256]) {
  for (int i = threadIdx.x; i < 256; i += blockDim.x) {
    base[0][i] = (uint8_t)base_of((uint8_t)i);
    base[1][i] = (uint8_t)base_of(complement_of((uint8_t)i));
  }
}

// One warp per frame, a codon per lane.  A stop-free stretch is known as a
// whole at its stop, so its letters are masked then, by the warp that wrote
// them.  (A thread per frame, a byte at a time: 220 us for 20,000 reads, now
// 110.)
__global__ void __launch_bounds__(kFrameWarps * 32) k_translate_frames(TranslateArgs a) {
  __shared__ uint8_t codon[64];
  __shared__ uint8_t base[2][256];
  stage_bases(base);
  stage_codons(codon);  // ends with a barrier
  const int lane = threadIdx.x & 31;
  const uint64_t warps = (uint64_t)gridDim.x * kFrameWarps;
  for (uint64_t i = blockIdx.x * (uint64_t)kFrameWarps + threadIdx.x / 32; i <= 6 * a.n_reads; i += warps) {
    if (i == 6 * a.n_reads) {  // the scans' total slots
      if (lane == 0) {
        a.keep[i] = 0;
        a.kept_len[i] = 0;
      }
      break;
    }
    const uint64_t r = i / 6;
    const int f = (int)(i % 6), o = f % 3;
    const uint8_t* nt = a.nt + a.nt_off[r];
    const uint64_t L = a.nt_off[r + 1] - a.nt_off[r];
    const uint64_t from = a.scratch_off[i], n = a.scratch_off[i + 1] - from;
    uint8_t* out = a.scratch + from;
    // translate.rs:98-118: stop-free stretches shorter than min_len become X
    const uint64_t min_len = min_orf_of(L, a.min_orf);
    uint64_t begin = 0;  // of the stretch at hand
    const auto mask_to = [&](uint64_t end) {
      if (end - begin >= min_len) return;
      __syncwarp();
      for (uint64_t k = begin + lane; k < end; k += 32) out[k] = kXLetterDev;
    };
    for (uint64_t c0 = 0; c0 < n; c0 += 32) {
      const uint64_t c = c0 + lane;
      uint8_t v = kXLetterDev;
      if (c < n) {
        uint32_t b[3];
#pragma unroll
        for (int k = 0; k < 3; ++k) {
          const uint64_t p = o + 3 * c + k;  // position in the strand
          b[k] = f < 3 ? base[0][nt[p]] : base[1][nt[L - 1 - p]];
        }
        v = (b[0] | b[1] | b[2]) > 3 ? kXLetterDev : codon[b[0] * 16 + b[1] * 4 + b[2]];
        out[c] = v;
      }
      for (uint32_t stops = __ballot_sync(0xFFFFFFFFu, c < n && v == kStopLetterDev); stops; stops &= stops - 1) {
        const uint64_t at = c0 + __ffs(stops) - 1;
        mask_to(at);
        begin = at + 1;
      }
    }
    mask_to(n);
    __syncwarp();
    // workflow.rs:118: a frame without a letter below X is not searched
    bool real = false;
    for (uint64_t c0 = 0; c0 < n && !real; c0 += 32)
      real = __any_sync(0xFFFFFFFFu, c0 + lane < n && out[c0 + lane] < kXLetterDev);
    if (lane == 0) {
      a.keep[i] = real ? 1 : 0;
      a.kept_len[i] = real ? n : 0;
    }
  }
}

__global__ void __launch_bounds__(kFrameWarps * 32) k_compact_frames(TranslateArgs a) {
  const int lane = threadIdx.x & 31;
  const uint64_t warps = (uint64_t)gridDim.x * kFrameWarps;
  for (uint64_t i = blockIdx.x * (uint64_t)kFrameWarps + threadIdx.x / 32; i <= 6 * a.n_reads; i += warps) {
    if (i == 6 * a.n_reads) {  // offsets[n_targets] = letters of all kept frames
      if (lane == 0) a.out_off[a.kept_index[i]] = a.kept_off[i];
      break;
    }
    if (!a.keep[i]) continue;
    const uint64_t t = a.kept_index[i];
    const uint64_t n = a.kept_len[i];
    const uint8_t* src = a.scratch + a.scratch_off[i];
    uint8_t* dst = a.out + a.kept_off[i];
    for (uint64_t c = lane; c < n; c += 32) dst[c] = src[c];
    if (lane == 0) {
      a.out_off[t] = a.kept_off[i];
      a.out_query[t] = (uint32_t)(i / 6);
      a.out_frame[t] = (uint8_t)(i % 6);
    }
  }
}

// Blocks of one warp per frame, at most eight to an SM (each stages its tables).
unsigned frame_blocks(uint64_t n_reads) {
  return (unsigned)std::min<uint64_t>((6 * n_reads + kFrameWarps) / kFrameWarps, 148 * 8);
}

}  // namespace

void launch_frame_lengths(const uint64_t* nt_off, uint64_t n_reads, uint64_t* len, cudaStream_t st) {
  count_launch();
  k_frame_lengths<<<ceil_div(6 * n_reads + 1, 256), 256, 0, st>>>(nt_off, n_reads, len);
  DRG_CUDA(cudaGetLastError());
}

void launch_translate_frames(const TranslateArgs& a, cudaStream_t st) {
  count_launch();
  k_translate_frames<<<frame_blocks(a.n_reads), kFrameWarps * 32, 0, st>>>(a);
  DRG_CUDA(cudaGetLastError());
}

void launch_compact_frames(const TranslateArgs& a, cudaStream_t st) {
  count_launch();
  k_compact_frames<<<frame_blocks(a.n_reads), kFrameWarps * 32, 0, st>>>(a);
  DRG_CUDA(cudaGetLastError());
}

}  // namespace drg
