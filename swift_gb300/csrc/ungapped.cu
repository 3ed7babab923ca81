// Gapless pass: the exact Smith-Waterman result of every pair whose best
// alignment provably holds no gap, without a dynamic program.
//
// Unrolling the recurrence (sw.cu) from a cell gives a chain of moves whose
// costs add up to the cell's score.  The first gap move of a chain costs
// gap_open (its neighbour was reached by DIAG or is NONE), every later gap
// and mismatch less than zero (packed scoring: mismatch, gap_open < 0,
// gap_open <= gap_ext < 0), and each of the Q rows matches at most once, so
// a chain with a gap scores at most
//     B = match * Q + gap_open.
// Let M be the largest gapless score: over the diagonals of the pair, the
// best local sum of match / mismatch.  A cell's score is at least its
// diagonal's local sum (DIAG enters the maximum unconditionally).  If M > B,
// no cell scores M or more through a gap, so the cells of score M are the
// cells whose diagonal sum is M, every cell of such a chain holds its
// diagonal sum, and the traceback is that diagonal from the first maximum
// back to the last cell whose sum is 0 (NONE wins at 0).  Score, first
// row-major maximum, start, end and strings follow from the diagonal alone.
// If M <= B, the pair's score is at most B whatever its gaps: a read with
// one such alignment is done, since no other pair of it can reach it.
//
// Finding M > B: every mismatched or trimmed row loses at least `match`
// against a whole match, so such a diagonal mismatches at most
// k = (-gap_open - 1) / match of its Q rows (4 with the default scoring),
// rows outside the window counted.  Query and window are 2-bit codes; rows
// 16..31 of the query are compared with the window at every start by a
// funnel shift, an exclusive or and a population count (8 instructions per
// diagonal), and a diagonal with at most k mismatches there (one in 30,000
// by chance) is checked whole, after the scan.
//
// Layout: one thread per record; the codes of the reference (16 bases a
// word, in L2) and of the reads, both strands, are read in place, so no
// window or query is written out for the records this settles.  Bound by
// the ALU pipe (88 %): at 100-base reads and 300-base windows a warp takes 3,600
// instructions for its 32 records, 2,500 of them on that pipe (4.13 M records
// 0.56 ms).
//
// gapless_bound_kernel applies the same argument with a smaller bound to the
// pairs that remain, once the LCS pass has run: the matches of a chain are a
// common subsequence, so B = match * LCS(query, window) + gap_open.  That
// settles alignments with more mismatches, and those that the window cuts
// off, as it does every read longer than R - back bases.
#include "internal.h"

namespace swift {
namespace {

// class of four A, C, G, T bytes (either case): A 0, C 1, G 2, T 3
__device__ __forceinline__ uint32_t class4(uint32_t x) { return ((x >> 1) ^ (x >> 2)) & 0x03030303u; }

// the 2-bit classes of four bytes side by side, first byte lowest
__device__ __forceinline__ uint32_t squeeze4(uint32_t cls) { return (cls * 0x01041040u) >> 24; }

// whether four bytes are all upper-case A, C, G or T: rebuilt from classes
__device__ __forceinline__ bool acgt4(uint32_t x, uint32_t cls) {
  const uint32_t t = cls | (cls >> 4);
  return __byte_perm(0x54474341u, 0u, (t & 0x33u) | ((t >> 8) & 0x3300u)) == x;
}

// sixteen 2-bit codes in the opposite order
__device__ __forceinline__ uint32_t reverse2(uint32_t x) {
  x = __brev(x);
  return ((x >> 1) & 0x55555555u) | ((x & 0x55555555u) << 1);
}

constexpr int kPackReads = 32;  // reads per block, 8 lanes each

// Per read its class (0: the first Q bytes are all upper-case A, C, G, T;
// else 1) and, for class 0, the 2-bit codes of those Q bases and of their
// reverse complement, code_words(longest Q) words each, zero past Q.
__global__ void __launch_bounds__(kPackReads * 8) pack_reads_kernel(ReadPackArgs a) {
  __shared__ uint32_t fwd[kPackReads][kReadCodeWords + 1];
  const int sub = threadIdx.x >> 3, l = threadIdx.x & 7;
  const int64_t r = (int64_t)blockIdx.x * kPackReads + sub;
  const bool in = r < a.n_reads;
  const DevRead rd = in ? a.rd[r] : DevRead{0, 0, 0, 0};
  const int Q = !in ? 0 : a.read_q ? a.read_q[r] : a.Q;
  bool bad = !in || rd.len < Q || Q > 16 * a.words;
  if (!bad) {
    const uintptr_t ad = (uintptr_t)(a.reads + rd.seq_off);
    const uint32_t* wp = reinterpret_cast<const uint32_t*>(ad & ~(uintptr_t)3);
    const uint32_t sh = (uint32_t)(ad & 3) * 8;
    for (int w = l; w < a.words; w += 8) {
      uint32_t code = 0;
#pragma unroll
      for (int g = 0; g < 4; ++g) {
        const int left = Q - 16 * w - 4 * g;  // bases from these four bytes on
        if (left <= 0) break;
        // (the second load stays inside the buffer's padding)
        const uint32_t x = __funnelshift_r(wp[4 * w + g], wp[4 * w + g + 1], sh);
        const uint32_t keep = left >= 4 ? ~0u : (1u << (8 * left)) - 1u;
        const uint32_t cls = class4(x) & keep;
        bad |= !acgt4((x & keep) | (0x41414141u & ~keep), cls);
        code |= squeeze4(cls) << (8 * g);
      }
      fwd[sub][w] = code;
    }
  }
  const uint32_t group = 0xFFu << (threadIdx.x & 24);
  bad = __any_sync(group, bad);
  __syncwarp(group);
  if (!in) return;
  if (l == 0) a.read_cls[r] = bad ? 1 : 0;
  if (bad) return;
  const int nw = (Q + 15) >> 4, pad = 2 * (16 * nw - Q);
  uint32_t* out = a.codes + r * 2 * a.words;
  for (int w = l; w < a.words; w += 8) {
    out[w] = fwd[sub][w];
    uint32_t rc = 0;
    if (w < nw) {
      // reversed words hold the query's end first, after the padding
      const uint32_t x = reverse2(fwd[sub][nw - 1 - w]);
      const uint32_t y = w + 1 < nw ? reverse2(fwd[sub][nw - 2 - w]) : 0u;
      rc = ~__funnelshift_r(x, y, pad);
      const int left = Q - 16 * w;
      if (left < 16) rc &= (1u << (2 * left)) - 1u;
    }
    out[a.words + w] = rc;
  }
}

// one bit (the lower of its two) per base in which two words of codes differ
__device__ __forceinline__ uint32_t differ(uint32_t x, uint32_t y) {
  const uint32_t d = x ^ y;
  return (d | (d >> 1)) & 0x55555555u;
}

constexpr int kGaplessThreads = 128;

__global__ void __launch_bounds__(kGaplessThreads) gapless_kernel(GaplessArgs a) {
  const int64_t j = (int64_t)blockIdx.x * kGaplessThreads + threadIdx.x;
  if (j >= a.n) return;
  const int32_t read = a.m_read[j], strand = a.m_strand[j], ri = a.m_ri[j];
  const int32_t dist = max(0, a.m_rp[j] - a.back);
  const DevRecord& rec = a.recs[ri];
  const int Q = a.read_q ? a.read_q[read] : a.Q, R = a.R;
  const uint64_t cat0 = rec.cat_start, len = rec.cat_len;
  uint8_t state = kGaplessOther;
  DevPair pr;
  pr.read = read;
  pr.strand = strand;
  pr.ref_idx = ri;
  pr.ref_dist = dist;
  pr.win_len = R;
  pr.flags = 0;
  DevAln al;
  al.score = al.start = al.end = al.len = 0;
  // a whole window of A, C, G, T (either case) inside a regular record
  bool plain = rec.regular && a.read_cls[read] == 0 && len >= (uint64_t)dist + (uint64_t)R &&
               Q >= 32 + a.max_mis && a.match * Q + a.gap_open >= 0;
  const uint64_t g0 = cat0 + (uint64_t)dist;
  if (plain) {
    const uint64_t g1 = g0 + R - 1, o0 = g0 >> 5, o1 = g1 >> 5;
    uint32_t odd = 0;
    for (uint64_t o = o0; o <= o1; ++o) {
      uint32_t b = a.odd[o];
      if (o == o0) b &= ~0u << (g0 & 31);
      if (o == o1) b &= ~0u >> (31 - (g1 & 31));
      odd |= b;
    }
    plain = odd == 0;
  }
  if (plain) {
    state = kGaplessBounded;
    const uint32_t* q = a.codes + ((int64_t)read * 2 + strand) * a.words;
    const int64_t r0 = (int64_t)(g0 >> 4);
    const uint32_t rsh = (uint32_t)(g0 & 15) * 2;
    const int64_t rlast = a.ref_words - 1;
    auto raw = [&](int64_t i) { return __ldg(a.ref + min(r0 + i, rlast)); };
    const int k = a.max_mis, m = a.match, x = a.mismatch;
    int best = a.match * Q + a.gap_open, best_row = 0, best_first = 0, best_d = 0;
    // the whole of diagonal d (column = row + d, both from 0)
    auto check = [&](int d) {
      // codes of the window from column 16 w + d; columns outside it differ
      auto diff = [&](int w) -> uint32_t {
        const int c = 16 * w + d;  // first column of the word
        const int64_t b = (int64_t)g0 + c;
        uint32_t win;
        if (b >= 0) {
          const int64_t i = min(b >> 4, rlast);
          win = __funnelshift_r(__ldg(a.ref + i), __ldg(a.ref + min(i + 1, rlast)), (uint32_t)(b & 15) * 2);
        } else {
          win = __ldg(a.ref) << (2 * (int)-b);
        }
        uint32_t e = differ(win, q[w]);
        if (c < 0) e |= 0x55555555u & ((1u << (2 * -c)) - 1u);
        const int in = min(R - c, 32);  // columns of the word inside the window
        if (in < 16) e |= in <= 0 ? 0x55555555u : 0x55555555u & (~0u << (2 * in));
        const int rows = Q - 16 * w;
        if (rows < 16) e &= (1u << (2 * rows)) - 1u;
        return e;
      };
      const int nw = (Q + 15) >> 4;
      int mis = 0;
      for (int w = 0; w < nw && mis <= k; ++w) mis += __popc(diff(w));
      if (mis > k) return;
      // the best local sum over the runs between mismatches; a run's sum is
      // largest at its last row, and a sum of 0 or less starts over
      int u = 0, first = 0, row = 0;
      auto run_to = [&](int end) {  // rows [row, end) match
        u += m * (end - row);
        if (end > row &&
            (u > best || (u == best && best_row > 0 &&
                          (end < best_row || (end == best_row && d < best_d))))) {
          best = u;
          best_row = end;  // one-based row of the maximum
          best_first = first;
          best_d = d;
        }
      };
      for (int w = 0; w < nw; ++w) {
        for (uint32_t e = diff(w); e; e &= e - 1) {
          const int at = 16 * w + ((__ffs(e) - 1) >> 1);
          run_to(at);
          u += x;
          row = at + 1;
          if (u <= 0) {
            u = 0;
            first = row;
          }
        }
      }
      run_to(Q);
    };
    // rows 16..31 against the window at columns p = 16 + d; the diagonals
    // that pass are checked after the scan, all lanes of the warp together
    // (at once, each alone, they took two thirds of the kernel)
    uint64_t found = 0;
    int n_found = 0;
    const uint32_t qa = q[1];
    const int p_lo = 16 - k, p_hi = 16 + R - Q + k;
    uint32_t lo = raw(0), hi = raw(1);
    uint32_t w0 = __funnelshift_r(lo, hi, rsh);
    for (int t = 0; 16 * t <= p_hi; ++t) {
      lo = hi;
      hi = raw(t + 2);
      const uint32_t w1 = __funnelshift_r(lo, hi, rsh);
      uint32_t hits = 0;
#pragma unroll
      for (int s = 0; s < 16; ++s)
        if (__popc(differ(__funnelshift_r(w0, w1, 2 * s), qa)) <= k) hits |= 1u << s;
      w0 = w1;
      for (; hits; hits &= hits - 1) {
        const int p = 16 * t + __ffs(hits) - 1;
        if (p < p_lo || p > p_hi) continue;
        if (n_found < 4) {
          found |= (uint64_t)p << (16 * n_found);
          ++n_found;
        } else {
          check(p - 16);
        }
      }
    }
    for (int f = 0; f < n_found; ++f) check((int)((found >> (16 * f)) & 0xFFFFu) - 16);
    if (best_row > 0) {
      state = kGaplessDone;
      al.score = best;
      al.start = best_first + best_d + 1;
      al.len = best_row - best_first;
      al.end = al.start + al.len - 1;
      pr.flags = kPairGapless;
      pr.win_len = best_first;
    }
  }
  a.pairs[j] = pr;
  a.aln[j] = al;
  a.state[j] = state;
}

constexpr int kBoundWarps = 8;
// window codes with room before column 0 and past the end, so that a query
// word is compared at any diagonal
constexpr int kBoundPad = kReadCodeWords;
constexpr int kBoundWords = kBoundPad + (kFastMaxR + 15) / 16 + kReadCodeWords + 2;

// The listed packed pairs whose LCS bound leaves no gapped chain at or above
// their best diagonal: result and reversed strings are written; the others
// are listed in `rest`.  One warp per pair: its codes go to shared memory,
// then a lane takes every 32nd diagonal.  A diagonal of v rows inside the
// window can pass the bound B only with at most (match * v - B - 1) / match
// mismatches, which most exceed within a word or two.  100 K reads of 251
// bases: 274 us, and 1.8 ms less of trace pass and walk.
__global__ void __launch_bounds__(kBoundWarps * 32) gapless_bound_kernel(FastArgs a, int32_t* rest,
                                                                         int32_t* n_rest) {
  __shared__ uint32_t cq_all[kBoundWarps][kReadCodeWords], cw_all[kBoundWarps][kBoundWords];
  __shared__ int32_t left[kBoundWarps];
  const int wib = threadIdx.x >> 5, lane = threadIdx.x & 31;
  uint32_t *cq = cq_all[wib], *cw = cw_all[wib];
  const int64_t n = *a.count;
  const int m = a.match, x = a.mismatch, R = a.R;
  // the block's warps stay together: the appends are block-wide
  for (int64_t i0 = (int64_t)blockIdx.x * kBoundWarps; i0 < n; i0 += (int64_t)gridDim.x * kBoundWarps) {
    const int64_t i = i0 + wib;
    const int32_t p = i < n ? a.list[i] : -1;
    bool settled = false;
    if (p >= 0) {
      const int Q = a.q_len ? a.q_len[p] : a.Q;
      const char *q = a.q + (int64_t)p * a.q_stride, *w = a.w + (int64_t)p * a.w_stride;
      // codes of 16 bytes (rows are 16-byte aligned, zero past their end)
      auto codes = [](const char* b) -> uint32_t {
        const uint4 v = __ldg(reinterpret_cast<const uint4*>(b));
        return squeeze4(class4(v.x)) | squeeze4(class4(v.y)) << 8 | squeeze4(class4(v.z)) << 16 |
               squeeze4(class4(v.w)) << 24;
      };
      __syncwarp();
      for (int t = lane; t < kReadCodeWords; t += 32) cq[t] = 16 * t < Q ? codes(q + 16 * t) : 0u;
      for (int t = lane; t < kBoundWords; t += 32) {
        const int c = 16 * (t - kBoundPad);
        cw[t] = c >= 0 && c < R ? codes(w + c) : 0u;
      }
      __syncwarp();
      const int bound = max(a.ub[p] + a.gap_open, 0);
      int best = bound, best_row = 0, best_first = 0, best_d = 0;
      for (int d = lane - (Q - 1); d < R; d += 32) {
        const int r0 = max(0, -d), r1 = min(Q, R - d);  // rows inside the window
        if (m * (r1 - r0) <= bound) continue;
        const int most = (m * (r1 - r0) - bound - 1) / m;
        auto diff = [&](int wd) -> uint32_t {
          const int c = 16 * (wd + kBoundPad) + d;
          uint32_t e = differ(__funnelshift_r(cw[c >> 4], cw[(c >> 4) + 1], (uint32_t)(c & 15) * 2), cq[wd]);
          if (16 * wd < r0) e &= ~0u << (2 * (r0 - 16 * wd));
          if (16 * wd + 16 > r1) e &= (1u << (2 * (r1 - 16 * wd))) - 1u;
          return e;
        };
        const int w0 = r0 >> 4, w1 = (r1 + 15) >> 4;
        int mis = 0;
        for (int wd = w0; wd < w1 && mis <= most; ++wd) mis += __popc(diff(wd));
        if (mis > most) continue;
        // the best local sum, as in gapless_kernel
        int u = 0, first = r0, row = r0;
        auto run_to = [&](int end) {
          u += m * (end - row);
          if (end > row && (u > best || (u == best && best_row > 0 && end < best_row))) {
            best = u;
            best_row = end;
            best_first = first;
            best_d = d;
          }
        };
        for (int wd = w0; wd < w1; ++wd) {
          for (uint32_t e = diff(wd); e; e &= e - 1) {
            const int at = 16 * wd + ((__ffs(e) - 1) >> 1);
            run_to(at);
            u += x;
            row = at + 1;
            if (u <= 0) {
              u = 0;
              first = row;
            }
          }
        }
        run_to(r1);
      }
      // first row-major maximum over the lanes (a lane's diagonals go up, so
      // it kept the first column of a row)
#pragma unroll
      for (int s = 16; s > 0; s >>= 1) {
        const int ob = __shfl_xor_sync(0xffffffffu, best, s);
        const int orow = __shfl_xor_sync(0xffffffffu, best_row, s);
        const int of = __shfl_xor_sync(0xffffffffu, best_first, s);
        const int od = __shfl_xor_sync(0xffffffffu, best_d, s);
        if (orow > 0 && (best_row == 0 || ob > best ||
                         (ob == best && (orow < best_row || (orow == best_row && od < best_d))))) {
          best = ob;
          best_row = orow;
          best_first = of;
          best_d = od;
        }
      }
      settled = best_row > 0;
      if (settled) {
        const int len = best_row - best_first;
        if (lane == 0) {
          DevAln al;
          al.score = best;
          al.start = best_first + best_d + 1;
          al.end = al.start + len - 1;
          al.len = len;
          a.aln[p] = al;
        }
        char *qc = a.qcons + (int64_t)p * a.cons_stride, *rc = a.rcons + (int64_t)p * a.cons_stride;
        for (int t = lane; t < len; t += 32) {
          qc[t] = q[best_row - 1 - t];
          rc[t] = w[best_row - 1 + best_d - t];
        }
      }
    }
    __syncthreads();
    if (lane == 0) left[wib] = p >= 0 && !settled ? p : -1;
    __syncthreads();
    const int32_t mine = threadIdx.x < kBoundWarps ? left[threadIdx.x] : -1;
    block_append(mine >= 0, mine, rest, n_rest);
  }
}

__global__ void left_kernel(LeftArgs a) {
  const int64_t j = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (j >= a.n || !a.open[j]) return;
  const uint32_t t = a.at[j];
  a.l_read[t] = a.m_read[j];
  a.l_strand[t] = a.m_strand[j];
  a.l_ri[t] = a.m_ri[j];
  a.l_rp[t] = a.m_rp[j];
  a.l_of[t] = (int32_t)j;
  if (a.group_start) a.l_start[t] = a.group_start[j];
}

}  // namespace

int gapless_max_mismatches(int match, int mismatch, int gap_open, int gap_ext) {
  if (!(match > 0 && mismatch < 0 && gap_open < 0 && gap_ext < 0 && gap_ext >= gap_open)) return -1;
  const int k = (-gap_open - 1) / match;
  return k <= kGaplessMaxMis ? k : -1;
}

void launch_pack_reads(cudaStream_t st, const ReadPackArgs& a) {
  if (a.n_reads <= 0) return;
  pack_reads_kernel<<<(unsigned)((a.n_reads + kPackReads - 1) / kPackReads), kPackReads * 8, 0, st>>>(a);
}

int launch_gapless_bound(cudaStream_t st, const FastArgs& a, int64_t max_pairs, int32_t* rest,
                         int32_t* n_rest) {
  if (max_pairs <= 0) return 0;
  if ((a.q_stride | a.w_stride) % 16 != 0 || a.R > kFastMaxR || a.Q > kMaxQ) return 0;
  const int64_t blocks = std::min<int64_t>((max_pairs + kBoundWarps - 1) / kBoundWarps, 152 * 8);
  gapless_bound_kernel<<<(unsigned)blocks, kBoundWarps * 32, 0, st>>>(a, rest, n_rest);
  return 1;
}

void launch_left(cudaStream_t st, const LeftArgs& a) {
  if (a.n <= 0) return;
  left_kernel<<<(unsigned)((a.n + 255) / 256), 256, 0, st>>>(a);
}

void launch_gapless(cudaStream_t st, const GaplessArgs& a) {
  if (a.n <= 0) return;
  gapless_kernel<<<(unsigned)((a.n + kGaplessThreads - 1) / kGaplessThreads), kGaplessThreads, 0, st>>>(a);
}

}  // namespace swift
