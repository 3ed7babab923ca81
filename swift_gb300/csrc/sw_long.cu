// Phase 2 for long pairs (queries up to 4096, windows up to 8192 bases):
// one CTA per pair, the reference kernel's recurrence and tie rules
// (src/smithWaterman.cu:510-645, 911-1026) in int32 cells.
//
// Cells use the packed passes' encoding, Hx = 16 H + onehot(direction) + B,
// so one add-max chain gives H and the reference's direction with its tie
// precedence, and the next cells' gap penalties come from the code bits; at
// these lengths 16 H exceeds 16 bits, so a cell is one 32-bit lane.
//
// Layout.  The 256 threads own consecutive strips of RPL query rows (RPL =
// 4, 8, 12 or 16, the smallest that covers the query).  Within a warp, lane
// t sweeps the window one column behind lane t-1 (shuffles carry the bottom
// row down).  Between warps, lane 31 writes its bottom row's H and UP
// candidate per column to a shared ring that lane 0 of the next warp reads;
// warp w runs two 32-column stages behind warp w-1, one __syncthreads per
// stage, so every value is written before it is read and a ring of 128
// columns is never overrun.  Each thread streams its 2-bit direction codes
// per wavefront step to global scratch (four steps per 16-byte store);
// sw_long_walk_kernel then walks the reference's traceback, one warp per
// pair, carrying the cell score to tell NONE from LEFT.
//
// Pairs of A, C, G and T only whose scores fit run sw_long16_kernel below,
// two query strips per thread in 16-bit halves.
#include <type_traits>

#include "internal.h"

namespace swift {
namespace {

constexpr int kLW = 8;           // warps per CTA
constexpr int kLT = kLW * 32;    // threads per CTA
constexpr int kStage = 32;       // wavefront steps per stage
constexpr int kRing = 128;       // ring columns between neighbouring warps
constexpr int kWild = 0x100;     // 'N' matches every byte

__device__ __forceinline__ int upcase(uint8_t c) {
  return (unsigned)(c - 'a') < 26u ? c - 'a' + 'A' : c;
}

constexpr int kColMask = (1 << 17) - 1;

__device__ __forceinline__ uint32_t prmt_b(uint32_t a, uint32_t b, uint32_t s) {
  uint32_t d;
  asm("prmt.b32 %0, %1, %2, %3;" : "=r"(d) : "r"(a), "r"(b), "r"(s));
  return d;
}

// base class of an ACGTN pair byte: A 0, C 1, G 2, T 3, N 4 (either case)
__device__ __forceinline__ int class5(uint8_t c) {
  const int u = upcase(c);
  return u == 'C' ? 1 : u == 'G' ? 2 : u == 'T' ? 3 : u == 'N' ? 4 : 0;
}

// PROF: the pair holds only ACGTN bytes (either case) and 16 m Q stays below
// 2^18.  Then the substitution score is one byte permute of a per-row
// profile (window classes A, C, G, T, N), and a row's first maximum is one
// max over keys 2^17 H' + (2^17 - 1 - column), H' = H + B / 16 (16 H + B
// times 2^13, whose low 17 bits are zero): the largest H, and on equal H the
// smallest column.  Other pairs compare bytes.
template <int RPL, bool PROF>
__global__ void __launch_bounds__(kLT, 2) sw_long_kernel(LongArgs a) {
  extern __shared__ __align__(16) uint8_t smem[];
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int64_t item = (int64_t)blockIdx.x;
  if (item >= a.n) return;
  const int32_t p = a.list[item];
  const int Q = a.q_len[p], R = a.r_len[p];
  const char* qg = a.qry + a.q_off[p];
  const char* wg = a.ref + a.r_off[p];
  // shared: up-cased window (int16 per column), rings for the 7 warp boundaries
  int16_t* wu = reinterpret_cast<int16_t*>(smem);                    // [R + 1]
  int32_t* ring = reinterpret_cast<int32_t*>(smem + ((2 * (a.max_r + 1) + 15) & ~15));
  // ring[(b * 2 + 0) * kRing + col % kRing]: UP candidate of boundary b's upper row
  // ring[(b * 2 + 1) * kRing + col % kRing]: its H (code bits cleared)
  for (int c = tid; c < R; c += kLT) {
    if (PROF) {  // byte-permute selector: the class's byte, sign-extended
      const uint32_t k = (uint32_t)class5((uint8_t)wg[c]);
      wu[c + 1] = (int16_t)(k | ((k | 8u) << 4) | ((k | 8u) << 8) | ((k | 8u) << 12));
    } else {
      const int u = upcase((uint8_t)wg[c]);
      wu[c + 1] = (int16_t)(u == 'N' ? kWild : u);
    }
  }
  const int B = a.bias;
  const int B8 = B + 8;
  const int CU = 16 * a.gap_open + 2, CL = 16 * a.gap_open + 1;
  const int KU = 8 * (a.gap_ext - a.gap_open), KL = 16 * (a.gap_ext - a.gap_open);
  const int SM = 16 * a.match + 4, SX = 16 * a.mismatch + 4;
  int qv[RPL], h16p[RPL], xl[RPL], bestv[RPL], bestc[RPL];
  uint32_t pf0[PROF ? RPL : 1], pf1[PROF ? RPL : 1];
  const uint32_t sm8 = (uint32_t)(uint8_t)(int8_t)SM, sx8 = (uint32_t)(uint8_t)(int8_t)SX;
#pragma unroll
  for (int k = 0; k < RPL; ++k) {
    const int i = tid * RPL + k;
    if (PROF) {
      // scores against window classes A C G T (pf0) and N (pf1 byte 0);
      // rows past the query mismatch everything (and stay out of the maximum)
      const int qc = i < Q ? class5((uint8_t)qg[i]) : -1;
      uint32_t v0 = 0;
#pragma unroll
      for (int w = 0; w < 4; ++w)
        v0 |= ((qc == w || qc == 4) ? sm8 : sx8) << (8 * w);
      pf0[k] = v0;
      pf1[k] = qc >= 0 ? sm8 : sx8;
      bestv[k] = B * 8192 + kColMask;  // H = 0 at column 0: no H = 0 cell beats it
    } else {
      if (i < Q) {
        const int u = upcase((uint8_t)qg[i]);
        qv[k] = u == 'N' ? kWild : u;
      } else {
        qv[k] = -1;  // past the query: matches nothing (kept out of the maximum)
      }
      bestv[k] = B;
    }
    h16p[k] = B;
    xl[k] = B;
    bestc[k] = 0;
  }
  const int S4 = (R + 31 + 3) & ~3;  // steps of one thread's direction words
  // the pair's own slot: 256 threads x S4 words from dir_off[item]
  uint32_t* dirs = a.dirs + a.dir_off[item] + (int64_t)tid * S4;
  __syncthreads();
  int send_u = B, send_h = B, diag = B;
  // One wavefront step: this lane's column j against its RPL rows.  FULL:
  // every lane's column lies in 1..R (a warp-uniform fact of the step), so
  // no lane is masked and the rows' state updates in place.
  auto step = [&](const int s, auto full) -> uint32_t {
    constexpr bool kFull = decltype(full)::value;
    int up = __shfl_up_sync(0xffffffffu, send_u, 1);
    const int rh = __shfl_up_sync(0xffffffffu, send_h, 1);
    const int j = s - lane + 1;  // this lane's column
    const bool in = kFull || (j >= 1 && j <= R);
    if (lane == 0) {
      if (warp == 0) {
        up = B;  // row 0
      } else if (in) {
        up = ring[((warp - 1) * 2 + 0) * kRing + (j & (kRing - 1))];
      }
    }
    uint32_t acc = 0;
    if (in) {
      const int rv = wu[j];
      const int cj = kColMask - j;
      int dg = diag;
#pragma unroll
      for (int k = 0; k < RPL; ++k) {
        int sc;
        if (PROF) {
          sc = (int)prmt_b(pf0[k], pf1[k], (uint32_t)(uint16_t)rv);
        } else {
          const bool hit = qv[k] == rv || qv[k] == kWild || (rv == kWild && qv[k] >= 0);
          sc = hit ? SM : SX;
        }
        // DIAG against LEFT off the chain down the rows, then UP and NONE
        const int dl = __viaddmax_s32(dg, sc, xl[k] + CL);
        const int hx = __vimax3_s32(dl, up + CU, B8);
        dg = h16p[k];
        const int h16 = hx & ~15;
        h16p[k] = h16;
        up = (hx & 2) * KU + h16;
        xl[k] = (hx & 1) * KL + h16;
        if (PROF) {
          bestv[k] = max(bestv[k], h16 * 8192 + cj);
        } else if (h16 > bestv[k]) {
          bestv[k] = h16;
          bestc[k] = j;
        }
        // 2 DIAG, 1 UP, 0 LEFT / NONE: code bits 2..1 to bits 2k+1..2k
        if (k == 0) {
          acc |= ((uint32_t)hx >> 1) & 3u;
        } else {
          acc |= ((uint32_t)hx << (2 * k - 1)) & (3u << (2 * k));
        }
      }
      send_u = up;
      send_h = h16p[RPL - 1];
      if (lane == 31 && warp + 1 < kLW) {
        ring[(warp * 2 + 0) * kRing + (j & (kRing - 1))] = up;
        ring[(warp * 2 + 1) * kRing + (j & (kRing - 1))] = send_h;
      }
    }
    // the diagonal of the next step: lane above's bottom H at this column
    // (lane 0: from the ring; column 0 is H = 0)
    if (lane == 0) {
      diag = (warp == 0 || !in) ? B : ring[((warp - 1) * 2 + 1) * kRing + (j & (kRing - 1))];
    } else {
      diag = rh;
    }
    return acc;
  };
  const int steps = R + 31;                          // a warp's wavefront
  // warps whose rows all lie past the query compute nothing (their lanes'
  // rows are out of the maximum, and the walk never reads them); the stage
  // count follows the last warp that computes
  const int act = min(kLW, (Q + 32 * RPL - 1) / (32 * RPL));
  const int n_stages = 2 * (act - 1) + (steps + kStage - 1) / kStage;
  for (int stage = 0; stage < n_stages; ++stage) {
    const int s_lo = (stage - 2 * warp) * kStage;
    if (warp < act && s_lo >= 0 && s_lo < steps) {
#pragma unroll 1
      for (int s0 = s_lo; s0 < s_lo + kStage; s0 += 4) {
        uint4 v;
        if (s0 >= 31 && s0 + 3 <= R - 1) {  // lane 31 past column 0, lane 0 short of R + 1
          v.x = step(s0, std::true_type());
          v.y = step(s0 + 1, std::true_type());
          v.z = step(s0 + 2, std::true_type());
          v.w = step(s0 + 3, std::true_type());
        } else {
          v.x = step(s0, std::false_type());
          v.y = step(s0 + 1, std::false_type());
          v.z = step(s0 + 2, std::false_type());
          v.w = step(s0 + 3, std::false_type());
        }
        if (s0 < S4) __stcg(reinterpret_cast<uint4*>(dirs + s0), v);
      }
    }
    __syncthreads();
  }
  // first maximum in row-major order: per thread, then over the CTA
  int bv = 0, br = 0x7fffffff, bc = 0;
#pragma unroll
  for (int k = 0; k < RPL; ++k) {
    const int i = tid * RPL + k;
    const int v = PROF ? (bestv[k] >> 17) << 4 : bestv[k];
    if (i < Q && v > bv) {
      bv = v;
      br = i + 1;
      bc = PROF ? kColMask - (bestv[k] & kColMask) : bestc[k];
    }
  }
  __shared__ int red_v[kLW], red_r[kLW], red_c[kLW];
#pragma unroll
  for (int d = 16; d > 0; d >>= 1) {
    const int ov = __shfl_xor_sync(0xffffffffu, bv, d);
    const int orr = __shfl_xor_sync(0xffffffffu, br, d);
    const int oc = __shfl_xor_sync(0xffffffffu, bc, d);
    if (ov > bv || (ov == bv && orr < br)) {
      bv = ov;
      br = orr;
      bc = oc;
    }
  }
  if (lane == 0) {
    red_v[warp] = bv;
    red_r[warp] = br;
    red_c[warp] = bc;
  }
  __syncthreads();
  if (tid == 0) {
    for (int w = 1; w < kLW; ++w) {
      if (red_v[w] > bv || (red_v[w] == bv && red_r[w] < br)) {
        bv = red_v[w];
        br = red_r[w];
        bc = red_c[w];
      }
    }
    const int score = bv > B ? (bv - B) >> 4 : 0;
    a.best[p] = make_int2(score, score > 0 ? br * (R + 1) + bc : 0);
  }
}

// The same recurrence in packed 16-bit halves, for pairs of A, C, G, T bytes
// (either case) with 4 * match * Q + bias below 2^15 (long16_max_q).
//
// Cells are 4 * H + code + B with code 3 DIAG or NONE, 2 UP, 1 LEFT: one
// three-way maximum gives H and the direction (on equal H DIAG before UP
// before LEFT; DIAG and NONE need no telling apart, a cell is NONE exactly
// when H = 0), and a cleared code bit selects the next cells' gap penalties.
//
// Layout.  Thread t owns two strips of RH query rows, virtual lane 2 t in the
// low half and 2 t + 1, the next RH rows, in the high half, one window column
// behind: the warp is a wavefront of 64 strips.  The low strip's bottom row
// moves to the high half of the next step by one funnel shift, which also
// brings in the lane above's high strip (one shuffle).  The window selector
// of a column holds the low half's base and, a column back, the high half's.
// Steps in which some lane's column lies outside the window score mismatches
// there: cells left of the window then keep H = 0, and cells right of it stay
// below the window's maximum.  Warps follow one another 5 stages of 16 steps
// apart (a strip's bottom row leaves the warp 62 steps after it enters), over
// rings of 64 columns.
//
// First maximum.  A lane only keeps the maximum of its cells over 4 steps;
// where it reaches the warp's largest so far, which happens while the
// alignment itself passes and rarely else, it puts those steps' cells aside
// and goes on; only the last ones put aside, and equal maxima, are looked
// through cell by cell.  (Looking at once made every warp of the CTA wait for
// the one the alignment passes: 3.7 ms for queries of 3 to 4 kb, whose
// barriers took half of it, against 3.5 ms for pairs of all sizes.)  A cell of the
// final maximum is never missed, since the warp's largest so far never
// exceeds it.
//
// Per two cells of a strip 12.5 instructions, 6.5 on the ALU pipe, where the
// int32 kernel takes 28 and 18 (500 pairs of 1-4 kb by 2-8 kb: 3.5 ms, 13.4
// before over four launches).  Over a whole launch 19.5 and 10.1 per two cells of
// the pairs (300 of them, one wave): the step's shuffles, ring, selectors and
// tests are shared by 4 to 16 rows, and rows past the query and skewed columns
// count too.  The ALU pipe is busy 56 % of the time; the largest stall is the
// barrier between stages, where warps that have not started or have ended wait.
constexpr int kStage16 = 16;
constexpr int kLag16 = 5;    // stages between neighbouring warps
constexpr int kRing16 = 64;  // ring columns
constexpr int kPad16 = 64;   // selectors before column 0
constexpr int kSel16 = kPad16 + 96;  // and in all beside the window's columns

template <int RH>
__device__ __forceinline__ void long16_pair(const LongArgs& a, const int64_t item, const int32_t p,
                                            const int Q, const int R, uint8_t* smem) {
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const char* qg = a.qry + a.q_off[p];
  const char* wg = a.ref + a.r_off[p];
  uint16_t* wsel = reinterpret_cast<uint16_t*>(smem);  // [kPad16 + column]
  uint32_t* ring = reinterpret_cast<uint32_t*>(smem + ((2 * (a.max_r + kSel16) + 15) & ~15));
  for (int c = tid; c < R + kSel16; c += kLT) {
    const int j = c - kPad16;
    const uint32_t lo = j >= 1 && j <= R ? (uint32_t)class5((uint8_t)wg[j - 1]) : 0u;
    const uint32_t hi = j >= 2 && j <= R + 1 ? (uint32_t)class5((uint8_t)wg[j - 2]) : 0u;
    wsel[c] = (uint16_t)(lo | ((lo | 8u) << 4) | ((4u + hi) << 8) | (((4u + hi) | 8u) << 12));
  }
  const uint32_t B = (uint32_t)a.bias;
  const uint32_t BB = B * 0x00010001u, B3 = BB + 0x00030003u;
  const uint32_t CU = (uint32_t)((4 * a.gap_open + 2) * 65537);
  const uint32_t CL = (uint32_t)((4 * a.gap_open + 1) * 65537);
  const uint32_t KU = (uint32_t)(4 * (a.gap_ext - a.gap_open));
  const uint32_t KL = (uint32_t)(2 * (a.gap_ext - a.gap_open));
  const uint32_t sm = (uint32_t)(uint8_t)(int8_t)(4 * a.match + 3);
  const uint32_t sx = (uint32_t)(uint8_t)(int8_t)(4 * a.mismatch + 3);
  const uint32_t all_x = sx * 0x01010101u;
  const uint32_t SX = ((uint32_t)(4 * a.mismatch + 3) & 0xFFFFu) * 0x00010001u;
  uint32_t pf0[RH], pf1[RH], h[RH], xl[RH];
#pragma unroll
  for (int k = 0; k < RH; ++k) {
    const int i0 = 2 * tid * RH + k, i1 = i0 + RH;
    pf0[k] = i0 < Q ? all_x ^ ((sm ^ sx) << (8 * class5((uint8_t)qg[i0]))) : all_x;
    pf1[k] = i1 < Q ? all_x ^ ((sm ^ sx) << (8 * class5((uint8_t)qg[i1]))) : all_x;
    h[k] = BB;
    xl[k] = BB;
  }
  const int S4 = (R + 63 + 3) & ~3;
  uint32_t* dirs = a.dirs + a.dir_off[item] + (int64_t)tid * S4;
  __syncthreads();
  const int act = min(kLW, (Q + 64 * RH - 1) / (64 * RH));  // warps with rows of the query
  uint32_t send_u = BB, send_h = BB, diag = BB;
  uint32_t bm = 0;         // maximum of the block's cells
  uint32_t hs[3][RH];      // cells of the block's steps but the last
  uint32_t W = B + 4;      // largest cell of the warp so far (from H = 1)
  // the lane's maximum; its first row and column, or, while pending, the
  // cells of the only 4 steps that hold it so far (snap, from step snap_s0)
  uint32_t rv = 0;
  int rr = 0, rc = 0, snap_s0 = 0;
  bool pending = false;
  uint32_t* snap = a.dirs + a.dir_off[item] + (int64_t)kLT * S4 + tid * (4 * RH);
  // (rr, rc) takes the first cell of value rv in the 4 steps from s0 on
  auto look_all = [&](int s0, const uint32_t* cells) {
    for (int u = 0; u < 4; ++u)
      for (int k = 0; k < RH; ++k) {
        const uint32_t both = cells[u * RH + k];
        for (int hf = 0; hf < 2; ++hf) {
          const uint32_t c = hf ? both >> 16 : both & 0xFFFFu;
          const int row = (2 * tid + hf) * RH + k + 1, col = s0 + u - 2 * lane + 1 - hf;
          if (c == rv && row <= Q && col >= 1 && col <= R && (row < rr || (row == rr && col < rc))) {
            rr = row;
            rc = col;
          }
        }
      }
  };
  auto step = [&](const int s, auto edge) -> uint32_t {
    constexpr bool kEdge = decltype(edge)::value;
    uint32_t ru = __shfl_up_sync(0xffffffffu, send_u, 1);
    uint32_t rh = __shfl_up_sync(0xffffffffu, send_h, 1);
    const int j = s - 2 * lane + 1;  // the low half's column; the high half's is j - 1
    if (lane == 0) {
      ru = rh = BB;  // row 0
      if (warp > 0 && (!kEdge || j <= R)) {
        const uint32_t x = ring[(warp - 1) * kRing16 + (j & (kRing16 - 1))];
        ru = x << 16;
        rh = x;
      }
    }
    uint32_t up = __funnelshift_r(ru, send_u, 16);
    const uint32_t hin = __funnelshift_r(rh, send_h, 16);
    const uint32_t ws = wsel[kPad16 + j];
    uint32_t in = 0;  // halves whose column lies inside the window
    if (kEdge) in = (j >= 1 && j <= R ? 0xFFFFu : 0u) | (j >= 2 && j <= R + 1 ? 0xFFFF0000u : 0u);
    uint32_t dg = diag, acc = 0, pair = 0;
#pragma unroll
    for (int k = 0; k < RH; ++k) {
      uint32_t sc = prmt_b(pf0[k], pf1[k], ws);
      if (kEdge) sc = (sc & in) | (SX & ~in);
      const uint32_t dl = __viaddmax_s16x2(dg, sc, xl[k] + CL);
      const uint32_t hx = __vimax3_s16x2(dl, up + CU, B3);
      dg = h[k];
      const uint32_t hh = hx & 0xFFFCFFFCu;
      h[k] = hh;
      const uint32_t bu = ~hx & 0x00010001u, bl = ~hx & 0x00020002u;  // 1 UP, 2 LEFT
      up = bu * KU + hh;
      xl[k] = bl * KL + hh;
      // the strip's codes, last row lowest (multiply-adds: FMA pipe)
      acc = k == 0 ? bu : acc * a.four + bu;
      acc = bl * a.one + acc;
      if (k & 1)
        bm = __vimax3_s16x2(bm, pair, hh);
      else
        pair = hh;
    }
    send_u = up;
    send_h = h[RH - 1];
    diag = hin;
    if (lane == 31 && warp + 1 < act)
      ring[warp * kRing16 + ((j - 1) & (kRing16 - 1))] = (up >> 16) | (send_h & 0xFFFF0000u);
    return acc;
  };
  auto keep = [&](int u) {
#pragma unroll
    for (int k = 0; k < RH; ++k) hs[u][k] = h[k];
  };
  const int steps = R + 63;
  const int n_stages = kLag16 * (act - 1) + (steps + kStage16 - 1) / kStage16;
  for (int stage = 0; stage < n_stages; ++stage) {
    const int s_lo = (stage - kLag16 * warp) * kStage16;
    if (warp < act && s_lo >= 0 && s_lo < steps) {
#pragma unroll 1
      for (int s0 = s_lo; s0 < s_lo + kStage16; s0 += 4) {
        uint4 v;
        bm = 0;
        if (s0 >= 63 && s0 + 3 <= R - 1) {
          v.x = step(s0, std::false_type());
          keep(0);
          v.y = step(s0 + 1, std::false_type());
          keep(1);
          v.z = step(s0 + 2, std::false_type());
          keep(2);
          v.w = step(s0 + 3, std::false_type());
        } else {
          v.x = step(s0, std::true_type());
          keep(0);
          v.y = step(s0 + 1, std::true_type());
          keep(1);
          v.z = step(s0 + 2, std::true_type());
          keep(2);
          v.w = step(s0 + 3, std::true_type());
        }
        if (s0 < S4) __stcg(reinterpret_cast<uint4*>(dirs + s0), v);
        const uint32_t most = max(bm & 0xFFFFu, bm >> 16);
        if (__any_sync(0xffffffffu, most >= W)) {
          if (most >= W && most >= rv) {
            if (most > rv) {
              rv = most;
              pending = true;
            } else {  // the same maximum again: the first of them so far
              if (pending) {
                rr = rc = 0x7fffffff;
                look_all(snap_s0, snap);
                pending = false;
              }
            }
            uint32_t cells[4 * RH];
#pragma unroll
            for (int k = 0; k < RH; ++k) {
              cells[k] = hs[0][k];
              cells[RH + k] = hs[1][k];
              cells[2 * RH + k] = hs[2][k];
              cells[3 * RH + k] = h[k];
            }
            uint4* to = reinterpret_cast<uint4*>(snap);
#pragma unroll
            for (int q = 0; q < RH; ++q)
              to[q] = make_uint4(cells[4 * q], cells[4 * q + 1], cells[4 * q + 2], cells[4 * q + 3]);
            if (pending)
              snap_s0 = s0;
            else
              look_all(s0, snap);
          }
          // (rows past the query and columns past the window stay below the
          // pair's maximum, so W never passes it)
          W = max(W, __reduce_max_sync(0xffffffffu, most));
        }
      }
    }
    __syncthreads();
  }
  // first maximum in row-major order over the CTA
  if (pending) {
    rr = rc = 0x7fffffff;
    look_all(snap_s0, snap);
  }
  if (rr == 0x7fffffff) rv = 0;  // (past the query or the window only)
  __shared__ uint32_t red_v[kLW];
  __shared__ int red_r[kLW], red_c[kLW];
#pragma unroll
  for (int d = 16; d > 0; d >>= 1) {
    const uint32_t ov = __shfl_xor_sync(0xffffffffu, rv, d);
    const int orr = __shfl_xor_sync(0xffffffffu, rr, d);
    const int oc = __shfl_xor_sync(0xffffffffu, rc, d);
    if (ov > rv || (ov == rv && orr < rr)) {
      rv = ov;
      rr = orr;
      rc = oc;
    }
  }
  if (lane == 0) {
    red_v[warp] = rv;
    red_r[warp] = rr;
    red_c[warp] = rc;
  }
  __syncthreads();
  if (tid == 0) {
    for (int w = 1; w < kLW; ++w) {
      if (red_v[w] > rv || (red_v[w] == rv && red_r[w] < rr)) {
        rv = red_v[w];
        rr = red_r[w];
        rc = red_c[w];
      }
    }
    const int score = rv > B ? (int)((rv - B) >> 2) : 0;
    a.best[p] = make_int2(score, score > 0 ? rr * (R + 1) + rc : 0);
  }
}

// rows of a half for a query: 2, 4, 6 or 8
__host__ __device__ inline int long16_rows(int Q) { return 2 * ((Q + 1023) / 1024); }

// Pairs of all sizes in one launch (largest first), so that small ones fill
// the SMs that large ones leave free.
__global__ void __launch_bounds__(kLT, 2) sw_long16_kernel(LongArgs a) {
  extern __shared__ __align__(16) uint8_t smem[];
  const int64_t item = (int64_t)blockIdx.x;
  if (item >= a.n) return;
  const int32_t p = a.list[item];
  const int Q = a.q_len[p], R = a.r_len[p];
  switch (long16_rows(Q)) {
    case 2: long16_pair<2>(a, item, p, Q, R, smem); break;
    case 4: long16_pair<4>(a, item, p, Q, R, smem); break;
    case 6: long16_pair<6>(a, item, p, Q, R, smem); break;
    default: long16_pair<8>(a, item, p, Q, R, smem); break;
  }
}

// Traceback walk over the long kernels' direction codes (the same rules as
// sw_walk_kernel), one warp per pair.
//
// A walk is a chain of dependent reads.  The warp fetches a tile of 256
// direction words at once: of the threads whose rows the walk passes next,
// the steps around the diagonal from its cell (plus the query and window
// bytes there).  Within the tile the lanes look at 32 cells of the diagonal
// together, and a run of DIAG moves, most of an alignment, is one step of the
// walk; gap moves go one by one.  (One thread per pair read four words at a
// time, and some walk of its warp waited for memory on almost every move: 4.2
// ms for queries of 3 to 4 kb; with tiles but move by move 0.9 ms, 110
// instructions a move; 0.15 ms now.)
constexpr int kTileWords = 256;
constexpr int kTileSteps = 32;  // of a stream: 16 columns a diagonal crosses in it, 9
                                // and more before them, about 5 past (gaps)
constexpr int kTileStreams = kTileWords / kTileSteps;
constexpr int kTileBytes = 256;  // of query and of window, before the cell
constexpr int kWalkWarps = 4;

// P16: the directions are sw_long16_kernel's; else sw_long_kernel's with rpl
// rows per thread.
template <bool P16>
__global__ void __launch_bounds__(kWalkWarps * 32) sw_long_walk_kernel(LongArgs a, int rpl_of) {
  __shared__ __align__(16) uint32_t tile_all[kWalkWarps][kTileWords];
  __shared__ char q_all[kWalkWarps][kTileBytes], w_all[kWalkWarps][kTileBytes];
  __shared__ int lo_all[kWalkWarps][kTileStreams];
  const int wib = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int64_t item = (int64_t)blockIdx.x * kWalkWarps + wib;
  if (item >= a.n) return;  // (no block-wide synchronisation below)
  uint32_t* tile = tile_all[wib];
  char *qs = q_all[wib], *ws = w_all[wib];
  int* lo = lo_all[wib];  // per stream: its first step in the tile
  const int32_t p = a.list[item];
  const int R = a.r_len[p];
  const int rpl = P16 ? 2 * long16_rows(a.q_len[p]) : rpl_of, half = rpl / 2;
  const char* qg = a.qry + a.q_off[p];
  const char* wg = a.ref + a.r_off[p];
  const int S4 = (R + (P16 ? 63 : 31) + 3) & ~3;
  const uint32_t* dirs = a.dirs + a.dir_off[item];
  const int W = R + 1;
  const int2 b = a.best[p];
  int cr = b.y / W, cc = b.y % W;
  int h = b.x;
  // the cell's thread, row in it, and wavefront lane
  int t = cr > 0 ? (cr - 1) / rpl : 0, k = cr > 0 ? (cr - 1) - t * rpl : 0;
  auto lane_of = [&](int tt, int kk) -> int {
    return P16 ? 2 * (tt & 31) + (kk >= half ? 1 : 0) : tt & 31;
  };
  int wl = lane_of(t, k);
  int m = kTileStreams, lo_m = 0;  // its stream in the tile (none yet) and that one's first step
  int rows0 = 0, cols0 = 0;        // the tile's cell
  auto fetch = [&]() {  // the tile from the cell on
    rows0 = cr;
    cols0 = cc;
    __syncwarp();
#pragma unroll
    for (int v = 0; v < kTileWords / 128; ++v) {
      const int at = (v * 32 + lane) * 4, st = at / kTileSteps, tt = t - st;
      // the step at which a diagonal enters thread tt's rows
      const int enter = st == 0 ? cc + wl - 1 : cc - (k + 1 + (st - 1) * rpl) + lane_of(tt, rpl - 1) - 1;
      const int first = max((enter + 8 - (kTileSteps - 1)) & ~3, 0);
      const int s = first + (at & (kTileSteps - 1));
      uint4 x = make_uint4(0, 0, 0, 0);
      if (tt >= 0 && s + 4 <= S4)
        x = __ldcg(reinterpret_cast<const uint4*>(dirs + (int64_t)tt * S4 + s));
      *reinterpret_cast<uint4*>(tile + at) = x;
      if ((at & (kTileSteps - 1)) == 0) lo[st] = first;
    }
    for (int i = lane; i < kTileBytes; i += 32) {
      if (i < cr) qs[i] = qg[cr - 1 - i];
      if (i < cc) ws[i] = wg[cc - 1 - i];
    }
    __syncwarp();
    m = 0;
    lo_m = lo[0];
  };
  // the cell's code (a tile holds at most 128 rows and 160 columns, so its
  // bytes too)
  auto code = [&]() -> uint32_t {
    if (m >= kTileStreams || (uint32_t)(cc + wl - 1 - lo_m) >= (uint32_t)kTileSteps) fetch();
    const uint32_t word = tile[m * kTileSteps + (cc + wl - 1 - lo_m)];
    const int sh = !P16 ? 2 * k : k >= half ? 16 + 2 * (rpl - 1 - k) : 2 * (half - 1 - k);
    return (word >> sh) & 3u;
  };
  enum : int { kNone = 0, kDiag = 1, kUp = 2, kLeft = 3 };
  constexpr uint32_t kUpCode = 1u, kLeftCode = P16 ? 2u : 0u;
  auto dir_of = [](uint32_t c, int hh) -> int {
    if (P16) return c == kUpCode ? kUp : c == kLeftCode ? kLeft : (hh == 0 ? kNone : kDiag);
    return c == 2u ? kDiag : c == kUpCode ? kUp : (hh == 0 ? kNone : kLeft);
  };
  const int ma = a.match, x = a.mismatch, o = a.gap_open, e = a.gap_ext;
  char* qc = a.qcons ? a.qcons + (int64_t)p * a.cons_stride : nullptr;
  char* rc = a.rcons ? a.rcons + (int64_t)p * a.cons_stride : nullptr;
  int d = (cr == 0 || cc == 0) ? kNone : dir_of(code(), h);
  int tick = -1, nref = -1, start = 0;
  // the cell has moved to (cr, cc): its thread, row and lane
  auto moved = [&]() {
    const int tt = (cr - 1) / rpl;
    m += t - tt;
    t = tt;
    k = (cr - 1) - t * rpl;
    wl = lane_of(t, k);
    if (m < kTileStreams) lo_m = lo[m];
  };
  while (d != kNone) {
    if (d == kDiag) {
      // A run of DIAG moves at once: lane i looks at the cell i moves on.
      const int row = cr - lane, col = cc - lane;
      bool diag = false, eq = false;
      char qb = 0, rb = 0;
      if (row >= 1 && col >= 1) {
        const int tt = (row - 1) / rpl, kk = (row - 1) - tt * rpl, mm = m + t - tt;
        const int step = col + lane_of(tt, kk) - 1;
        if (mm < kTileStreams && (uint32_t)(step - lo[mm]) < (uint32_t)kTileSteps) {
          const uint32_t word = tile[mm * kTileSteps + (step - lo[mm])];
          const int sh = !P16 ? 2 * kk : kk >= half ? 16 + 2 * (rpl - 1 - kk) : 2 * (half - 1 - kk);
          diag = ((word >> sh) & 3u) == (P16 ? 0u : 2u);
          qb = qs[rows0 - row];
          rb = ws[cols0 - col];
          const int uq = upcase((uint8_t)qb), ur = upcase((uint8_t)rb);
          eq = uq == ur || uq == 'N' || ur == 'N';
        }
      }
      const uint32_t em = __ballot_sync(0xffffffffu, eq);
      // the lane's cell before its own move (P16: a code of DIAG is NONE at 0)
      const int e0 = __popc(em & ((1u << lane) - 1));
      const int hl = h - ma * e0 - x * (lane - e0);
      const uint32_t stop = ~__ballot_sync(0xffffffffu, diag && (!P16 || hl != 0));
      const int r = stop ? __ffs(stop) - 1 : 32;  // at least 1: the cell itself
      if (lane < r && qc) {
        rc[tick + 1 + lane] = rb;
        qc[tick + 1 + lane] = qb;
      }
      const int er = __popc(r == 32 ? em : em & ((1u << r) - 1));
      h -= ma * er + x * (r - er);
      tick += r;
      nref += r;
      cr -= r;
      cc -= r;
      start = cc + 1;
      if (cr == 0 || cc == 0) break;
      moved();
      d = dir_of(code(), h);
      continue;
    }
    // a gap move
    const bool up = d == kUp;
    ++tick;
    nref += up ? 0 : 1;
    if (lane == 0 && qc) {
      rc[tick] = up ? '-' : ws[cols0 - cc];
      qc[tick] = up ? qs[rows0 - cr] : '-';
    }
    start = cc;
    cr -= up ? 1 : 0;
    cc -= up ? 0 : 1;
    if (cr == 0 || cc == 0) break;
    if (up) moved();
    const uint32_t pc = code();
    // it costs gap_ext when the predecessor itself moved the same way
    h -= (up ? pc == kUpCode : pc == kLeftCode) ? e : o;
    d = dir_of(pc, h);
  }
  if (lane == 0) {
    DevAln out;
    out.score = b.x;
    out.start = start;
    out.end = start + nref;
    out.len = tick + 1;
    a.aln[p] = out;
  }
}

template <int RPL>
int launch_long_rpl(cudaStream_t st, const LongArgs& a, bool prof) {
  const size_t smem = ((2 * (a.max_r + 1) + 15) & ~15) + (size_t)(kLW - 1) * 2 * kRing * 4;
  if (prof)
    sw_long_kernel<RPL, true><<<(unsigned)a.n, kLT, smem, st>>>(a);
  else
    sw_long_kernel<RPL, false><<<(unsigned)a.n, kLT, smem, st>>>(a);
  return 1;
}

}  // namespace

int long_rows_per_lane(int Q) {
  return Q <= 4 * kLT ? 4 : Q <= 8 * kLT ? 8 : Q <= 12 * kLT ? 12 : Q <= 16 * kLT ? 16 : 0;
}

// (and 32 words a thread for the cells sw_long16_kernel puts aside)
int64_t long_slot_words(int R) { return (int64_t)kLT * (((R + 63 + 3) & ~3) + 32); }

int long_bias(int gap_open) { return ((-(16 * gap_open + 1)) + 15) & ~15; }

bool long_prof_ok(int m, int x, int gap_open, int max_q) {
  return 16 * m + 4 <= 127 && 16 * x + 4 >= -128 &&
         16ll * m * max_q + long_bias(gap_open) + 16 < (1ll << 18);
}

static int long16_bias(int gap_open) { return ((-(4 * gap_open + 1)) + 3) & ~3; }

int long16_max_q(int m, int x, int o, int e) {
  if (!(m > 0 && x < 0 && o < 0 && e < 0 && e >= o)) return 0;
  if (4 * m + 3 > 127 || 4 * x + 3 < -128 || o < -4096) return 0;
  // the largest cell, 4 m Q + B + 3, and its gap candidates stay below 2^15
  const int room = 32767 - long16_bias(o) - 4 * (e - o) - 8;
  return room <= 0 ? 0 : room / (4 * m);
}

int launch_sw_long(cudaStream_t st, const LongArgs& args, int rpl, int kind) {
  if (args.n <= 0) return 0;
  // shared memory: window (2 B per column) + rings, 23 KB at the longest window
  if (((2 * (args.max_r + kSel16) + 15) & ~15) + (kLW - 1) * 2 * kRing * 4 > 48 * 1024) return 0;
  LongArgs a = args;
  a.one = 1;
  a.four = 4;
  a.bias = kind == kLong16 ? long16_bias(a.gap_open) : long_bias(a.gap_open);
  if (kind == kLongProf && !long_prof_ok(a.match, a.mismatch, a.gap_open, 256 * rpl)) return 0;
  if (kind == kLong16 && long16_max_q(a.match, a.mismatch, a.gap_open, a.gap_ext) <= 0) return 0;
  const unsigned walks = (unsigned)((a.n + kWalkWarps - 1) / kWalkWarps);
  if (kind == kLong16) {
    const size_t smem = ((2 * (a.max_r + kSel16) + 15) & ~15) + (size_t)(kLW - 1) * kRing16 * 4;
    sw_long16_kernel<<<(unsigned)a.n, kLT, smem, st>>>(a);
    sw_long_walk_kernel<true><<<walks, kWalkWarps * 32, 0, st>>>(a, 0);
    return 2;
  }
  const bool prof = kind == kLongProf;
  const int k = rpl == 4    ? launch_long_rpl<4>(st, a, prof)
                : rpl == 8  ? launch_long_rpl<8>(st, a, prof)
                : rpl == 12 ? launch_long_rpl<12>(st, a, prof)
                : rpl == 16 ? launch_long_rpl<16>(st, a, prof)
                            : 0;
  if (k == 0) return 0;
  sw_long_walk_kernel<false><<<walks, kWalkWarps * 32, 0, st>>>(a, rpl);
  return 2;
}

}  // namespace swift
