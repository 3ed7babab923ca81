// Phase 2: Smith-Waterman with traceback, the semantics of the reference's
// GPU kernel smithWaterman (src/smithWaterman.cu:360-395, 510-645, 911-1026):
//
//   H[i][0] = H[0][j] = 0, every boundary cell has direction NONE
//   s = match if U(q[i-1]) == U(r[j-1]) or either is 'N', else mismatch
//   d = H[i-1][j-1] + s
//   t = H[i-1][j] + (dir[i-1][j] == UP   ? gap_ext : gap_open)
//   l = H[i][j-1] + (dir[i][j-1] == LEFT ? gap_ext : gap_open)
//   H = 0, dir = NONE; d > H -> DIAG; t > H -> UP; l > H -> LEFT (strict)
//
// (the gap penalty depends on the neighbour's own chosen direction; there
// is no separate E/F matrix).  Score = max H; the reported cell is the first
// maximum in row-major order.  The traceback walks directions from that cell
// and stops before a NONE cell or after a cell whose predecessor lies in row
// 0 or column 0; it emits reversed consensus strings from the original
// (not upper-cased) bytes.
//
// Kernel layout: one warp per pair.  Lane t owns query rows t*RPL+1 ..
// t*RPL+RPL and sweeps the window columns one step behind lane t-1 (an
// anti-diagonal wavefront of row strips).  The bottom row's H and its
// downward gap candidate pass to the next lane with one shuffle per step.
// 2-bit directions of the lane's rows are packed per column into shared
// memory; lane 0 walks them for the traceback.
#include <stdlib.h>

#include <mutex>

#include "internal.h"

namespace swift {
namespace {

constexpr int kSwWarps = 4;
enum : uint32_t { kNone = 0, kDiag = 1, kUp = 2, kLeft = 3 };

__device__ __forceinline__ uint32_t upper(uint32_t c) {
  return (c - 'a') < 26u ? c - 'a' + 'A' : c;
}

template <int RPL>
struct DirWord;
template <>
struct DirWord<4> { using T = uint8_t; };
template <>
struct DirWord<8> { using T = uint16_t; };
template <>
struct DirWord<10> { using T = uint32_t; };

// One pair on one warp; base is the warp's shared-memory slice.
//
// CODED (any scoring whose values, times 4, stay in 32 bits: coded_ok): cells
// are 4 * H + code with code 3 NONE, 2 DIAG, 1 UP, 0 LEFT, so one maximum over
// the candidates
//     4 * d + 2, 4 * t + 1, 4 * l, 3
// gives H and the direction with the precedence of the strict updates.  A
// launch of few pairs lasts as long as one pair's chain of steps, which this
// shortens: per row one maximum, a mask, a compare and an add follow the row
// above, where the three compared updates one after another took twice that
// (a batch call of 16 pairs of 100 x 300 79 us, 124 before; of 20,000 0.86 ms,
// 1.25 before; of 20,000 of 250 x 500 4.1 ms, 9.6 before).
template <int RPL, bool CODED>
__device__ __forceinline__ void generic_pair(const SwArgs& a, int64_t pair, uint8_t* base,
                                             int lane) {
  using DW = typename DirWord<RPL>::T;
  const int Q = a.q_len ? a.q_len[pair] : a.Q, R = a.R;
  uint8_t* wsh = base;                                  // R bytes (rounded to 16)
  DW* dirs = reinterpret_cast<DW*>(base + ((R + 15) & ~15));  // (R+1) x 32
  const char* qg = a.q + pair * a.q_stride;
  const char* wg = a.w + pair * a.w_stride;
  for (int c = lane; c < R; c += 32) wsh[c] = (uint8_t)upper((uint8_t)wg[c]);
  constexpr int S = CODED ? 4 : 1;  // a unit of score
  const int m = S * a.match + (CODED ? 2 : 0), x = S * a.mismatch + (CODED ? 2 : 0);
  const int uo = S * a.gap_open + (CODED ? 1 : 0), ue = S * a.gap_ext + (CODED ? 1 : 0);
  const int lo = S * a.gap_open, le = S * a.gap_ext;
  // my rows (those past the query match nothing but N, keep to themselves
  // and stay out of the maximum)
  uint32_t qu[RPL];
  int hprev[RPL], eleft[RPL], best[RPL], bestj[RPL];
  int nrows = Q - lane * RPL;
  nrows = nrows < 0 ? 0 : (nrows > RPL ? RPL : nrows);
#pragma unroll
  for (int k = 0; k < RPL; ++k) {
    int i = lane * RPL + k;
    qu[k] = i < Q ? upper((uint8_t)qg[i]) : 0x100u;
    hprev[k] = 0;
    eleft[k] = lo;  // H[i][0] = 0 with direction NONE
    best[k] = 0;
    bestj[k] = 0;
  }
  __syncwarp();
  int send_h = 0, send_f = uo, diag_h = 0;
  const int steps = R + 31;
  for (int s = 0; s < steps; ++s) {
    int recv_h = __shfl_up_sync(0xffffffffu, send_h, 1);
    int recv_f = __shfl_up_sync(0xffffffffu, send_f, 1);
    if (lane == 0) {
      recv_h = 0;
      recv_f = uo;
    }
    const int j = s - lane + 1;
    if (j >= 1 && j <= R && nrows > 0) {
      const uint32_t wc = wsh[j - 1];
      const bool wn = wc == 'N';
      int hd = diag_h;
      int fu = recv_f;
      uint32_t bits = 0;
#pragma unroll
      for (int k = 0; k < RPL; ++k) {
        const int d = hd + ((qu[k] == wc || qu[k] == 'N' || wn) ? m : x);
        hd = hprev[k];
        if (CODED) {
          const int v = max(max(max(d, eleft[k]), 3), fu);
          const int h = v & ~3, c = v & 3;
          hprev[k] = h;
          fu = h + (c == 1 ? ue : uo);
          eleft[k] = h + (c == 0 ? le : lo);
          if (best[k] < h) {
            best[k] = h;
            bestj[k] = j;
          }
          bits |= (uint32_t)(c ^ 3) << (2 * k);
        } else {
          int v = 0;
          uint32_t dir = kNone;
          if (v < d) { v = d; dir = kDiag; }
          if (v < fu) { v = fu; dir = kUp; }
          if (v < eleft[k]) { v = eleft[k]; dir = kLeft; }
          hprev[k] = v;
          fu = v + (dir == kUp ? ue : uo);
          eleft[k] = v + (dir == kLeft ? le : lo);
          if (best[k] < v) {
            best[k] = v;
            bestj[k] = j;
          }
          bits |= dir << (2 * k);
        }
      }
      dirs[j * 32 + lane] = (DW)bits;
      send_h = hprev[RPL - 1];
      send_f = fu;
    }
    diag_h = recv_h;
  }
  // first maximum in row-major order
  int bh = 0, br = 0x7fffffff, bc = 0;
#pragma unroll
  for (int k = 0; k < RPL; ++k) {
    if (k < nrows && bh < best[k]) {
      bh = best[k];
      br = lane * RPL + k + 1;
      bc = bestj[k];
    }
  }
#pragma unroll
  for (int d = 16; d > 0; d >>= 1) {
    const int oh = __shfl_xor_sync(0xffffffffu, bh, d);
    const int orr = __shfl_xor_sync(0xffffffffu, br, d);
    const int oc = __shfl_xor_sync(0xffffffffu, bc, d);
    if (oh > bh || (oh == bh && orr < br)) {
      bh = oh;
      br = orr;
      bc = oc;
    }
  }
  __syncwarp();
  if (lane != 0) return;
  // The traceback: each move emits its consensus bytes; it ends at a NONE
  // cell or at the border.  Row and column, and the row's lane and place in
  // it, are kept as the walk moves.
  // (consensus strings are optional: coordinates only when the caller passes none)
  const bool cons = a.qcons != nullptr;
  char* qc = cons ? a.qcons + pair * a.cons_stride : nullptr;
  char* rc = cons ? a.rcons + pair * a.cons_stride : nullptr;
  int cr = bh > 0 ? br : 0, cc = bh > 0 ? bc : 0;
  int ln = cr > 0 ? (cr - 1) / RPL : 0, k = cr > 0 ? (cr - 1) % RPL : 0;
  int tick = -1, nref = -1, start = 0;
  while (cr > 0 && cc > 0) {
    const uint32_t dir = ((uint32_t)dirs[cc * 32 + ln] >> (2 * k)) & 3u;
    if (dir == kNone) break;
    const bool up = dir != kLeft, left = dir != kUp;  // row / column move
    ++tick;
    nref += left ? 1 : 0;
    if (cons) {
      rc[tick] = left ? wg[cc - 1] : '-';
      qc[tick] = up ? qg[cr - 1] : '-';
    }
    start = cc;
    cr -= up ? 1 : 0;
    cc -= left ? 1 : 0;
    if (up && --k < 0) {
      k = RPL - 1;
      --ln;
    }
  }
  DevAln out;
  out.score = CODED ? bh >> 2 : bh;
  out.start = start;
  out.end = start + nref;
  out.len = tick + 1;
  a.aln[pair] = out;
}

// 4 times any value of the recurrence stays within 31 bits: scores change by
// at most the largest magnitude a move, over at most Q + R moves
bool coded_ok(const SwArgs& a) {
  const int64_t most = std::max(std::max(std::llabs((long long)a.match), std::llabs((long long)a.mismatch)),
                                std::max(std::llabs((long long)a.gap_open), std::llabs((long long)a.gap_ext)));
  return 4 * most * (a.Q + a.R + 2) < (1ll << 30);
}

// Warps stride over the pairs (the list's length is known on the device
// only, so the grid is capped rather than sized by it).  W warps per block:
// fewer for long windows, whose direction words fill more shared memory.
template <int RPL, int W, bool CODED>
__global__ void __launch_bounds__(W * 32) sw_generic_kernel(SwArgs a, int per_warp_bytes) {
  extern __shared__ __align__(16) uint8_t smem[];
  const int wib = threadIdx.x >> 5, lane = threadIdx.x & 31;
  uint8_t* base = smem + (size_t)wib * per_warp_bytes;
  const int64_t n = a.list ? (int64_t)*a.count : a.n;
  for (int64_t i = (int64_t)blockIdx.x * W + wib; i < n; i += (int64_t)gridDim.x * W) {
    generic_pair<RPL, CODED>(a, a.list ? (int64_t)a.list[i] : i, base, lane);
    __syncwarp();
  }
}

template <int RPL>
int per_warp_bytes(int R) {
  return ((R + 15) & ~15) + (R + 1) * 32 * (int)sizeof(typename DirWord<RPL>::T);
}

constexpr size_t kGenericSmemMax = 200 * 1024;

template <int RPL, int W, bool CODED>
int launch_generic_w(cudaStream_t st, const SwArgs& a, int pw) {
  const size_t smem = (size_t)pw * W;
  // The opt-in above 48 KB is a per-device function attribute: set on every
  // launch (cheap), so a second device or context needs no state here, and
  // always to the most, since another thread's launch may come between.
  if (smem > 48 * 1024 &&
      cudaFuncSetAttribute(sw_generic_kernel<RPL, W, CODED>,
                           cudaFuncAttributeMaxDynamicSharedMemorySize,
                           (int)kGenericSmemMax) != cudaSuccess)
    return SWIFT_E_CUDA;
  int64_t blocks = (a.n + W - 1) / W;
  if (a.list) {  // the list's length is on the device: a few waves stride over it
    int dev = 0, sms = 0;
    if (cudaGetDevice(&dev) == cudaSuccess &&
        cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) == cudaSuccess && sms > 0)
      blocks = std::min<int64_t>(blocks, (int64_t)sms * 16 * 4 / W);
  }
  sw_generic_kernel<RPL, W, CODED><<<(unsigned)blocks, W * 32, smem, st>>>(a, pw);
  return SWIFT_OK;
}

template <int RPL, int W>
int launch_generic_w(cudaStream_t st, const SwArgs& a, int pw) {
  return coded_ok(a) ? launch_generic_w<RPL, W, true>(st, a, pw)
                     : launch_generic_w<RPL, W, false>(st, a, pw);
}

template <int RPL>
int launch_generic(cudaStream_t st, const SwArgs& a, std::string* err) {
  int pw = per_warp_bytes<RPL>(a.R);
  pw = (pw + 15) & ~15;
  int rc;
  if ((size_t)pw * kSwWarps <= kGenericSmemMax)
    rc = launch_generic_w<RPL, kSwWarps>(st, a, pw);
  else if ((size_t)pw * 2 <= kGenericSmemMax)
    rc = launch_generic_w<RPL, 2>(st, a, pw);
  else if ((size_t)pw <= kGenericSmemMax)
    rc = launch_generic_w<RPL, 1>(st, a, pw);
  else {
    *err = "window too long for the on-chip traceback";
    return SWIFT_E_LIMIT;
  }
  if (rc != SWIFT_OK) *err = "generic kernel: shared-memory opt-in failed";
  return rc;
}

}  // namespace

// Per-pair results for swift_sw_batch_noalloc, held in module memory that is
// reserved when the module loads, so that call needs no allocation.  Each
// record is written by the kernel before anything reads it: nothing here has
// to start at zero.  Every caller on a device shares this one array.
__device__ __align__(256) DevAln g_static_aln[kStaticSwPairs];

int static_sw_scratch(int device, DevAln** out, std::string* err) {
  // The symbol's address is looked up once per device, with that device
  // current (the caller has made it so), and kept.
  constexpr int kDevices = 64;
  static std::mutex mu;
  static DevAln* addr[kDevices] = {};
  if (device < 0 || device >= kDevices) {
    *err = "device ordinal outside 0..63";
    return SWIFT_E_ARG;
  }
  std::lock_guard<std::mutex> lock(mu);
  if (!addr[device]) {
    void* p = nullptr;
    const cudaError_t e = cudaGetSymbolAddress(&p, g_static_aln);
    if (e != cudaSuccess) {
      *err = std::string("cudaGetSymbolAddress: ") + cudaGetErrorString(e);
      return SWIFT_E_CUDA;
    }
    addr[device] = static_cast<DevAln*>(p);
  }
  *out = addr[device];
  return SWIFT_OK;
}

int launch_sw(cudaStream_t st, const SwArgs& a, std::string* err) {
  if (a.n <= 0) return SWIFT_OK;
  if (a.Q < 1 || a.Q > kMaxQ || a.R < 1 || a.R > kMaxR) {
    *err = "Smith-Waterman dimensions outside 1..320 x 1..1024";
    return SWIFT_E_LIMIT;
  }
  if (a.Q <= 128) return launch_generic<4>(st, a, err);
  if (a.Q <= 256) return launch_generic<8>(st, a, err);
  return launch_generic<10>(st, a, err);
}

}  // namespace swift

// ---------------------------------------------------------------------------
// Peak of the packed-int16 max-plus instruction (__vimax3_s16x2_relu: the
// three-way max with zero floor of two 16-bit cells), measured on this GPU:
// one full wave of 256-thread blocks, eight independent chains per thread.
// Two cells per instruction is the Smith-Waterman roofline denominator.
namespace swift {
namespace {
constexpr int kCalIters = 4096;
__global__ void __launch_bounds__(256) dpx_calibration_kernel(uint32_t* out, uint32_t seed) {
  uint32_t x[8];
#pragma unroll
  for (int k = 0; k < 8; ++k) x[k] = seed * (threadIdx.x + 1) + k * 0x01010101u;
  const uint32_t c = seed + 0x00010001u;
  for (int it = 0; it < kCalIters; ++it) {
#pragma unroll
    for (int k = 0; k < 8; ++k) x[k] = __vimax3_s16x2_relu(x[k], x[(k + 1) & 7], c);
  }
  uint32_t acc = 0;
#pragma unroll
  for (int k = 0; k < 8; ++k) acc ^= x[k];
  out[blockIdx.x * blockDim.x + threadIdx.x] = acc;
}
}  // namespace

int measure_dpx_peak(cudaStream_t st, int device, double* instr_per_s) {
  int sms = 0;
  if (cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device) != cudaSuccess)
    return SWIFT_E_CUDA;
  const int blocks = sms * 8, threads = 256;
  uint32_t* out = nullptr;
  if (cudaMallocAsync(&out, (size_t)blocks * threads * 4, st) != cudaSuccess) return SWIFT_E_CUDA;
  cudaEvent_t e0, e1;
  cudaEventCreate(&e0);
  cudaEventCreate(&e1);
  double best = 0;
  for (int rep = 0; rep < 4; ++rep) {
    cudaEventRecord(e0, st);
    dpx_calibration_kernel<<<blocks, threads, 0, st>>>(out, 7u + rep);
    cudaEventRecord(e1, st);
    cudaEventSynchronize(e1);
    float ms = 0;
    cudaEventElapsedTime(&ms, e0, e1);
    double ops = (double)blocks * threads * kCalIters * 8.0 / 32.0;  // warp instructions
    if (ms > 0 && rep > 0) best = ops * 32.0 / (ms * 1e-3) > best ? ops * 32.0 / (ms * 1e-3) : best;
  }
  cudaEventDestroy(e0);
  cudaEventDestroy(e1);
  cudaFreeAsync(out, st);
  cudaError_t e = cudaStreamSynchronize(st);
  *instr_per_s = best;  // lane instructions per second
  return e == cudaSuccess ? SWIFT_OK : SWIFT_E_CUDA;
}

}  // namespace swift
