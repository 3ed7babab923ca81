// swift_sw_batch on the packed 16-bit passes: its pairs, any bytes at any
// alignment, laid out in 16-byte rows and split by their bytes.  Each pair's
// bytes are moved once, by a warp (20,000 pairs of 100 x 300: 12 us beside 204
// us of trace pass and 21 of walk, which writes the strings where the caller
// wants them; the int32 kernel took 1.23 ms).
#include "internal.h"

namespace swift {
namespace {

constexpr int kBatchWarps = 8;

// all four bytes A, C, G or T, either case
__device__ __forceinline__ bool bases4(uint32_t x) {
  const uint32_t u = x & 0xDFDFDFDFu;
  const uint32_t cls = ((u >> 1) ^ (u >> 2)) & 0x03030303u;  // A 0, C 1, G 2, T 3
  const uint32_t t = cls | (cls >> 4);
  return __byte_perm(0x54474341u, 0u, (t & 0x33u) | ((t >> 8) & 0x3300u)) == u;
}

// len bytes at src to a row of `stride` bytes, zero past len; false when one
// is not a base.  The loads are words that hold a byte of [src, src + len).
__device__ __forceinline__ bool row(const char* src, int len, char* dst, int stride, int lane) {
  const uintptr_t ad = (uintptr_t)src;
  const uint32_t* wp = reinterpret_cast<const uint32_t*>(ad & ~(uintptr_t)3);
  const int off = (int)(ad & 3);
  bool ok = true;
  for (int i = 4 * lane; i < stride; i += 128) {
    uint32_t x = 0;
    if (i < len) {
      const uint32_t lo = wp[i >> 2];
      const uint32_t hi = off && i + 4 - off < len ? wp[(i >> 2) + 1] : 0u;
      x = __funnelshift_r(lo, hi, 8 * off);
      const int left = len - i;
      const uint32_t keep = left >= 4 ? ~0u : (1u << (8 * left)) - 1u;
      x &= keep;
      ok &= bases4(x | (0x41414141u & ~keep));
    }
    *reinterpret_cast<uint32_t*>(dst + i) = x;
  }
  return ok;
}

__global__ void __launch_bounds__(kBatchWarps * 32) pack_batch_kernel(BatchArgs a) {
  __shared__ bool plain[kBatchWarps];
  const int wib = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int64_t i0 = (int64_t)blockIdx.x * kBatchWarps, i = i0 + wib;
  bool ok = true;
  if (i < a.n) {
    ok = row(a.q + i * (a.Q + 1), a.Q, a.qbuf + i * a.q_stride, (int)a.q_stride, lane);
    ok &= row(a.w + i * (a.R + 1), a.R, a.wbuf + i * a.w_stride, (int)a.w_stride, lane);
  }
  ok = __all_sync(0xffffffffu, ok);
  if (lane == 0) plain[wib] = ok;
  __syncthreads();
  const int t = threadIdx.x;
  const bool in = t < kBatchWarps && i0 + t < a.n;
  block_append(in && plain[t], (int32_t)(i0 + t), a.fast, a.n_fast);
  block_append(in && !plain[t], (int32_t)(i0 + t), a.gen, a.n_gen);
}

}  // namespace

void launch_pack_batch(cudaStream_t st, const BatchArgs& a) {
  if (a.n <= 0) return;
  pack_batch_kernel<<<(unsigned)((a.n + kBatchWarps - 1) / kBatchWarps), kBatchWarps * 32, 0, st>>>(a);
}

}  // namespace swift
