// Shared pieces of the row-streaming mat-vec kernels (gemv_uniform.cu,
// gemv_fused.cu): a warp owns whole rows, the input vector sits piece-major in
// shared memory, 16 bytes of weights per lane and load.
#ifndef HQ_GEMV_ROWS_CUH_
#define HQ_GEMV_ROWS_CUH_
#include <algorithm>
#include <type_traits>

#include "hq_common.cuh"

namespace hq {
namespace rows {

constexpr int kThreads = 512;
constexpr int kWarps = kThreads / 32;
constexpr int kInFlight = 8;            // 16-byte loads per lane in flight
constexpr int kRows = 2;                // adjacent rows a warp works on at a time

// Dynamic shared memory of a launch whose inputs take `need` bytes.  A grid of at most
// one CTA per SM asks for more than half an SM: the next launch starts early, and two
// of its CTAs would otherwise share an SM that the running one leaves free while other
// SMs get none (int4 4096 x 11008, 128 CTAs, back to back 13.6 us, alone on their SMs
// 10.0; 4096 x 28672 28.5 and 19.7; fp16 4096 x 28672 43.7 and 39.3; one CTA per SM
// without the early start takes the same in a graph and 1.6 to 2 us more as calls).
inline size_t smem_request(size_t need, int grid) {
  constexpr size_t kOverHalf = 116 * 1024;
  return grid <= sm_count() && need < kOverHalf ? kOverHalf : need;
}

// How the row pairs are divided: in blocks of 16, pair CTA * 16 + warp goes to a warp first; dealt one by one,
// pair warp * CTAs + CTA; then every CTAs * 16-th.  Dealt, every SM has the same number; in blocks, 4096
// pairs leave 108 of 148 SMs with 32 and 40 with 16 where 28 are even, and 512 pairs use 32 SMs.  us of a
// call among others, blocks -> one by one, int4 (int8): 1024 x 4096 3.9 -> 2.8 (4.8 -> 3.6),
// 1024 x 16384 11.2 -> 7.7 (15.6 -> 13.2), 2368 x 4096 4.1 -> 3.3 (5.6 -> 5.0), 5120 x 5120 8.0 -> 6.7 (9.8 -> 8.5),
// 8192 x 8192 12.0 -> 11.8 (14.7 -> 14.5), 14336 x 4096 11.3 -> 10.0 (14.5 -> 13.0).  Blocks are kept
//  * where they fill the SMs with one CTA each (int4 4096 x 4096 4.30, one by one 4.37), or with two and
//    4-bit rows of up to 3 KiB (8192 x 2048 4.33 and 4.45, 9000 x 4096 6.33 and 6.62, 9000 x 6144 10.64 and
//    10.75), 8-bit ones of 2 (9000 x 2048 6.7 and 6.85; 8192 x 3072 8.01 and 7.84) or fp16 ones of 1 (2 KiB: one
//    by one 1 % less): the rows of a CTA follow one another;
//  * where the last of several rounds is less than a quarter full: it falls to a few CTAs and the next
//    launch starts on the other SMs (10000 x 8192 int4 14.7, one by one 15.8; 49152 x 2048 16.0 and 16.6).
//    From the fourth round on 4-bit rows do that up to half full, when one CTA of each SM has a pair per warp
//    more (32000 x 4096 17.1 and 17.6, 41000 x 2048 13.4 and 14.3); rows of up to 512 bytes from the fifth
//    (32000 x 1024 gains 3 %, 41000 x 1024 loses 6; up to 1 KiB 33000 x 2048 gains 3), 8-bit and fp16 rows never (41000 x 2048 gain 3 and 2 %).
//    In the third round a third full is still few for plain 4-bit rows whose batches of 2 KiB are whole or
//    nearly so (22016 x 4096 12.8 and 13.4, x 8192 23.6 and 24.8; x 2048 9.7 and 9.2, x 6144 22.2 and 20.0).
// A share of consecutive pairs per CTA took registers that the loops need (8 bits 1.05 to 1.1), and so
// does a division that comes as a parameter (int4 in blocks, 4736 x 8192 7.2 us for 7.0, 22016 x 4096 13.9
// for 12.9): each is a kernel of its own.  The plain 8-bit kernel alone is the faster one with parameters (28672 x
// 2048 12.64 us, 12.9 without, 10000 x 1024 4.66 and 4.78; pairs one by one the same).
struct Share {
  int ctas;
  bool dealt;
};
inline Share share_rows(int rows, size_t row_bytes, int bits, bool plain) {
  const int pairs = rows / kRows + (rows % kRows != 0), sms = sm_count();
  const int blocks = pairs / kWarps + (pairs % kWarps != 0);  // CTAs of a pair per warp
  const int ctas = blocks <= sms ? std::min(pairs, sms) : 2 * sms, round = ctas * kWarps;
  const int rounds = pairs / round;  // whole ones
  const bool whole_batches = row_bytes <= 4096 && (row_bytes + 256) % 2048 <= 256;
  double few = 0.25;
  if (bits == 4 && rounds >= 4) few = 0.5;
  if (bits == 4 && rounds == 3 && row_bytes > 512) few = row_bytes > 1024 ? 0.5 : 0.42;
  if (bits == 4 && rounds == 2 && plain && whole_batches) few = 0.34;
  const size_t short_rows = bits == 4 ? 3072 : bits == 8 ? 2048 : 1024;
  const bool in_blocks = blocks <= sms       ? blocks >= 0.85 * sms
                         : blocks <= 2 * sms ? blocks >= 1.65 * sms && row_bytes <= short_rows
                                             : pairs % round < few * round;
  if (in_blocks) return {std::min(blocks, 2 * sms), false};
  return {ctas, true};
}
template <bool DEALT>
__device__ __forceinline__ long long first_row(int warp) {
  return (DEALT ? (long long)warp * gridDim.x + blockIdx.x : (long long)blockIdx.x * kWarps + warp) * kRows;
}

// 4-bit rows of up to 4 KiB: the rows a warp starts with are on their way to L2 before the
// wait for the kernel before and the staging of the inputs.  us of a call among others:
// 4096 x 4096 4.8 -> 4.2, 28672 x 4096 17.0 -> 16.0, 8192 x 8192 12.0 -> 11.9, the two products of an
// MLP block 2048 - 5632 14.8 -> 12.9; few short rows gain a little too (512 x 1024 2.57 -> 2.49).
// Longer rows gain nothing (4096 x 11008 10.13 -> 10.27), and 8-bit rows of the same lengths
// lose: 512 x 1024 2.65 -> 3.01, 4096 x 1024 2.69 -> 3.36, 1024 x 4096 4.67 -> 5.40, 28672 x 4096 21.97 -> 25.5
// (8192 x 2048 alone 5.90 -> 5.05; 8192 x 8192 14.4 -> 17.4).
template <bool DEALT>
__device__ __forceinline__ void prefetch_first_rows(const unsigned char* mat, int rows, size_t row_bytes,
                                                    int lane, int warp) {
  const long long row = first_row<DEALT>(warp) + lane;
  if (row_bytes <= 4096 && lane < kRows && row < rows)
    prefetch_l2(mat + (size_t)row * row_bytes, (uint32_t)row_bytes);
}

__device__ __forceinline__ float sum4(__half2 a0, __half2 a1, __half2 a2, __half2 a3) {
  const float2 f = __half22float2(__hadd2(__hadd2(a0, a1), __hadd2(a2, a3)));
  return f.x + f.y;
}

// 16 bytes of weights of each of R rows against the matching inputs -> one fp32
// partial sum per row; the inputs are read once for the R rows.
// BITS = 16: 8 halves x 8 inputs; 8: 16 int8 x 16 inputs; 4: 32 nibbles x 32 inputs.
// xs points at the chunk's first 16-byte piece of inputs; its further pieces
// follow at a distance of `pitch` pieces (the inputs are stored piece-major so
// that the 32 lanes of a warp, which hold consecutive chunks, read consecutive
// 16-byte words: chunk-major, a chunk's 32 or 64 bytes apart, they would meet in
// the same banks two or four at a time).
template <int BITS, int R>
__device__ __forceinline__ void chunk_dot(const uint4 (&w)[R], const uint4* xs, int pitch,
                                          float (&part)[R]) {
  if (BITS == 16) {
    const uint4 x = xs[0];
#pragma unroll
    for (int r = 0; r < R; r++) {
      // one product per accumulator: summed in fp32 right away
      const float2 f0 = __half22float2(__hmul2(u32_as_half2(w[r].x), u32_as_half2(x.x))),
                   f1 = __half22float2(__hmul2(u32_as_half2(w[r].y), u32_as_half2(x.y))),
                   f2 = __half22float2(__hmul2(u32_as_half2(w[r].z), u32_as_half2(x.z))),
                   f3 = __half22float2(__hmul2(u32_as_half2(w[r].w), u32_as_half2(x.w)));
      part[r] = ((f0.x + f0.y) + (f1.x + f1.y)) + ((f2.x + f2.y) + (f3.x + f3.y));
    }
  } else if (BITS == 8) {
    const uint4 xa = xs[0], xb = xs[pitch];
    const uint32_t x2[8] = {xa.x, xa.y, xa.z, xa.w, xb.x, xb.y, xb.z, xb.w};
    const __half2 off = __float2half2_rn(1152.f);  // 1024 (exponent byte) + 128 (sign flip)
#pragma unroll
    for (int r = 0; r < R; r++) {
      const uint32_t ww[4] = {w[r].x, w[r].y, w[r].z, w[r].w};
      __half2 a0 = __float2half2_rn(0.f), a1 = a0, a2 = a0, a3 = a0;
#pragma unroll
      for (int i = 0; i < 4; i++) {
        const uint32_t t = ww[i] ^ 0x80808080u;
        const __half2 lo = __hsub2(u32_as_half2(__byte_perm(t, 0x64646464u, 0x4140)), off);
        const __half2 hi = __hsub2(u32_as_half2(__byte_perm(t, 0x64646464u, 0x4342)), off);
        if (i & 1) {
          a2 = __hfma2(lo, u32_as_half2(x2[2 * i]), a2);
          a3 = __hfma2(hi, u32_as_half2(x2[2 * i + 1]), a3);
        } else {
          a0 = __hfma2(lo, u32_as_half2(x2[2 * i]), a0);
          a1 = __hfma2(hi, u32_as_half2(x2[2 * i + 1]), a1);
        }
      }
      part[r] = sum4(a0, a1, a2, a3);
    }
  } else {
    // A word holds 8 nibbles = elements 0 .. 7.  (w & 0x000f000f) | 0x64006400 is
    // half2(1024 + e0, 1024 + e4), (w & 0x00f000f0) | 0x64006400 is half2(1024 +
    // 16 e1, 1024 + 16 e5); w >> 8 brings e2, e6 and e3, e7 to the same places.
    // One subtraction of 1024, or one fused x / 16 - 64, leaves the integers,
    // exactly: two logic operations and one fp16 instruction per two weights, no
    // table.  The inputs are staged in the matching order (pair_inputs).
    const __half2 k1024 = __float2half2_rn(1024.f), k16th = __float2half2_rn(0.0625f),
                  km64 = __float2half2_rn(-64.f);
    __half2 a[R][4];
#pragma unroll
    for (int r = 0; r < R; r++) a[r][0] = a[r][1] = a[r][2] = a[r][3] = __float2half2_rn(0.f);
#pragma unroll
    for (int i = 0; i < 4; i++) {
      const uint4 x = xs[i * pitch];
#pragma unroll
      for (int r = 0; r < R; r++) {
        const uint32_t wi = i == 0 ? w[r].x : i == 1 ? w[r].y : i == 2 ? w[r].z : w[r].w;
        const uint32_t hi = wi >> 8;
        const __half2 e04 = __hsub2(u32_as_half2((wi & 0x000f000fu) | 0x64006400u), k1024);
        const __half2 e15 = __hfma2(u32_as_half2((wi & 0x00f000f0u) | 0x64006400u), k16th, km64);
        const __half2 e26 = __hsub2(u32_as_half2((hi & 0x000f000fu) | 0x64006400u), k1024);
        const __half2 e37 = __hfma2(u32_as_half2((hi & 0x00f000f0u) | 0x64006400u), k16th, km64);
        a[r][0] = __hfma2(e04, u32_as_half2(x.x), a[r][0]);
        a[r][1] = __hfma2(e15, u32_as_half2(x.y), a[r][1]);
        a[r][2] = __hfma2(e26, u32_as_half2(x.z), a[r][2]);
        a[r][3] = __hfma2(e37, u32_as_half2(x.w), a[r][3]);
      }
    }
#pragma unroll
    for (int r = 0; r < R; r++) part[r] = sum4(a[r][0], a[r][1], a[r][2], a[r][3]);
  }
}

// 8 consecutive inputs (x0,x1)(x2,x3)(x4,x5)(x6,x7) in the order the 4-bit
// conversion above produces its weights: (x0,x4)(x1,x5)(x2,x6)(x3,x7)
__device__ __forceinline__ uint4 pair_inputs(const uint4& v) {
  return make_uint4(__byte_perm(v.x, v.z, 0x5410), __byte_perm(v.x, v.z, 0x7632),
                    __byte_perm(v.y, v.w, 0x5410), __byte_perm(v.y, v.w, 0x7632));
}

}  // namespace rows
}  // namespace hq
#endif  // HQ_GEMV_ROWS_CUH_
