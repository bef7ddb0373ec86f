// Shared pieces of the row-streaming mat-vec kernels (gemv_uniform.cu,
// gemv_fused.cu): a warp owns whole rows, two adjacent ones at a time, the input vector sits in
// shared memory, 16 bytes of weights per lane and row; the products on mma.sync, through a ring of cp.async copies
// or from registers.
//
// What bounds it: HBM, and for 4 bits the logic pipe (five operations of two cycles for eight weights).  us in
// graphs, fp16 multiply-adds with eight loads per lane -> this form (with RMSNorm and SwiGLU): int4 8192 x 8192 11.9
// -> 9.8 (13.5 -> 11.0), 28672 x 4096 15.6 -> 13.3 (16.8 -> 14.9), 4096 x 14336 11.8 -> 8.2 (12.9 -> 9.7), 4096 x
// 4096 4.5 -> 3.9 (5.2 -> 4.7); int8 8192 x 8192 14.3 -> 13.8 (15.7 -> 13.3), 28672 x 4096 21.6 -> 21.2 (22.8 ->
// 19.9), 4096 x 14336 15.2 -> 11.7 (17.3 -> 13.2), 1024 x 16384 13.0 -> 8.4; fp16 8192 x 8192 22.5 -> 22.8 (24.0 ->
// 23.9), 4096 x 4096 8.5 -> 7.3, 10962 x 1600 8.4 -> 8.1.  Sums of 32 to 64 products were rounded to fp16; now products
// are exact and sums fp32.
#ifndef HQ_GEMV_ROWS_CUH_
#define HQ_GEMV_ROWS_CUH_
#include <limits.h>

#include <algorithm>
#include <type_traits>

#include "hq_common.cuh"

namespace hq {
namespace rows {

constexpr int kThreads = 512;
constexpr int kWarps = kThreads / 32;
constexpr int kRows = 2;                // adjacent rows a warp works on at a time
constexpr int kDepth = 4;               // pieces of 512 bytes of both rows on their way to a warp
constexpr int kSlot = kRows * 512;
constexpr size_t kRing = (size_t)kWarps * kDepth * kSlot;
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
//    (32000 x 1024 gains 3 %, 41000 x 1024 loses 6; up to 1 KiB 33000 x 2048 gains 3), 8-bit and fp16 rows never
//    (41000 x 2048 gain 3 and 2 %).  In the third round a third full is still few for plain 4-bit rows whose
//    batches of 2 KiB are whole or nearly so (22016 x 4096 12.8 and 13.4, x 8192 23.6 and 24.8; x 2048 9.7 and
//    9.2, x 6144 22.2 and 20.0).
// A share of consecutive pairs per CTA took registers that the loops need (8 bits 1.05 to 1.1), and so does a
// division that comes as a parameter (int4 in blocks, 4736 x 8192 7.2 us for 7.0, 22016 x 4096 13.9 for
// 12.9): each is a kernel of its own.  The plain 8-bit kernel alone is the faster one with parameters (28672 x
// 2048 12.64 us, 12.9 without, 10000 x 1024 4.66 and 4.78; pairs one by one the same).
// (Figures of this comment: fp16 multiply-adds, loads into registers.  With the present forms, 1650 layers in graphs: these
// lines take 0.2 to 0.3 % more than the better division of each layer, always one by one 0.2 to 0.5, always blocks 8 to 10.)
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
// Shared memory that a launch of the ring takes besides its inputs, the kernels' static arrays among it; CTAs that fit
// an SM (228 KiB, one of them reserved per CTA).
inline bool ring_fits(size_t input_bytes, int ctas_per_sm) {
  const size_t need = kRing + input_bytes + 128;
  return need <= 227 * 1024 && ctas_per_sm * (need + 1024) <= 228 * 1024;
}
// Whether the rows come through the ring or into registers, eight loads per lane at a time.  us in graphs, weights from
// HBM, registers -> ring, "fused" with RMSNorm and SwiGLU:
//  * where one CTA of the ring fits an SM and two of the registers' form do, a CTA per SM takes the ring, pairs dealt one by one
//    (two per SM and the ring would be two waves): int4 8192 x 28672 25.8 -> 21.3, two waves 25.3, fused 29.6, 24.4 and 29.1;
//    int8 39.1, 38.6 and 39.5, fused 41.7, 40.7 and 44.5.  8 and 16 bits with up to 1.4 or 1.5 pairs per warp, whose second
//    turn is nearly empty, keep two CTAs and the registers (int8 5120 x 27648 26.7 and 30.7, fp16 5072 x 33536 55.8 and 71);
//  * with one CTA per SM the ring, whose first weights are asked for before the inputs are staged: int4 1024 x 4096 3.0 -> 2.6,
//    fused 1024 x 2048 3.4 -> 2.7, int8 768 x 1152 2.42 -> 2.35, 1024 x 16384 9.8 -> 8.4, fp16 1024 x 4096 5.2 -> 4.5.
//    Not plain int4 rows of one or two steps in up to four pairs per SM (1030 x 1024 1.86 -> 2.00), nor those of three and four in
//    blocks (4096 x 4096 3.87 -> 4.10).  Up to 1.1 pairs per SM, too few for lines of their own, the lines
//    of before: rows of more than four steps, 4 bits of eight (the ring would take 0.84 to 0.91 of the time over 250 layers of
//    32 to 600 rows, 1.03 at most);
//  * with two, 4 bits: rows of more than four steps, or two whole rounds of pairs (its requests run on across the ends of
//    rows; 49152 x 1024 9.8 -> 8.2, 22016 x 4096 12.3 -> 10.6, 8192 x 2048 3.75 -> 4.3, 16000 x 2048 5.6 -> 5.9);
//  * 8 bits: rows of more than four steps (28672 x 4096 fused 21.3 -> 19.9), or some whole rounds (15142 x 512 fused 5.1 ->
//    4.5, 49152 x 1024 11.35 -> 10.8; 16000 x 2048 7.6 -> 8.0, 41000 x 2048 15.3 -> 16.4);
//  * 16 bits: the registers where rounds are many or the last one is full, their loads following one another as closely
//    (10962 x 1600 8.1 -> 9.2, 28672 x 4096 fused 38.0 -> 39.9, 8192 x 8192 fused 23.7 -> 25.3; 12288 x 4096 17.9 -> 17.2, fused
//    12288 x 2176 11.8 -> 10.9, 22528 x 1280 11.1 -> 10.7, 9000 x 1024 4.94 -> 4.60).
// Over 1345 layers of 512 to 57344 rows and 1024 to 57344 inputs 0.82 of the time of the fp16 multiply-adds, worst 1.03 (fp16
// 9396 x 8064 24.2 -> 25.0).
inline bool takes_ring(int rows, int steps, int bits, size_t input_bytes, bool plain, Share* share) {
  if (!ring_fits(input_bytes, 1)) return false;
  const int pairs = rows / kRows + (rows % kRows != 0), sms = sm_count();
  const bool two = pairs > sms * kWarps;  // CTAs per SM
  if (two && !ring_fits(input_bytes, 2)) {
    if (bits != 4 && pairs < (bits == 8 ? 1.4 : 1.5) * sms * kWarps) return false;
    *share = {sms, true};
    return true;
  }
  if (!two) {
    if (pairs <= 1.1 * sms) return steps > (bits == 4 ? 8 : 4);
    if (bits != 4 || !plain || steps > 4) return true;
    return steps > 2 ? share->dealt : pairs > 4 * sms;
  }
  const double rounds = pairs / (2.0 * sms * kWarps);
  const int whole = (int)rounds;
  if (bits == 4) return steps > 4 || whole >= 2;
  if (bits == 8) return steps > 4 || whole >= (steps > 3 ? 5 : plain || steps <= 2 ? 1 : 2);
  if (steps <= 4) return plain || whole >= 2;
  if (plain) return share->dealt && rounds < (steps <= 6 ? 2.5 : 1.4);
  if (!share->dealt) return steps <= 6 ? whole >= 2 : whole < 3;
  return rounds - whole < 0.4 && (steps <= 6 ? whole >= 2 : whole == 1);
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

// 16 bytes into the registers of v, if `there`.  Behind a branch the value is another than the one it replaces, and
// the compiler waited for loads of a turn before it asked for the next (8 bits 1.03 -> 0.86 of the time of fp16
// multiply-adds over 530 layers).
__device__ __forceinline__ void load_in_place(uint4& v, const void* at, bool there) {
  asm volatile(
      "{\n .reg .pred p;\n setp.ne.u32 p, %5, 0;\n"
      " @p ld.global.L1::no_allocate.v4.u32 {%0,%1,%2,%3}, [%4];\n}\n"
      : "+r"(v.x), "+r"(v.y), "+r"(v.z), "+r"(v.w)
      : "l"(at), "r"((uint32_t)there));
}

// 16 bytes from global to shared memory; zeros where there are none
__device__ __forceinline__ void copy_16(uint32_t dst, const void* src, bool there) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(there ? 16 : 0) : "memory");
}
template <int PENDING>
__device__ __forceinline__ void wait_copies() {
  asm volatile("cp.async.wait_group %0;" ::"n"(PENDING) : "memory");
}

// D += A B on mma.sync m16n8k16, fp16 products, fp32 sums
__device__ __forceinline__ void mma_16816(float (&d)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3,
                                          uint32_t b0, uint32_t b1) {
  asm("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
      : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
      : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}

// The sums of a warp's two rows.  Lane (g, t) = (lane / 4, lane % 4) feeds what it holds of the first row
// as row g of A, of the second as row g + 8 and its inputs as column g of B: the four lanes of g meet
// in D[g][g] and D[g + 8][g], the other elements are products of one lane's weights and another's inputs that
// nobody reads.  Products are exact and added in fp32.  Two sets of sums, taken in turn, halve the chain of
// instructions that wait for one another; 4 bits: codes in place are numbers 2^-24 q and 2^-20 q, a set for each.
template <int BITS>
struct PairSums {
  static constexpr int kSets = 2;
  float d[kSets][4];
  __device__ __forceinline__ void clear() {
#pragma unroll
    for (int s = 0; s < kSets; s++) d[s][0] = d[s][1] = d[s][2] = d[s][3] = 0.f;
  }
  // The sum of the first row in lane 0, of the second in lane 4.  The diagonal lies in the lanes 0 and 4, 9
  // and 13, 18 and 22, 27 and 31.
  __device__ __forceinline__ float total(int lane) const {
    const bool odd = lane & 4;
    float e[kRows];  // this lane's element of either row
#pragma unroll
    for (int r = 0; r < kRows; r++) {
      e[r] = odd ? d[0][2 * r + 1] : d[0][2 * r];
      const float second = odd ? d[1][2 * r + 1] : d[1][2 * r];
      e[r] = BITS == 4 ? fmaf(e[r], 16777216.f, second * 1048576.f) : e[r] + second;
    }
    float v = (odd ? e[1] : e[0]) + __shfl_xor_sync(0xffffffffu, odd ? e[0] : e[1], 4);
    v += __shfl_xor_sync(0xffffffffu, v, 9);
    return v + __shfl_xor_sync(0xffffffffu, v, 18);
  }
};

// 16-byte pieces of inputs that belong to 16 bytes of weights (a chunk).
template <int BITS>
constexpr int kPieces = 16 / BITS;
// The inputs in shared memory, zeros up to a whole step of 32 chunks, so that the eight lanes of a read, which hold
// consecutive chunks, meet in no bank.  With a ring a chunk's pieces follow one another, turned by
// turn(chunk): copies of 16 bytes from one line to places further apart are slow (int4 1024 x 4096 4.0 us for 2.5).  Else
// the first pieces of a step's chunks lie together, then the second, ...: a read's address is a constant further on (int4
// 16000 x 2048 5.5 us, turned 6.2).
template <int BITS>
constexpr int kStepBytes = 32 * 16 * kPieces<BITS>;
template <int BITS>
__device__ __forceinline__ int turn(int chunk) {
  return kPieces<BITS> == 4 ? (chunk >> 1) & 3 : kPieces<BITS> == 2 ? (chunk >> 2) & 1 : 0;
}
// where piece i of the vector lies
template <int BITS, bool RING>
__device__ __forceinline__ int input_at(int i) {
  const int chunk = i / kPieces<BITS>, piece = i % kPieces<BITS>;
  return RING ? i ^ turn<BITS>(chunk) : (chunk / 32 * kPieces<BITS> + piece) * 32 + chunk % 32;
}
// piece Q of a lane's chunk, from its place `at` in a step (input_at of the lane's first piece)
template <int BITS, bool RING, int Q>
__device__ __forceinline__ uint4 input_piece(const uint4* step, int at) {
  return RING ? step[at ^ Q] : step[at + 32 * Q];
}
template <int BITS>
__host__ __device__ constexpr int input_steps(int n) {
  return (int)(((size_t)n * 2 + kStepBytes<BITS> - 1) / kStepBytes<BITS>);
}
template <int BITS>
inline size_t input_bytes(int n) { return (size_t)input_steps<BITS>(n) * kStepBytes<BITS>; }

// 8 consecutive inputs (x0,x1)(x2,x3)(x4,x5)(x6,x7) in the order the 4-bit
// conversion above produces its weights: (x0,x4)(x1,x5)(x2,x6)(x3,x7)
__device__ __forceinline__ uint4 pair_inputs(const uint4& v) {
  return make_uint4(__byte_perm(v.x, v.z, 0x5410), __byte_perm(v.x, v.z, 0x7632),
                    __byte_perm(v.y, v.w, 0x5410), __byte_perm(v.y, v.w, 0x7632));
}

// Brings the input vector to shared memory, behind the wait for the kernel before: ask() before the warp's first
// weights (behind those it would wait for all of them: int4 4096 x 14336 with RMSNorm and SwiGLU 9.8 -> 11.7 us), then
// every thread turns its own pieces, in(i) to out(i, piece).  With a ring they come by cp.async (held in registers they
// cost the loops theirs: int8 41000 x 2048 14.5 -> 16.0 us), else by loads, which are there sooner (9000 x 1024 int4
// 2.9 and 3.6).
template <int BITS, bool RING>
struct Inputs {
  const __half* vec;
  __half* xs;
  int n, tid;
  unsigned site;
  __device__ __forceinline__ bool in_vector(const uint4* at) const {
    return HQ_IN_BOUNDS(at, 16, vec, (size_t)n * 2, site);
  }
  __device__ __forceinline__ void ask() const {
    const int pieces = input_steps<BITS>(n) * (kStepBytes<BITS> / 16);
    const uint32_t to = (uint32_t)__cvta_generic_to_shared(xs);
    for (int i = RING ? tid : n / 8 + tid; i < pieces; i += kThreads) {
      const uint4* at = reinterpret_cast<const uint4*>(vec) + i;
      if (RING) copy_16(to + (uint32_t)input_at<BITS, RING>(i) * 16u, at, i < n / 8 && in_vector(at));
      else reinterpret_cast<uint4*>(xs)[input_at<BITS, RING>(i)] = make_uint4(0, 0, 0, 0);
    }
    if (RING) asm volatile("cp.async.commit_group;" ::: "memory");
  }
  __device__ __forceinline__ void arrived() const {
    if (RING) wait_copies<kDepth>();
  }
  __device__ __forceinline__ uint4 in(int i) const {
    if (RING) return reinterpret_cast<const uint4*>(xs)[input_at<BITS, RING>(i)];
    const uint4* at = reinterpret_cast<const uint4*>(vec) + i;
    return in_vector(at) ? ld_dependent_u4(at) : make_uint4(0, 0, 0, 0);
  }
  // stored (4 bits: in the order of their conversion) and added to `sum`
  __device__ __forceinline__ void out(int i, const uint4& v, float& sum) const {
    reinterpret_cast<uint4*>(xs)[input_at<BITS, RING>(i)] = BITS == 4 ? pair_inputs(v) : v;
    const float2 f0 = __half22float2(u32_as_half2(v.x)), f1 = __half22float2(u32_as_half2(v.y)),
                 f2 = __half22float2(u32_as_half2(v.z)), f3 = __half22float2(u32_as_half2(v.w));
    sum += ((f0.x + f0.y) + (f1.x + f1.y)) + ((f2.x + f2.y) + (f3.x + f3.y));
  }
};

template <int OFFSET>
__device__ __forceinline__ uint4 lds_piece(uint32_t at) {
  uint4 v;
  asm volatile("ld.shared.v4.u32 {%0,%1,%2,%3}, [%4+%5];"
               : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w)
               : "r"(at), "n"(OFFSET)
               : "memory");
  return v;
}

// 16 bytes of weights of each of two rows against the matching inputs.
// BITS = 16: 8 halves x 8 inputs; 8: 16 int8 x 16 inputs; 4: 32 nibbles x 32 inputs.
// xs: the inputs of the step, the lane's first piece at `first`.
// The whole warp takes part; past a row's end the inputs are zero.
template <int BITS, bool RING>
__device__ __forceinline__ void chunk_mma(const uint4 (&w)[kRows], const uint4* xs, int first,
                                          PairSums<BITS>& sums) {
  const uint32_t wa[4] = {w[0].x, w[0].y, w[0].z, w[0].w}, wb[4] = {w[1].x, w[1].y, w[1].z, w[1].w};
  if constexpr (BITS == 16) {
    const uint4 x = input_piece<BITS, RING, 0>(xs, first);
    mma_16816(sums.d[0], wa[0], wb[0], wa[1], wb[1], x.x, x.y);
    mma_16816(sums.d[1], wa[2], wb[2], wa[3], wb[3], x.z, x.w);
  } else if constexpr (BITS == 8) {
    const __half2 off = __float2half2_rn(1152.f);  // 1024 (exponent byte) + 128 (sign flip)
    auto halves = [&](uint32_t v, uint32_t (&h)[2]) {
      const uint32_t f = v ^ 0x80808080u;
      h[0] = half2_as_u32(__hsub2(u32_as_half2(__byte_perm(f, 0x64646464u, 0x4140)), off));
      h[1] = half2_as_u32(__hsub2(u32_as_half2(__byte_perm(f, 0x64646464u, 0x4342)), off));
    };
    const uint4 x[2] = {input_piece<BITS, RING, 0>(xs, first), input_piece<BITS, RING, 1>(xs, first)};
#pragma unroll
    for (int i = 0; i < 4; i++) {
      uint32_t a[2], b[2];
      halves(wa[i], a);
      halves(wb[i], b);
      const uint4& xi = x[i / 2];
      mma_16816(sums.d[i % 2], a[0], b[0], a[1], b[1], i % 2 ? xi.z : xi.x, i % 2 ? xi.w : xi.y);
    }
  } else {
    // A word holds 8 nibbles = elements 0 .. 7.  In (w & 0x000f000f) the elements 0 and 4 are the
    // numbers 2^-24 e (fp16 below its normal range), in (w & 0x00f000f0) 1 and 5 are 2^-20 e; w >> 8 brings 2, 6
    // and 3, 7 to the same places: five operations for eight weights, where integers of full size took
    // four subtractions more and fp16 multiply-adds eight in all.  The inputs are staged in the
    // matching order (pair_inputs).
    auto word = [&](uint32_t a, uint32_t b, const uint4& x) {
      const uint32_t ha = a >> 8, hb = b >> 8;
      mma_16816(sums.d[0], a & 0x000f000fu, b & 0x000f000fu, ha & 0x000f000fu, hb & 0x000f000fu, x.x, x.z);
      mma_16816(sums.d[1], a & 0x00f000f0u, b & 0x00f000f0u, ha & 0x00f000f0u, hb & 0x00f000f0u, x.y, x.w);
    };
    word(wa[0], wb[0], input_piece<BITS, RING, 0>(xs, first));
    word(wa[1], wb[1], input_piece<BITS, RING, 1>(xs, first));
    word(wa[2], wb[2], input_piece<BITS, RING, 2>(xs, first));
    word(wa[3], wb[3], input_piece<BITS, RING, 3>(xs, first));
  }
}

// The row pairs row0, row0 + stride, ... of a warp, a pair at a time: begin() asks for the first weights,
// run_rows() multiplies and calls finish(row0, total), see PairSums::total.
// RING: 512 bytes of each row at a time come by cp.async, up to four such pieces ahead, across the ends of
// the rows and from before the inputs are staged; every lane reads what it copied itself.  Else eight 16-byte
// loads per lane and turn, or (fp16, few registers besides them) each piece's next loads behind its product (fused rows
// 1.05 -> 0.92 of the time of fp16 multiply-adds over 190 layers; plain ones 0.93 -> 0.92; 4 and 8 bits spill).
template <int BITS, bool RING>
struct PairStream {
  const unsigned char* mat;
  uint32_t row0, stride, rows;  // (below 2^31 + stride)
  int lane, chunks, steps;      // 16-byte chunks of a row, 32 of them a step
  size_t row_bytes;
  unsigned site;
  // ring: this lane's place in it, the step that is requested next
  uint32_t mine, next_row;
  int left, run;                // chunks of the row from this lane's on; steps of the pair
  const unsigned char *src0, *src1;

  __device__ __forceinline__ PairStream(const unsigned char* mat_, long long first, int stride_, int rows_, int n,
                                        unsigned char* ring, int lane_, unsigned site_)
      : mat(mat_), row0((uint32_t)first), stride((uint32_t)stride_), rows((uint32_t)rows_), lane(lane_),
        chunks((int)((size_t)n * BITS / 128)), steps(input_steps<BITS>(n)), row_bytes((size_t)n * BITS / 8), site(site_),
        mine((uint32_t)__cvta_generic_to_shared(ring) + (uint32_t)lane_ * 16u), next_row((uint32_t)first) {}
  __device__ __forceinline__ bool in_matrix(const unsigned char* at) const {
    return HQ_IN_BOUNDS(at, 16, mat, (size_t)rows * row_bytes, site);
  }
  __device__ __forceinline__ void aim() {
    if (next_row < rows) {
      src0 = mat + (size_t)next_row * row_bytes + lane * 16;
      src1 = next_row + 1 < rows ? src0 + row_bytes : src0;  // (behind the last row: its sum goes nowhere)
      left = chunks - lane;
      run = steps;
    } else {
      src0 = src1 = mat;
      left = INT_MIN / 2;
      run = INT_MAX;
    }
  }
  // what is past a row's end is zeros
  __device__ __forceinline__ void copy(uint32_t dst, const unsigned char* at) const {
    copy_16(dst, at, left > 0 && in_matrix(at));
  }
  __device__ __forceinline__ void request(uint32_t slot) {
    copy(mine + slot, src0);
    copy(mine + slot + 512, src1);
    src0 += 512;
    src1 += 512;
    left -= 32;
    if (--run == 0) {
      next_row += stride;
      aim();
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  }
  __device__ __forceinline__ void begin() {
    if constexpr (RING) {
      aim();
#pragma unroll
      for (int d = 0; d < kDepth; d++) request(d * kSlot);
    }
  }
  // xs: the inputs
  template <class Finish>
  __device__ __forceinline__ void run_rows(const __half* xs, Finish finish) {
    const uint4* const x0 = reinterpret_cast<const uint4*>(xs);
    const int first = input_at<BITS, RING>(lane * kPieces<BITS>);
    if constexpr (RING) {
      uint32_t slot = 0;
      for (; row0 < rows; row0 += stride) {
        PairSums<BITS> sums;
        sums.clear();
        const uint4* x = x0;
        for (int s = 0; s < steps; s++) {
          wait_copies<kDepth - 1>();
          const uint4 w[kRows] = {lds_piece<0>(mine + slot), lds_piece<512>(mine + slot)};
          chunk_mma<BITS, RING>(w, x, first, sums);
          request(slot);  // behind the products: the slot has been read
          slot = (slot + kSlot) & (kDepth * kSlot - 1);
          x += kStepBytes<BITS> / 16;
        }
        finish(row0, sums.total(lane));
      }
    } else {
      constexpr int kPerRow = 4;
      constexpr bool kTurns = BITS == 16;
      for (; row0 < rows; row0 += stride) {
        const unsigned char* src = mat + (size_t)row0 * row_bytes;
        PairSums<BITS> sums;
        sums.clear();
        uint4 w[kPerRow][kRows];
        auto load = [&](int u, int s) {
          const int c = s * 32 + lane;
#pragma unroll
          for (int r = 0; r < kRows; r++) {
            const unsigned char* at = src + (size_t)r * row_bytes + (size_t)c * 16;
            const bool there = c < chunks && row0 + r < rows && in_matrix(at);
            w[u][r] = make_uint4(0, 0, 0, 0);  // a row past the end contributes zeros
            if constexpr (BITS == 4) {
              if (there) w[u][r] = ld_ordered_stream_u4(at);
            } else {
              load_in_place(w[u][r], at, there);
            }
          }
        };
        if (kTurns) {
#pragma unroll
          for (int u = 0; u < kPerRow; u++) load(u, u);
        }
        for (int s0 = 0; s0 < steps; s0 += kPerRow) {
          if (!kTurns) {
#pragma unroll
            for (int u = 0; u < kPerRow; u++) load(u, s0 + u);
          }
#pragma unroll
          for (int u = 0; u < kPerRow; u++) {
            if (s0 + u >= steps) break;
            chunk_mma<BITS, RING>(w[u], x0 + (s0 + u) * (kStepBytes<BITS> / 16), first, sums);
            if (kTurns && s0 + u + kPerRow < steps) load(u, s0 + u + kPerRow);
          }
        }
        finish(row0, sums.total(lane));
      }
    }
  }
};

}  // namespace rows
}  // namespace hq
#endif  // HQ_GEMV_ROWS_CUH_
