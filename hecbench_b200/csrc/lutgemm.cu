// LUT-GEMM binary-coding mat-vec (nqmv / nqmv_bias) for sm_100a.
//
// Layouts (lut-gemm-cuda/nQWeight_fp16.h:24-26, main.cu:118-134):
//   bW     uint32[K/32][nb][M]   bit t of a word <-> input k = 32*row + t, 1 => +1
//   alpha  half[K/group][nb][M]
//   q_bias half[K/group][M]      (nullable)
//   out[m] = sum_g [ q_bias[g][m]*sum_{k in g} x_k
//                    + sum_b alpha[g][b][m] * sum_{k in g} (2*bit_b[k][m]-1)*x_k ]
//
// Like the reference (mv_fp16.h:133-227) the +-sums over 8 inputs are looked up
// by bit-plane byte in a table built from x, but:
//  * a CTA of 512 threads owns a K tile of 128 inputs (4 packed rows; 64 inputs
//    for alpha groups of 192, 320, ... inputs) and a range of columns; lane
//    (c,j) of a warp handles byte j of the words of columns 4c..4c+3 and reads
//    replica c of table (row, j): the 16 tables are stored with one 256-byte
//    line per (row pair, byte value) holding [row parity][replica c][byte-lane
//    j], so every lane of a warp reads its own bank - no lookup ever conflicts
//    - and, the table block sitting at a FIXED address of the shared window,
//    the address of a lookup is ONE byte-permute of the packed word and a
//    per-lane constant, plus an immediate offset that selects the row;
//  * shared memory carries the lookups and nothing else: packed words, alphas
//    and bias go from global memory straight into registers (128-bit streaming
//    loads, the four lanes of a column quad reading the same 16 bytes), one
//    column step ahead of their use, and the first step is requested before
//    the tables are built;
//  * table entries and all sums are fp32 (the reference uses fp16 throughout
//    and half2 atomics on the output);
//  * the four lanes of a column quad are combined with two shuffles, each CTA
//    adds its tile's partial sums to an fp32 scratch row with one 16-byte
//    vector reduction per column quad, and the last CTA of each column range to
//    finish converts that range of the scratch to fp16, stores the output and
//    re-zeroes the scratch.
#include <algorithm>
#include <cstdlib>
#include <mutex>

#include "hq_common.cuh"

namespace hq {
namespace {

// CTA shapes: 512 threads with a 128-input tile (one CTA per SM), or 256 threads
// with a 64-input tile and two CTAs per SM - the two then run out of phase, one
// streaming packed words while the other builds its tables.
// Shared-window address at which a CTA's dynamic region starts: the 1 KiB the
// system reserves per CTA (the kernels have no static shared memory).  The
// host checks the device attribute before launching; kSlack bytes of padding
// absorb a start up to kSlack later.
constexpr int kDynBase = 1024;
constexpr int kSlack = 256;
// completion counters at the end of the workspace: one per column range
constexpr int kCounterWords = 64;

// Compile-time layout of one variant.  TR: packed rows (32 inputs each) per K
// tile.  Dynamic shared memory:
//   [flag 16 B][build scratch: compact tables + inputs][padding][tables TR/2 x 64 KiB]
// The tables start at the FIXED shared-window address kLutImm so that the
// address of a lookup is a byte-permute plus an immediate.
template <int TR>
struct Layout {
  static constexpr int kCompactWords = TR * 256 * 4;  // [row][byte value][j]
  static constexpr int kBuildBytes = kCompactWords * 4 + TR * 32 * 4;
  static constexpr int kFlagBytes = 16;
  static constexpr int kLutBytes = (TR / 2) * 65536;
  static constexpr int kLutImm = (kDynBase + kSlack + kFlagBytes + kBuildBytes + 255) / 256 * 256;
  static constexpr int kSmem = kLutImm - kDynBase + kLutBytes;
  static_assert(kSmem <= 227 * 1024, "shared memory budget");
};

__device__ __forceinline__ void red_add_v4_f32(float* addr, float a, float b, float c, float d) {
  asm volatile("red.global.add.v4.f32 [%0], {%1, %2, %3, %4};" ::"l"(addr), "f"(a), "f"(b), "f"(c),
               "f"(d)
               : "memory");
}
template <int IMM>
__device__ __forceinline__ float lds_f32_imm(uint32_t addr) {
  // not volatile: the tables are constant once built, so the scheduler is free
  // to batch these loads
  float v;
  asm("ld.shared.f32 %0, [%1+%2];" : "=f"(v) : "r"(addr), "n"(IMM));
  return v;
}
// One launch handles NB bit planes b0 .. b0+NB-1 of nb_total (more planes than
// fit the register budget are split over launches that accumulate into the
// same scratch row; only the last one converts it).  RPG: packed rows that
// share one alpha group inside a tile.  counters: one completion counter per
// column range (per_range != 0) or a single one.
template <int TR, int NB, int RPG, int kThreads>
__global__ void __launch_bounds__(kThreads, (kThreads == 256 ? 2 : 1))
lutgemm_kernel(const uint32_t* bW, const __half* alpha,
               const __half* q_bias, const __half* x,
               __half* __restrict__ out, float* __restrict__ ws, unsigned* __restrict__ counters,
               int M, int K, int rows_per_group, int cols_per_cta, int nb_total, int b0,
               int finalize, int per_range) {
  using L = Layout<TR>;
  constexpr int kWarps = kThreads / 32;
  constexpr int kGroups = TR / RPG;
  constexpr int kLutImm = L::kLutImm;
  extern __shared__ __align__(16) unsigned char dsm[];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const uint32_t dsm_addr = (uint32_t)__cvta_generic_to_shared(dsm);
  // the host has checked where the dynamic region starts; never taken
  if (dsm_addr < (uint32_t)kDynBase || dsm_addr > (uint32_t)(kDynBase + kSlack)) return;
  unsigned char* lut = dsm + ((uint32_t)kLutImm - dsm_addr);
  unsigned* s_last = reinterpret_cast<unsigned*>(dsm);
  float* compact = reinterpret_cast<float*>(dsm + L::kFlagBytes);
  float* xs = compact + L::kCompactWords;  // the tile's inputs
  const int tile = blockIdx.y;
  const int row0 = tile * TR;  // first packed row of the tile
  const int total_rows = K >> 5;
  const int nrows = min(TR, total_rows - row0);
  const int m_begin = blockIdx.x * cols_per_cta;
  const int m_end = min(M, m_begin + cols_per_cta);
  const int g0 = row0 / rows_per_group;  // alpha group of the tile's first row

  // the next kernel of the stream may become resident while this grid drains;
  // nothing is read or written before every earlier kernel has completed.  Back to
  // back this takes 2 to 3 us off a call: 12288 x 12288, 3 planes, 30.7 -> 28.4 us,
  // 4096 x 4096 10.3 -> 7.8, 1024 x 1024 7.9 -> 5.4
  pdl_launch_dependents();
  pdl_wait();
  // ---- stage the tile's inputs (zero beyond K) ----
  if (tid < TR * 32) {
    const int k = row0 * 32 + tid;
    xs[tid] = (k < K && HQ_IN_BOUNDS(x + k, 2, x, (size_t)K * 2, 206)) ? __half2float(ld_dependent_f16(x + k)) : 0.f;
  }
  // ---- column steps of this warp: step s handles columns m0 + s*kWarps*32 ..+3 ----
  const int j = lane & 3;   // byte of the word this lane looks up
  const int cq = lane >> 2; // column quad inside the 32-column step
  const int m0 = m_begin + warp * 32 + cq * 4;
  const int nsteps = (m_end - (m_begin + warp * 32) + kWarps * 32 - 1) / (kWarps * 32);
  const uint32_t* src0 = bW + ((size_t)row0 * nb_total + b0) * M + m0;

  uint4 wv[TR][NB];
  uint2 av[kGroups][NB + 1];
#pragma unroll
  for (int r = 0; r < TR; r++)
#pragma unroll
    for (int b = 0; b < NB; b++) wv[r][b] = make_uint4(0, 0, 0, 0);
#pragma unroll
  for (int gi = 0; gi < kGroups; gi++)
#pragma unroll
    for (int b = 0; b <= NB; b++) av[gi][b] = make_uint2(0, 0);

  // packed words of row r for the step whose first column (for this quad) is m
  // extents of the caller's buffers, used only by the index-checked build
  const size_t bw_bytes = (size_t)total_rows * nb_total * M * 4;
  const size_t alpha_bytes = (size_t)(total_rows / rows_per_group) * nb_total * M * 2;
  const size_t bias_bytes = (size_t)(total_rows / rows_per_group) * M * 2;
  (void)bw_bytes; (void)alpha_bytes; (void)bias_bytes;
  auto load_row = [&](int r, int m) {
    if (r < nrows) {
#pragma unroll
      for (int b = 0; b < NB; b++) {
        const uint32_t* src = src0 + (size_t)(r * nb_total + b) * M + (m - m0);
        if (HQ_IN_BOUNDS(src, 16, bW, bw_bytes, 201)) wv[r][b] = ld_ordered_stream_u4(src);
      }
    }
  };
  auto load_group = [&](int gi, int m) {
    if (gi * RPG < nrows) {
      const int g = g0 + gi;
#pragma unroll
      for (int b = 0; b < NB; b++) {
        const __half* src = alpha + ((size_t)g * nb_total + b0 + b) * M + m;
        if (HQ_IN_BOUNDS(src, 8, alpha, alpha_bytes, 202)) av[gi][b] = ld_ordered_u2(src);
      }
      if (q_bias != nullptr && HQ_IN_BOUNDS(q_bias + (size_t)g * M + m, 8, q_bias, bias_bytes, 203))
        av[gi][NB] = ld_ordered_u2(q_bias + (size_t)g * M + m);
    }
  };
  if (nsteps > 0 && m0 < m_end) {
#pragma unroll
    for (int r = 0; r < TR; r++) load_row(r, m0);
#pragma unroll
    for (int gi = 0; gi < kGroups; gi++) load_group(gi, m0);
  }
  __syncthreads();

  // ---- phase A: thread = (byte value, some of the rows); signed sums of 8 inputs ----
  {
    constexpr int kRowSets = kThreads / 256;      // threads per byte value
    constexpr int kRowsEach = TR / kRowSets;      // rows per thread
    const int bv = tid & 255, rp = tid >> 8;
    uint32_t sgn[8];
#pragma unroll
    for (int t = 0; t < 8; t++) sgn[t] = ((bv >> t) & 1) ? 0u : 0x80000000u;
#pragma unroll
    for (int rr = 0; rr < kRowsEach; rr++) {
      const int r = rp * kRowsEach + rr;
      float v[4];
#pragma unroll
      for (int jj = 0; jj < 4; jj++) {
        const float4 xa = *reinterpret_cast<const float4*>(xs + r * 32 + jj * 8);
        const float4 xb = *reinterpret_cast<const float4*>(xs + r * 32 + jj * 8 + 4);
        const float s0 = __uint_as_float(__float_as_uint(xa.x) ^ sgn[0]) +
                         __uint_as_float(__float_as_uint(xa.y) ^ sgn[1]);
        const float s1 = __uint_as_float(__float_as_uint(xa.z) ^ sgn[2]) +
                         __uint_as_float(__float_as_uint(xa.w) ^ sgn[3]);
        const float s2 = __uint_as_float(__float_as_uint(xb.x) ^ sgn[4]) +
                         __uint_as_float(__float_as_uint(xb.y) ^ sgn[5]);
        const float s3 = __uint_as_float(__float_as_uint(xb.z) ^ sgn[6]) +
                         __uint_as_float(__float_as_uint(xb.w) ^ sgn[7]);
        v[jj] = (s0 + s1) + (s2 + s3);
      }
      *reinterpret_cast<float4*>(compact + (r * 256 + bv) * 4) = make_float4(v[0], v[1], v[2], v[3]);
    }
  }
  __syncthreads();
  // ---- phase B: replicate each (row, byte) entry 8 times into its table line ----
  // line (row pair p, byte b) at lut + p*65536 + b*256; inside: [row parity][c][j] floats
  {
    const int c = lane & 7, bl = lane >> 3;
#pragma unroll 4
    for (int it = 0; it < TR * 256 / (kWarps * 4); it++) {
      const int e = (it * kWarps + warp) * 4 + bl;  // row*256 + byte
      const int r = e >> 8, b = e & 255;
      const float4 v = *reinterpret_cast<const float4*>(compact + e * 4);
      *reinterpret_cast<float4*>(lut + (r >> 1) * 65536 + b * 256 + (r & 1) * 128 + c * 16) = v;
    }
  }
  __syncthreads();

  // ---- lookup phase ----
  // lookup of byte value b in row r: [byteperm(word, lane*4, sel) + kLutImm + (r>>1)*65536 + (r&1)*128]
  const uint32_t hi = (uint32_t)(lane * 4);
  const uint32_t sel = 0x7604u | ((uint32_t)j << 4);

  // bias uses the all-ones entry (byte 255): sum of this lane's 8 inputs per row
  float ones[kGroups];
#pragma unroll
  for (int gi = 0; gi < kGroups; gi++) {
    float o = 0.f;
#pragma unroll
    for (int r = gi * RPG; r < (gi + 1) * RPG; r++)
      o += *reinterpret_cast<const float*>(lut + (r >> 1) * 65536 + 255 * 256 + (r & 1) * 128 +
                                           lane * 4);
    ones[gi] = o;
  }

  for (int s = 0; s < nsteps; s++) {
    const int m = m0 + s * (kWarps * 32);
    const bool active = m < m_end;
    const int m_next = m + kWarps * 32;
    const bool next = (s + 1 < nsteps) && m_next < m_end;
    float acc[4] = {0.f, 0.f, 0.f, 0.f};
    if (active) {
#pragma unroll
      for (int gi = 0; gi < kGroups; gi++) {
        float t[NB][4];
#pragma unroll
        for (int rr = 0; rr < RPG; rr++) {
          const int r = gi * RPG + rr;
#pragma unroll
          for (int b = 0; b < NB; b++) {
            const uint32_t w4[4] = {wv[r][b].x, wv[r][b].y, wv[r][b].z, wv[r][b].w};
#pragma unroll
            for (int c = 0; c < 4; c++) {
              const uint32_t a = __byte_perm(w4[c], hi, sel);
              float v;
              if (r == 0) v = lds_f32_imm<kLutImm>(a);
              else if (r == 1) v = lds_f32_imm<kLutImm + 128>(a);
              else if (r == 2) v = lds_f32_imm<kLutImm + 65536>(a);
              else v = lds_f32_imm<kLutImm + 65536 + 128>(a);
              t[b][c] = (rr == 0) ? v : t[b][c] + v;
            }
          }
          if (next) load_row(r, m_next);  // the registers of this row are free again
        }
        if (gi * RPG < nrows) {  // rows past the end of K have no alpha
#pragma unroll
          for (int b = 0; b < NB; b++) {
            const float2 a01 = __half22float2(u32_as_half2(av[gi][b].x));
            const float2 a23 = __half22float2(u32_as_half2(av[gi][b].y));
            acc[0] = fmaf(a01.x, t[b][0], acc[0]);
            acc[1] = fmaf(a01.y, t[b][1], acc[1]);
            acc[2] = fmaf(a23.x, t[b][2], acc[2]);
            acc[3] = fmaf(a23.y, t[b][3], acc[3]);
          }
          if (q_bias != nullptr) {
            const float2 b01 = __half22float2(u32_as_half2(av[gi][NB].x));
            const float2 b23 = __half22float2(u32_as_half2(av[gi][NB].y));
            acc[0] = fmaf(b01.x, ones[gi], acc[0]);
            acc[1] = fmaf(b01.y, ones[gi], acc[1]);
            acc[2] = fmaf(b23.x, ones[gi], acc[2]);
            acc[3] = fmaf(b23.y, ones[gi], acc[3]);
          }
        }
        if (next) load_group(gi, m_next);
      }
    }
    // combine the four byte lanes of each column quad
#pragma unroll
    for (int c = 0; c < 4; c++) {
      acc[c] += __shfl_xor_sync(0xffffffffu, acc[c], 1);
      acc[c] += __shfl_xor_sync(0xffffffffu, acc[c], 2);
    }
    // every lane of the quad now holds the four column sums: lane j == 0 adds
    // them to the scratch row with one 16-byte reduction
    if (active && j == 0 && HQ_IN_BOUNDS(ws + m, 16, ws, (size_t)M * 4, 204))
      red_add_v4_f32(ws + m, acc[0], acc[1], acc[2], acc[3]);
  }

  // ---- the last CTA of a column range converts it to fp16 and re-zeroes the scratch ----
  if (!finalize) return;
  __threadfence();
  __syncthreads();
  if (tid == 0) {
    const unsigned total = per_range ? gridDim.y : gridDim.x * gridDim.y;
    const unsigned prev = atomicAdd(counters + (per_range ? blockIdx.x : 0), 1u);
    *s_last = (prev == total - 1) ? 1u : 0u;
  }
  __syncthreads();
  if (*s_last) {
    __threadfence();
    const int lo = per_range ? m_begin : 0, hi_m = per_range ? m_end : M;
    for (int mm = lo + tid * 4; mm < hi_m; mm += kThreads * 4) {
      if (!HQ_IN_BOUNDS(out + mm, 8, out, (size_t)M * 2, 205)) continue;
      const float4 v = __ldcg(reinterpret_cast<const float4*>(ws + mm));
      const __half2 h01 = __floats2half2_rn(v.x, v.y), h23 = __floats2half2_rn(v.z, v.w);
      *reinterpret_cast<uint2*>(out + mm) = make_uint2(half2_as_u32(h01), half2_as_u32(h23));
      *reinterpret_cast<float4*>(ws + mm) = make_float4(0.f, 0.f, 0.f, 0.f);
    }
    if (tid == 0) counters[per_range ? blockIdx.x : 0] = 0u;
  }
}

// asynchronous copies global -> shared of 16 / 8 bytes (behind the wait like any load)
__device__ __forceinline__ void cp_async_16(uint32_t dst, const void* src) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_async_8(uint32_t dst, const void* src) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(dst), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_async_wait() {
  asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory");
}
__device__ __forceinline__ uint4 lds_u4(uint32_t addr) {
  uint4 v;
  asm volatile("ld.shared.v4.u32 {%0,%1,%2,%3}, [%4];"
               : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w)
               : "r"(addr));
  return v;
}
__device__ __forceinline__ uint2 lds_u2(uint32_t addr) {
  uint2 v;
  asm volatile("ld.shared.v2.u32 {%0,%1}, [%2];" : "=r"(v.x), "=r"(v.y) : "r"(addr));
  return v;
}

__device__ __forceinline__ uint32_t lds_u32(uint32_t addr) {
  uint32_t v;
  asm volatile("ld.shared.u32 %0, [%1];" : "=r"(v) : "r"(addr));
  return v;
}
__device__ __forceinline__ float lds_f16(uint32_t addr) {
  unsigned short v;
  asm volatile("ld.shared.u16 %0, [%1];" : "=h"(v) : "r"(addr));
  return __half2float(__ushort_as_half(v));
}

// byte permute with the sign-replicating selectors, which __byte_perm masks out
__device__ __forceinline__ uint32_t permute(uint32_t a, uint32_t b, uint32_t sel) {
  uint32_t d;
  asm("prmt.b32 %0, %1, %2, %3;" : "=r"(d) : "r"(a), "r"(b), "r"(sel));
  return d;
}

// Look-up addresses of a lane.  Lane (c, q) of a warp owns column 4c + q of its 32 and looks up all four
// bytes of its words, byte (t + q) % 4 in turn t: in every turn the 32 lanes read 32 different
// (replica c, byte lane) cells of a table line, that is, 32 different banks.  The address - byte value in
// bits 8 to 15, the cell's offset in bits 0 to 7 - is one byte permute: the offsets of the four turns are the
// bytes of `cells` (below 128, so their sign is the zero of the upper bytes).
struct Lookup {
  uint32_t cells, sel[4];
  __device__ __forceinline__ explicit Lookup(int lane) {
    cells = 0;
#pragma unroll
    for (int t = 0; t < 4; t++) {
      const uint32_t byte = (uint32_t)(t + lane) & 3u;
      cells |= ((uint32_t)(lane >> 2) * 16u + byte * 4u) << (8 * t);
      sel[t] = 0xcc00u | (byte << 4) | (uint32_t)(4 + t);
    }
  }
  // the four entries of a word of packed row ROW, added to `sum`
  template <int IMM, int ROW>
  __device__ __forceinline__ float add(uint32_t word, float sum) const {
#pragma unroll
    for (int t = 0; t < 4; t++)
      sum += lds_f32_imm<IMM + (ROW >> 1) * 65536 + (ROW & 1) * 128>(permute(word, cells, sel[t]));
    return sum;
  }
  template <int IMM>
  __device__ __forceinline__ float add(int row, uint32_t word, float sum) const {  // row: known when unrolled
    return row == 0   ? add<IMM, 0>(word, sum)
           : row == 1 ? add<IMM, 1>(word, sum)
           : row == 2 ? add<IMM, 2>(word, sum)
                      : add<IMM, 3>(word, sum);
  }
};
// sum of a packed row's 32 inputs, from the table's all-ones entries
__device__ __forceinline__ float row_sum(const unsigned char* lut, int row, int lane) {
  const float4 v = *reinterpret_cast<const float4*>(lut + (row >> 1) * 65536 + 255 * 256 + (row & 1) * 128 + (lane >> 2) * 16);
  return (v.x + v.y) + (v.z + v.w);
}
__device__ __forceinline__ void red_add_f32(float* addr, float v) {
  asm volatile("red.global.add.f32 [%0], %1;" ::"l"(addr), "f"(v) : "memory");
}

// ---- ring form: one to four planes in one launch, long work per CTA -----------
// 128-input tiles and the tables of the register form.  Words, alphas and bias come through shared
// memory by asynchronous copies, kDepth column steps of a warp ahead (76 to 98 KB per SM under way,
// with one plane 41 to 49, instead of 29, and no registers held: four planes fit one launch where the
// register form takes two, each with its own tables).  The CTAs are persistent: a unit is one column range of one
// K tile, units are numbered range by range inside a tile, CTA c takes units c, c + gridDim.x, ...,
// and a warp's ring runs on through the ends of units, so words arrive while the tables of the
// next tile are built.  A lane owns one column and looks up all four bytes of its words (Lookup
// above): in the register form's division, one byte of four columns, a word goes to four lanes, and the
// reads of the words took as many shared-memory wavefronts as the look-ups (4.1 M at 12288 x 12288, 3
// planes, 60 % of the time); a lane's own column also needs no sum over lanes and a quarter of the
// products with the scales.  us of a call among others, quads -> own columns: 12288 x 12288, 3 planes 27.5 -> 23.8, 4 planes
// 32.7 -> 27.7; with the copies' addresses per unit and the inputs a unit ahead 20.2 and 25.2.  What bounds it: the
// end (3 us: fence, counters, conversion of a range by one CTA), the look-ups (5 us of issue and shared memory), the
// tables of a tile (eight copies of 1024 sums for each column range); without words and look-ups 12288 x 12288 still took
// 15.5 of 24.5 us before the addresses were moved.  On mma.sync instead of look-ups (bits in place as bytes, inputs as
// digits of 4 bits) 29.7 us: the s8 form takes 15 cycles per scheduler for 16 x 32 weights, the e4m3 form 24.
// Words from global memory straight into registers do not take this division: a lane's 4-byte loads
// are too short for HBM's latency (12288 x 12288, 1 plane 19.2 -> 24.8, 2 planes with groups of 64 26.0 -> 31.9).
constexpr int kRingThreads = 512;

// Compile-time layout.  NB: planes, RPG: packed rows per alpha group inside a tile.
// Dynamic shared memory:
//   [padding][tables 2 x 64 KiB][rings: kWarps x kDepth stages][inputs][flags]
// The tables start at the FIXED shared-window address kLutImm, as above.
template <int NB, int RPG>
struct RingLayout {
  static constexpr int kWarps = kRingThreads / 32;
  static constexpr int kGroups = 4 / RPG;
  static constexpr int kLutImm = (kDynBase + kSlack + 255) / 256 * 256;
  static constexpr int kLutBytes = 2 * 65536;
  // a stage: one column step of one warp, [row][plane][32 columns] words, then
  // [group][planes and bias][32 columns] halves
  static constexpr int kWordBytes = 4 * NB * 128;
  static constexpr int kParamBytes = kGroups * (NB + 1) * 64;
  static constexpr int kStage = kWordBytes + kParamBytes;
  static constexpr int kRing = kLutImm + kLutBytes;
  static constexpr int kTail = 4 * 32 * 4 + kCounterWords * 4;
  static constexpr int kBudget = 227 * 1024 - (kRing - kDynBase) - kTail;
  static constexpr int kFit = kBudget / (kWarps * kStage);
  static constexpr int kDepth = kFit > 4 ? 4 : kFit;
  static_assert(kDepth >= 2, "a ring of two stages");
  static constexpr int kInputs = kRing + kWarps * kDepth * kStage;
  static constexpr int kFlags = kInputs + 4 * 32 * 4;
  static constexpr int kSmem = kFlags + kCounterWords * 4 - kDynBase;
};

// b0, nb_total, counters and per_range as for lutgemm_kernel
template <int NB, int RPG>
__global__ void __launch_bounds__(kRingThreads, 1)
lutgemm_ring_kernel(const uint32_t* bW, const __half* alpha,
               const __half* q_bias, const __half* x,
               __half* __restrict__ out, float* __restrict__ ws, unsigned* __restrict__ counters,
               int M, int K, int rows_per_group, int cols_per_cta, int ranges, int tiles, int nb_total,
               int b0, int finalize, int per_range) {
  using L = RingLayout<NB, RPG>;
  constexpr int TR = 4, kThreads = kRingThreads;
  constexpr int kWarps = L::kWarps, kGroups = L::kGroups, kLutImm = L::kLutImm, kDepth = L::kDepth;
  extern __shared__ __align__(16) unsigned char dsm[];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const uint32_t dsm_addr = (uint32_t)__cvta_generic_to_shared(dsm);
  // the host has checked where the dynamic region starts; never taken
  if (dsm_addr < (uint32_t)kDynBase || dsm_addr > (uint32_t)(kDynBase + kSlack)) return;
  unsigned char* window = dsm - dsm_addr;  // generic address of shared-window address 0
  unsigned char* lut = window + kLutImm;
  float* xs = reinterpret_cast<float*>(window + L::kInputs);  // the tile's inputs
  volatile unsigned* flags = reinterpret_cast<unsigned*>(window + L::kFlags);
  const int total_rows = K >> 5;
  const int units = ranges * tiles;

  // the next kernel of the stream may become resident while this grid drains;
  // nothing is read or written before every earlier kernel has completed
  pdl_launch_dependents();
  {
    // the words of the first steps are on their way to L2 before the wait
    const int tile = (int)blockIdx.x / ranges, begin = ((int)blockIdx.x - tile * ranges) * cols_per_cta;
    const int cols = min(min(M, begin + cols_per_cta) - begin, kDepth * kWarps * 32);
    const int r = tid / NB, b = tid - r * NB;
    if (tid < TR * NB && tile * TR + r < total_rows && cols > 0)
      prefetch_l2(bW + ((size_t)(tile * TR + r) * nb_total + b0 + b) * M + begin, (uint32_t)cols * 4u);
  }
  pdl_wait();
  // the inputs of the first tile, which the tables wait for; later each unit's one unit ahead
  auto input_of = [&](int unit) {  // zero beyond K
    const int k = unit / ranges * (TR * 32) + tid;
    return tid < TR * 32 && unit < units && k < K && HQ_IN_BOUNDS(x + k, 2, x, (size_t)K * 2, 206) ? ld_dependent_f16(x + k)
                                                                                                  : __ushort_as_half(0);
  };
  __half x_next = input_of(blockIdx.x);

  // ---- the warp's ring ----
  // Step s of a unit is columns m_begin + (s * kWarps + warp) * 32 .. + 31.  The warp asks
  // for its steps kDepth ahead, through the ends of units, so words arrive while the tables
  // of the next tile are built.  Per step a lane copies up to kWordCopies runs of 16 bytes
  // of words and kParamCopies of 8 bytes of alphas and bias.
  constexpr int kWordCopies = (TR * NB * 8 + 31) / 32, kParamCopies = (kGroups * (NB + 1) * 8 + 31) / 32;
  const uint32_t ring = (uint32_t)(L::kRing + warp * (kDepth * L::kStage));
  const int seg = lane & 7;
  // extents of the caller's buffers, used only by the index-checked build
  const size_t bw_bytes = (size_t)total_rows * nb_total * M * 4;
  const size_t alpha_bytes = (size_t)(total_rows / rows_per_group) * nb_total * M * 2;
  const size_t bias_bytes = (size_t)(total_rows / rows_per_group) * M * 2;
  (void)bw_bytes; (void)alpha_bytes; (void)bias_bytes;
  // The lane's addresses are worked out once a unit (per step, with a division by the group's rows and
  // 64-bit products, they were 100 of the 370 instructions a step of three planes took).
  int f_unit = blockIdx.x, f_m = 0, f_end = 0;  // the next step to ask for: column of the lane's pieces, range's end
  const uint32_t* words_at[kWordCopies];
  const __half* params_at[kParamCopies];
  unsigned live = 0;  // copies that the unit has
  auto enter = [&] {  // f_unit -> its first step of this warp, skipping units without one
    for (; f_unit < units; f_unit += gridDim.x) {
      const int tile = f_unit / ranges, begin = (f_unit - tile * ranges) * cols_per_cta;
      f_end = min(M, begin + cols_per_cta);
      if (begin + warp * 32 >= f_end) continue;
      const int row0 = tile * TR, nrows = min(TR, total_rows - row0), g0 = row0 / rows_per_group;
      f_m = begin + warp * 32 + seg * 4;
      live = 0;
#pragma unroll
      for (int i = 0; i < kWordCopies; i++) {
        const int rp = (lane >> 3) + 4 * i, r = rp / NB, b = rp - r * NB;
        words_at[i] = bW + ((size_t)(row0 + r) * nb_total + b0 + b) * M + f_m;
        if (rp < TR * NB && r < nrows) live |= 1u << i;
      }
#pragma unroll
      for (int i = 0; i < kParamCopies; i++) {
        const int gb = (lane >> 3) + 4 * i, gi = gb / (NB + 1), b = gb - gi * (NB + 1);
        params_at[i] = b < NB ? alpha + ((size_t)(g0 + gi) * nb_total + b0 + b) * M + f_m : q_bias + (size_t)(g0 + gi) * M + f_m;
        if (gi < kGroups && gi * RPG < nrows && (b < NB || q_bias != nullptr)) live |= 256u << i;
      }
      return;
    }
  };
  const uint32_t words_to = (lane >> 3) * 128 + seg * 16, params_to = L::kWordBytes + (lane >> 3) * 64 + seg * 8;
  auto fetch = [&](uint32_t stage) {
    if (f_unit < units) {
      const bool inside = f_m < f_end;
#pragma unroll
      for (int i = 0; i < kWordCopies; i++) {
        if (inside && (live >> i & 1) && HQ_IN_BOUNDS(words_at[i], 16, bW, bw_bytes, 201))
          cp_async_16(stage + words_to + i * 512, words_at[i]);
        words_at[i] += kWarps * 32;
      }
#pragma unroll
      for (int i = 0; i < kParamCopies; i++) {
        const bool scale = ((lane >> 3) + 4 * i) % (NB + 1) < NB;
        (void)scale;
        if (inside && (live >> (8 + i) & 1) &&
            HQ_IN_BOUNDS(params_at[i], 8, scale ? alpha : q_bias, scale ? alpha_bytes : bias_bytes, scale ? 202 : 203))
          cp_async_8(stage + params_to + i * 256, params_at[i]);
        params_at[i] += kWarps * 32;
      }
      f_m += kWarps * 32;
      if (f_m - seg * 4 >= f_end) {
        f_unit += gridDim.x;
        enter();
      }
    }
    cp_async_commit();
  };
  enter();
#pragma unroll
  for (int d = 0; d < kDepth; d++) fetch(ring + d * L::kStage);

  const Lookup at(lane);
  uint32_t at_stage = 0;
  int built = -1;  // tile of the tables in place (kept only with more ranges than CTAs: millions of columns)
  float ones[kGroups];

  for (int unit = blockIdx.x; unit < units; unit += gridDim.x) {
    const int tile = unit / ranges, m_begin = (unit - tile * ranges) * cols_per_cta;
    const int m_end = min(M, m_begin + cols_per_cta);
    const int row0 = tile * TR, nrows = min(TR, total_rows - row0);
    if (tile != built) {
      built = tile;
      if (tid < TR * 32) xs[tid] = __half2float(x_next);
      __syncthreads();  // inputs in place, and no warp looks up in the old tables any more
      // ---- tables: thread = (byte value, some of the rows); signed sums of 8 inputs, each
      // stored 8 times.  Line (row pair p, byte b) at lut + p*65536 + b*256, inside
      // [row parity][replica c][j] floats; the lanes of a warp hold consecutive lines, so
      // they write different replicas at a time (conflict-free) ----
      constexpr int kRowSets = kThreads / 256;      // threads per byte value
      constexpr int kRowsEach = TR / kRowSets;      // rows per thread
      const int bv = tid & 255, rp = tid >> 8;
      uint32_t sgn[8];
#pragma unroll
      for (int t = 0; t < 8; t++) sgn[t] = ((bv >> t) & 1) ? 0u : 0x80000000u;
#pragma unroll
      for (int rr = 0; rr < kRowsEach; rr++) {
        const int r = rp * kRowsEach + rr;
        float v[4];
#pragma unroll
        for (int jj = 0; jj < 4; jj++) {
          const float4 xa = *reinterpret_cast<const float4*>(xs + r * 32 + jj * 8);
          const float4 xb = *reinterpret_cast<const float4*>(xs + r * 32 + jj * 8 + 4);
          const float s0 = __uint_as_float(__float_as_uint(xa.x) ^ sgn[0]) +
                           __uint_as_float(__float_as_uint(xa.y) ^ sgn[1]);
          const float s1 = __uint_as_float(__float_as_uint(xa.z) ^ sgn[2]) +
                           __uint_as_float(__float_as_uint(xa.w) ^ sgn[3]);
          const float s2 = __uint_as_float(__float_as_uint(xb.x) ^ sgn[4]) +
                           __uint_as_float(__float_as_uint(xb.y) ^ sgn[5]);
          const float s3 = __uint_as_float(__float_as_uint(xb.z) ^ sgn[6]) +
                           __uint_as_float(__float_as_uint(xb.w) ^ sgn[7]);
          v[jj] = (s0 + s1) + (s2 + s3);
        }
        unsigned char* line = lut + (r >> 1) * 65536 + bv * 256 + (r & 1) * 128;
#pragma unroll
        for (int c = 0; c < 8; c++)
          *reinterpret_cast<float4*>(line + ((c + lane) & 7) * 16) = make_float4(v[0], v[1], v[2], v[3]);
      }
      __syncthreads();
      // for the bias: sum of the group's inputs
#pragma unroll
      for (int gi = 0; gi < kGroups; gi++) {
        float o = 0.f;
#pragma unroll
        for (int r = gi * RPG; r < (gi + 1) * RPG; r++) o += row_sum(lut, r, lane);
        ones[gi] = o;
      }
    }
    x_next = input_of(unit + gridDim.x);

    // ---- lookups ----
    for (int m0 = m_begin + warp * 32; m0 < m_end; m0 += kWarps * 32) {
      cp_async_wait<kDepth - 1>();
      __syncwarp();
      const uint32_t stage = ring + at_stage * L::kStage;
      const uint32_t words = stage + lane * 4, params = stage + L::kWordBytes + lane * 2;
      const int m = m0 + lane;
      float acc = 0.f;
#pragma unroll
      for (int gi = 0; gi < kGroups; gi++) {
        if (gi * RPG >= nrows) break;  // rows past the end of K
        float t[NB];
#pragma unroll
        for (int b = 0; b < NB; b++) t[b] = 0.f;
#pragma unroll
        for (int r = gi * RPG; r < (gi + 1) * RPG; r++) {
#pragma unroll
          for (int b = 0; b < NB; b++) t[b] = at.add<kLutImm>(r, lds_u32(words + (r * NB + b) * 128), t[b]);
        }
#pragma unroll
        for (int b = 0; b < NB; b++) acc = fmaf(lds_f16(params + (gi * (NB + 1) + b) * 64), t[b], acc);
        if (q_bias != nullptr) acc = fmaf(lds_f16(params + (gi * (NB + 1) + NB) * 64), ones[gi], acc);
      }
      // every lane has read the stage (the look-ups that used its words are done)
      __syncwarp();
      fetch(stage);
      if (++at_stage == kDepth) at_stage = 0;
      if (m < m_end && HQ_IN_BOUNDS(ws + m, 4, ws, (size_t)M * 4, 204)) red_add_f32(ws + m, acc);
    }
  }
  cp_async_wait<0>();

  // ---- the last CTA of a column range converts it to fp16 and re-zeroes the scratch ----
  if (!finalize) return;
  __threadfence();
  if (tid < kCounterWords) flags[tid] = 0;
  __syncthreads();
  const int my_units = (units - (int)blockIdx.x + (int)gridDim.x - 1) / (int)gridDim.x;
  const int counted = per_range ? ranges : 1;
  for (int i = tid; i < my_units; i += kThreads) {
    const int range = per_range ? (int)((blockIdx.x + (unsigned)i * gridDim.x) % (unsigned)ranges) : 0;
    const unsigned total = per_range ? tiles : units;
    if (atomicAdd(counters + range, 1u) == total - 1) flags[range] = 1;
  }
  __syncthreads();
  for (int range = 0; range < counted; range++) {
    if (!flags[range]) continue;
    __threadfence();
    const int lo = per_range ? range * cols_per_cta : 0, hi_m = per_range ? min(M, lo + cols_per_cta) : M;
    // all of a thread's sums of 4096 columns are asked for before the first is used
    constexpr int kAtOnce = 2;
    for (int m0 = lo + tid * 4; m0 < hi_m; m0 += kAtOnce * kThreads * 4) {
      float4 v[kAtOnce];
#pragma unroll
      for (int i = 0; i < kAtOnce; i++) {
        const int mm = m0 + i * kThreads * 4;
        if (mm < hi_m && HQ_IN_BOUNDS(ws + mm, 16, ws, (size_t)M * 4, 204)) v[i] = __ldcg(reinterpret_cast<const float4*>(ws + mm));
      }
#pragma unroll
      for (int i = 0; i < kAtOnce; i++) {
        const int mm = m0 + i * kThreads * 4;
        if (mm >= hi_m || !HQ_IN_BOUNDS(out + mm, 8, out, (size_t)M * 2, 205)) continue;
        const __half2 h01 = __floats2half2_rn(v[i].x, v[i].y), h23 = __floats2half2_rn(v[i].z, v[i].w);
        *reinterpret_cast<uint2*>(out + mm) = make_uint2(half2_as_u32(h01), half2_as_u32(h23));
        *reinterpret_cast<float4*>(ws + mm) = make_float4(0.f, 0.f, 0.f, 0.f);
      }
    }
    if (tid == 0) counters[range] = 0u;
  }
}

// ---- bulk-copy form ---------------------------------------------------------
// The register form above keeps one column step of packed words in flight per
// warp, about 29 KB per SM, and waits out the HBM latency at every step.  This
// form asks the copy engine for the CTA's WHOLE column range right at the
// start: a CTA owns a 64-input K tile (two packed rows, 64 KB of tables) and up
// to kMaxStages steps of 512 columns.  Each of the 2*NB packed-word runs, NB
// alpha runs and the bias run of that range is contiguous in global memory and
// is fetched by TWO large bulk copies (cp.async.bulk, global -> shared), one
// per half of the range, each half completing on its own mbarrier - few large
// copies is what the copy engine is good at.  All copies are in flight while
// the tables are built, HBM streams without gaps, the first half is looked up
// while the second one lands, and the lookup phase reads its operands with
// quad-broadcast shared-memory loads (one wavefront per load).  Needs M % 8 == 0, alpha groups
// of a multiple of 64 inputs and 16-byte aligned alpha / bias (the alpha runs
// are copied in 16-byte units); other shapes take the register form.
constexpr int kBulkThreads = 512;
constexpr int kBulkWarps = kBulkThreads / 32;
constexpr int kBulkCols = kBulkWarps * 32;  // columns per step
constexpr int kMaxStages = 8;
constexpr uint32_t kMbarSpins = 1u << 22;

__device__ __forceinline__ void mbar_init(uint32_t bar, uint32_t count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bar), "r"(count) : "memory");
}
__device__ __forceinline__ void mbar_expect_tx(uint32_t bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes)
               : "memory");
}
__device__ __forceinline__ bool mbar_wait(uint32_t bar, uint32_t parity) {
  for (uint32_t i = 0; i < kMbarSpins; i++) {
    uint32_t done;
    asm volatile(
        "{\n .reg .pred p;\n"
        " mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n"
        " selp.u32 %0, 1, 0, p;\n}\n"
        : "=r"(done)
        : "r"(bar), "r"(parity)
        : "memory");
    if (done) return true;
  }
  return false;
}
__device__ __forceinline__ void bulk_load(uint32_t dst, const void* src, uint32_t bytes,
                                          uint32_t bar) {
  asm volatile(
      "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::
          "r"(dst), "l"(src), "r"(bytes), "r"(bar)
      : "memory");
}

// Shared memory: [flag 16 B][mbarriers 8 x 8 B][build scratch][padding][tables 64 KiB at
// kLutImm][2*NB word runs of the column range][NB alpha runs][bias run]
struct BulkLayout {
  static constexpr int kCompactWords = 2 * 256 * 4;
  static constexpr int kBuildBytes = kCompactWords * 4 + 2 * 32 * 4;
  static constexpr int kHeadBytes = 16 + kMaxStages * 8;
  static constexpr int kLutBytes = 65536;
  static constexpr int kLutImm = (kDynBase + kSlack + kHeadBytes + kBuildBytes + 255) / 256 * 256;
  static constexpr int kStage0 = kLutImm + kLutBytes;  // shared-window address of stage 0
};
template <int NB>
struct BulkStage {
  static constexpr int kBytes = 2 * NB * kBulkCols * 4 + (NB + 1) * kBulkCols * 2;
};

template <int NB>
__global__ void __launch_bounds__(kBulkThreads, 1)
lutgemm_bulk_kernel(const uint32_t* __restrict__ bW, const __half* __restrict__ alpha,
                    const __half* __restrict__ q_bias, const __half* __restrict__ x,
                    __half* __restrict__ out, float* __restrict__ ws,
                    unsigned* __restrict__ counters, int M, int K, int rows_per_group,
                    int cols_per_cta, int nb_total, int b0, int finalize, int per_range) {
  using L = BulkLayout;
  constexpr int kLutImm = L::kLutImm;
  extern __shared__ __align__(16) unsigned char dsm[];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const uint32_t dsm_addr = (uint32_t)__cvta_generic_to_shared(dsm);
  // the host has checked where the dynamic region starts; never taken
  if (dsm_addr < (uint32_t)kDynBase || dsm_addr > (uint32_t)(kDynBase + kSlack)) return;
  unsigned char* base0 = dsm - dsm_addr;  // generic address of shared-window address 0
  unsigned char* lut = base0 + kLutImm;
  unsigned* s_last = reinterpret_cast<unsigned*>(dsm);
  const uint32_t bars = dsm_addr + 16;
  float* compact = reinterpret_cast<float*>(dsm + L::kHeadBytes);
  float* xs = compact + L::kCompactWords;
  const int row0 = blockIdx.y * 2;  // first packed row of the tile
  const int total_rows = K >> 5;
  const int nrows = min(2, total_rows - row0);
  const int m_begin = blockIdx.x * cols_per_cta;
  const int m_end = min(M, m_begin + cols_per_cta);
  const int nsteps = (m_end - m_begin + kBulkCols - 1) / kBulkCols;
  const int g = row0 / rows_per_group;  // the tile's alpha group

  if (tid < 64) {
    const int k = row0 * 32 + tid;
    xs[tid] = (k < K) ? __half2float(x[k]) : 0.f;
  }
  if (tid == 0) {
    for (int s = 0; s < kMaxStages; s++) mbar_init(bars + 8 * s, 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  __syncthreads();
  // ---- request the whole column range: warp h asks for half h of every run ----
  const int steps_half = (nsteps + 1) / 2;            // steps in the first half
  const uint32_t range_cols = (uint32_t)cols_per_cta;  // run pitch in shared memory (columns)
  const uint32_t alpha_off = 2u * NB * range_cols * 4u;
  if (warp < 2 && warp * steps_half < nsteps) {
    const int h = warp;
    const int m = m_begin + h * steps_half * kBulkCols;
    const int m_hi = h == 0 ? min(m_end, m_begin + steps_half * kBulkCols) : m_end;
    const uint32_t cols = (uint32_t)(m_hi - m);  // multiple of 8
    const uint32_t stage = (uint32_t)L::kStage0;
    const uint32_t col0 = (uint32_t)(m - m_begin);
    const uint32_t bar = bars + 8 * h;
    const bool bias_on = q_bias != nullptr;
    // this lane's copy: packed words of (row r, plane b), alpha of plane b, or the bias
    const void* src = nullptr;
    uint32_t dst = 0, bytes = 0;
    if (lane < 2 * NB) {
      const int r = lane / NB, b = lane - r * NB;
      if (r < nrows) {
        src = bW + ((size_t)(row0 + r) * nb_total + b0 + b) * M + m;
        dst = stage + ((uint32_t)lane * range_cols + col0) * 4u;
        bytes = cols * 4u;
      }
    } else if (lane < 3 * NB) {
      const int b = lane - 2 * NB;
      src = alpha + ((size_t)g * nb_total + b0 + b) * M + m;
      dst = stage + alpha_off + ((uint32_t)b * range_cols + col0) * 2u;
      bytes = cols * 2u;
    } else if (lane == 3 * NB && bias_on) {
      src = q_bias + (size_t)g * M + m;
      dst = stage + alpha_off + ((uint32_t)NB * range_cols + col0) * 2u;
      bytes = cols * 2u;
    }
#ifdef HQ_BOUNDS_CHECK
    {
      // a copy that leaves its buffer is recorded and the whole stage is skipped
      const size_t groups = (size_t)(total_rows / rows_per_group);
      bool fine = true;
      if (bytes != 0) {
        if (lane < 2 * NB) fine = HQ_IN_BOUNDS(src, bytes, bW, (size_t)total_rows * nb_total * M * 4, 211);
        else if (lane < 3 * NB) fine = HQ_IN_BOUNDS(src, bytes, alpha, groups * nb_total * M * 2, 212);
        else fine = HQ_IN_BOUNDS(src, bytes, q_bias, groups * M * 2, 213);
      }
      if (__ballot_sync(0xffffffffu, !fine) != 0u) bytes = 0;
    }
#endif
    uint32_t total = bytes;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) total += __shfl_xor_sync(0xffffffffu, total, o);
    if (lane == 0) mbar_expect_tx(bar, total);
    __syncwarp();
    if (bytes != 0) bulk_load(dst, src, bytes, bar);
  }

  // ---- phase A: thread = (byte value, row); signed sums of 8 inputs ----
  {
    const int bv = tid & 255, r = tid >> 8;
    uint32_t sgn[8];
#pragma unroll
    for (int t = 0; t < 8; t++) sgn[t] = ((bv >> t) & 1) ? 0u : 0x80000000u;
    float v[4];
#pragma unroll
    for (int jj = 0; jj < 4; jj++) {
      const float4 xa = *reinterpret_cast<const float4*>(xs + r * 32 + jj * 8);
      const float4 xb = *reinterpret_cast<const float4*>(xs + r * 32 + jj * 8 + 4);
      const float s0 = __uint_as_float(__float_as_uint(xa.x) ^ sgn[0]) +
                       __uint_as_float(__float_as_uint(xa.y) ^ sgn[1]);
      const float s1 = __uint_as_float(__float_as_uint(xa.z) ^ sgn[2]) +
                       __uint_as_float(__float_as_uint(xa.w) ^ sgn[3]);
      const float s2 = __uint_as_float(__float_as_uint(xb.x) ^ sgn[4]) +
                       __uint_as_float(__float_as_uint(xb.y) ^ sgn[5]);
      const float s3 = __uint_as_float(__float_as_uint(xb.z) ^ sgn[6]) +
                       __uint_as_float(__float_as_uint(xb.w) ^ sgn[7]);
      v[jj] = (s0 + s1) + (s2 + s3);
    }
    *reinterpret_cast<float4*>(compact + (r * 256 + bv) * 4) = make_float4(v[0], v[1], v[2], v[3]);
  }
  __syncthreads();
  // ---- phase B: replicate each (row, byte) entry 8 times into its table line ----
  // line (byte b) at lut + b*256; inside: [row parity][c][j] floats
  {
    const int c = lane & 7, bl = lane >> 3;
#pragma unroll 4
    for (int it = 0; it < 2 * 256 / (kBulkWarps * 4); it++) {
      const int e = (it * kBulkWarps + warp) * 4 + bl;  // row*256 + byte
      const int r = e >> 8, b = e & 255;
      const float4 v = *reinterpret_cast<const float4*>(compact + e * 4);
      *reinterpret_cast<float4*>(lut + b * 256 + (r & 1) * 128 + c * 16) = v;
    }
  }
  __syncthreads();

  // ---- lookup phase ----
  const int j = lane & 3;   // byte of the word this lane looks up
  const int cq = lane >> 2; // column quad inside the warp's 32 columns
  const uint32_t hi = (uint32_t)(lane * 4);
  const uint32_t sel = 0x7604u | ((uint32_t)j << 4);
  // bias uses the all-ones entry (byte 255): sum of this lane's 8 inputs per row
  const float ones = *reinterpret_cast<const float*>(lut + 255 * 256 + lane * 4) +
                     *reinterpret_cast<const float*>(lut + 255 * 256 + 128 + lane * 4);
  const uint32_t col_off = (uint32_t)(warp * 32 + cq * 4);  // column inside the step
  bool ok = true;
  for (int s = 0; s < nsteps; s++) {
    const int m = m_begin + s * kBulkCols + (int)col_off;
    if (ok && !mbar_wait(bars + 8 * (s >= steps_half ? 1 : 0), 0)) ok = false;
    const bool active = m < m_end;
    float acc[4] = {0.f, 0.f, 0.f, 0.f};
    if (active) {
      const uint32_t stage = (uint32_t)L::kStage0;
      const uint32_t col = (uint32_t)(s * kBulkCols) + col_off;  // column inside the range
      float t[NB][4];
#pragma unroll
      for (int r = 0; r < 2; r++) {
#pragma unroll
        for (int b = 0; b < NB; b++) {
          // rows past the end of K were not copied: their tables are zero, any word will do
          const uint4 wv = lds_u4(stage + ((uint32_t)(r * NB + b) * range_cols + col) * 4u);
          const uint32_t w4[4] = {wv.x, wv.y, wv.z, wv.w};
#pragma unroll
          for (int c = 0; c < 4; c++) {
            const uint32_t a = __byte_perm(w4[c], hi, sel);
            const float v = r == 0 ? lds_f32_imm<kLutImm>(a) : lds_f32_imm<kLutImm + 128>(a);
            t[b][c] = (r == 0) ? v : t[b][c] + v;
          }
        }
      }
#pragma unroll
      for (int b = 0; b < NB; b++) {
        const uint2 av = lds_u2(stage + alpha_off + ((uint32_t)b * range_cols + col) * 2u);
        const float2 a01 = __half22float2(u32_as_half2(av.x));
        const float2 a23 = __half22float2(u32_as_half2(av.y));
        acc[0] = fmaf(a01.x, t[b][0], acc[0]);
        acc[1] = fmaf(a01.y, t[b][1], acc[1]);
        acc[2] = fmaf(a23.x, t[b][2], acc[2]);
        acc[3] = fmaf(a23.y, t[b][3], acc[3]);
      }
      if (q_bias != nullptr) {
        const uint2 bv = lds_u2(stage + alpha_off + ((uint32_t)NB * range_cols + col) * 2u);
        const float2 b01 = __half22float2(u32_as_half2(bv.x));
        const float2 b23 = __half22float2(u32_as_half2(bv.y));
        acc[0] = fmaf(b01.x, ones, acc[0]);
        acc[1] = fmaf(b01.y, ones, acc[1]);
        acc[2] = fmaf(b23.x, ones, acc[2]);
        acc[3] = fmaf(b23.y, ones, acc[3]);
      }
    }
#pragma unroll
    for (int c = 0; c < 4; c++) {
      acc[c] += __shfl_xor_sync(0xffffffffu, acc[c], 1);
      acc[c] += __shfl_xor_sync(0xffffffffu, acc[c], 2);
    }
    if (active && j == 0 && HQ_IN_BOUNDS(ws + m, 16, ws, (size_t)M * 4, 214))
      red_add_v4_f32(ws + m, acc[0], acc[1], acc[2], acc[3]);
  }
  // a wait that ran out: word kCounterWords - 1 of the counter block tells the host
  if (!ok && lane == 0) atomicExch(counters + (kCounterWords - 1), 1u);

  // ---- the last CTA of a column range converts it to fp16 and re-zeroes the scratch ----
  if (!finalize) return;
  __threadfence();
  __syncthreads();
  if (tid == 0) {
    const unsigned total = per_range ? gridDim.y : gridDim.x * gridDim.y;
    const unsigned prev = atomicAdd(counters + (per_range ? blockIdx.x : 0), 1u);
    *s_last = (prev == total - 1) ? 1u : 0u;
  }
  __syncthreads();
  if (*s_last) {
    __threadfence();
    const int lo = per_range ? m_begin : 0, hi_m = per_range ? m_end : M;
    for (int mm = lo + tid * 4; mm < hi_m; mm += kBulkThreads * 4) {
      if (!HQ_IN_BOUNDS(out + mm, 8, out, (size_t)M * 2, 215)) continue;
      const float4 v = __ldcg(reinterpret_cast<const float4*>(ws + mm));
      const __half2 h01 = __floats2half2_rn(v.x, v.y), h23 = __floats2half2_rn(v.z, v.w);
      *reinterpret_cast<uint2*>(out + mm) = make_uint2(half2_as_u32(h01), half2_as_u32(h23));
      *reinterpret_cast<float4*>(ws + mm) = make_float4(0.f, 0.f, 0.f, 0.f);
    }
    if (tid == 0) counters[per_range ? blockIdx.x : 0] = 0u;
  }
}

struct LaunchArgs {
  dim3 grid;
  cudaStream_t st;
  const uint32_t* bW;
  const __half* alpha;
  const __half* q_bias;
  const __half* x;
  __half* out;
  float* ws;
  unsigned* counters;
  int M, K, rows_per_group, cols_per_cta, nb_total, per_range;
};

template <int TR, int NB, int RPG>
int launch_one(const LaunchArgs& a, int b0, const __half* bias, int finalize) {
  using L = Layout<TR>;
  constexpr int kThreads = TR == 4 ? 512 : 256;
  constexpr auto kern = lutgemm_kernel<TR, NB, RPG, kThreads>;
  cudaError_t e = ensure_dynamic_smem<kern>(L::kSmem);
  if (e != cudaSuccess) return cuda_status(e);
  return cuda_status(launch_pdl(kern, a.grid, dim3(kThreads), L::kSmem, a.st, a.bW, a.alpha, bias,
                                a.x, a.out, a.ws, a.counters, a.M, a.K, a.rows_per_group,
                                a.cols_per_cta, a.nb_total, b0, finalize, a.per_range));
}

template <int NB, int RPG>
int launch_ring(const LaunchArgs& a, int b0, const __half* bias, int finalize) {
  using L = RingLayout<NB, RPG>;
  constexpr auto kern = lutgemm_ring_kernel<NB, RPG>;
  cudaError_t e = ensure_dynamic_smem<kern>(L::kSmem);
  if (e != cudaSuccess) return cuda_status(e);
  const long long units = (long long)a.grid.x * a.grid.y;
  const unsigned ctas = (unsigned)std::min<long long>(units, sm_count());
  return cuda_status(launch_pdl(kern, dim3(ctas), dim3(kRingThreads), L::kSmem, a.st, a.bW, a.alpha, bias,
                                a.x, a.out, a.ws, a.counters, a.M, a.K, a.rows_per_group, a.cols_per_cta,
                                (int)a.grid.x, (int)a.grid.y, a.nb_total, b0, finalize, a.per_range));
}

// Planes go in launches of up to four (three with alpha groups of 32 inputs, whose parameters leave
// the rings no room for a fourth) that accumulate into the same scratch row.  Only the first
// launch adds the bias term, only the last one converts the scratch row.  On tiles of 128
// inputs the ring form takes four planes, and fewer where a warp has some column steps (takes_ring);
// the register form takes the rest.  Five to eight planes as 4 + 1 to 4 + 4 take 0.75 to 1.00 of what 3 + 2
// to 3 + 3 + 2 took when both were in the quads' division.
template <int TR, int RPG>
int launch_planes(const LaunchArgs& a) {
  constexpr bool kFour = TR == 2 || RPG > 1;  // groups of 32 inputs: the rings hold three planes
  // The rings take over where a warp has some column steps: us, register form -> rings, at steps per warp
  // 3 planes: 1.3 (12288 x 1024) 7.2 -> 7.5, 1.5 (6400 x 2304) 7.8 -> 7.4, 1.7 (4096 x 4096) 7.9 -> 7.4, 3.5 (8192 x 4096)
  // 10.6 -> 8.9;
  // 2 planes: 1.7 7.0 -> 7.2, 2.6 (12288 x 2048) 7.9 -> 7.8, 2.7 (5120 x 5120) 8.5 -> 7.7, with groups of 64 9.4 -> 8.1, 5.2
  // (4096 x 12288) 12.9 -> 10.4;
  // 1 plane: 2.7 6.8 -> 7.0, 3.5 7.1 -> 7.3, 3.9 (3072 x 12288) 8.7 -> 8.2, 5.2 10.2 -> 8.9; with groups of 64, 2.6 7.1 -> 7.2,
  // 2.7 7.5 -> 7.0, 5.2 11.5 -> 9.3.
  // Groups of 32 inputs: as before, three planes in long units.
  const double steps = (double)a.M * a.grid.y / ((double)kRingThreads * sm_count());
  auto takes_ring = [&](int n) {
    if (TR != 4) return false;
    if (RPG == 1) return n == 3 && a.cols_per_cta >= 2 * kRingThreads && (long long)a.grid.x * a.grid.y > sm_count();
    return n == 4 || steps >= (n == 3 ? 1.5 : n == 1 && RPG == 4 ? 3.6 : 2.65);
  };
  const int nb = a.nb_total;
  for (int b0 = 0; b0 < nb;) {
    const int n = std::min(nb - b0, kFour ? 4 : 3);
    const int last = (b0 + n == nb) ? 1 : 0;
    const __half* bias = b0 == 0 ? a.q_bias : nullptr;
    int st;
    if (takes_ring(n)) {
      if constexpr (TR == 4 && RPG > 1) {
        st = n == 1   ? launch_ring<1, RPG>(a, b0, bias, last)
             : n == 2 ? launch_ring<2, RPG>(a, b0, bias, last)
             : n == 3 ? launch_ring<3, RPG>(a, b0, bias, last)
                      : launch_ring<4, RPG>(a, b0, bias, last);
      } else {
        st = launch_ring<3, RPG>(a, b0, bias, last);
      }
    } else if (n == 1) {
      st = launch_one<TR, 1, RPG>(a, b0, bias, last);
    } else if (n == 2) {
      st = launch_one<TR, 2, RPG>(a, b0, bias, last);
    } else if (TR == 2 && n == 4) {
      st = launch_one<TR, (TR == 2 ? 4 : 3), RPG>(a, b0, bias, last);
    } else {
      st = launch_one<TR, 3, RPG>(a, b0, bias, last);
    }
    if (st != HQ_OK) return st;
    b0 += n;
  }
  return HQ_OK;
}

template <int NB>
int launch_bulk_one(const LaunchArgs& a, int b0, const __half* bias, int finalize) {
  constexpr auto kern = lutgemm_bulk_kernel<NB>;
  const int stages = (a.cols_per_cta + kBulkCols - 1) / kBulkCols;
  const size_t smem = (size_t)BulkLayout::kStage0 - kDynBase + (size_t)stages * BulkStage<NB>::kBytes;
  cudaError_t e = ensure_dynamic_smem<kern>(smem);
  if (e != cudaSuccess) return cuda_status(e);
  kern<<<a.grid, kBulkThreads, smem, a.st>>>(a.bW, a.alpha, bias, a.x, a.out, a.ws, a.counters, a.M,
                                             a.K, a.rows_per_group, a.cols_per_cta, a.nb_total, b0,
                                             finalize, a.per_range);
  return launch_status();
}

// stages of 512 columns that fit beside the tables for NB planes per launch
inline int bulk_max_stages(int nb) {
  const int stage = 2 * nb * kBulkCols * 4 + (nb + 1) * kBulkCols * 2;
  const int room = 227 * 1024 - (BulkLayout::kStage0 - kDynBase);
  return std::min(kMaxStages, room / stage);
}

// Planes in groups of up to 3 per launch (what leaves room for 8 stages)
int launch_bulk_planes(const LaunchArgs& a) {
  constexpr int kMax = 3;
  const int nb = a.nb_total;
  for (int b0 = 0; b0 < nb; b0 += kMax) {
    const int n = nb - b0 < kMax ? nb - b0 : kMax;
    const int last = (b0 + n == nb) ? 1 : 0;
    const __half* bias = b0 == 0 ? a.q_bias : nullptr;
    int st;
    if (n == 1) st = launch_bulk_one<1>(a, b0, bias, last);
    else if (n == 2) st = launch_bulk_one<2>(a, b0, bias, last);
    else st = launch_bulk_one<3>(a, b0, bias, last);
    if (st != HQ_OK) return st;
  }
  return HQ_OK;
}

// Argument rules shared by both entry points; nothing is launched or touched
// when they fail.
int check_args(const void* out_half, const void* x_half, const uint32_t* bW, const void* alpha_half,
               const void* q_bias_half, int M, int K, int nb, int group_size) {
  if (!out_half || !x_half || !bW || !alpha_half) return HQ_ERR_NULL_POINTER;
  if (M <= 0 || K <= 0 || M % 4 != 0 || K % 32 != 0 || nb < 1 || nb > 8) return HQ_ERR_BAD_SHAPE;
  if (group_size <= 0 || group_size % 32 != 0 || K % group_size != 0) return HQ_ERR_BAD_SHAPE;
  if (!aligned16(bW) || !aligned8(alpha_half) || (q_bias_half && !aligned8(q_bias_half)) ||
      !aligned8(out_half))
    return HQ_ERR_MISALIGNED;
  const int rpg = group_size / 32;
  // groups of 96, 160, ... inputs would straddle tiles
  if (rpg != 1 && rpg % 2 != 0) return HQ_ERR_UNSUPPORTED;
  return HQ_OK;
}

}  // namespace
}  // namespace hq

extern "C" {

size_t hq_lutgemm_workspace_bytes(int M) {
  if (M <= 0) return 0;
  return ((size_t)M * 4 + 255) / 256 * 256 + 256;
}

int hq_lutgemm_nqmv(void* out_half, const void* x_half, const uint32_t* bW, const void* alpha_half,
                    const void* q_bias_half, int M, int K, int nb, int group_size, void* workspace,
                    size_t workspace_bytes, hq_stream_t stream) {
  using namespace hq;
  const int cst = check_args(out_half, x_half, bW, alpha_half, q_bias_half, M, K, nb, group_size);
  if (cst != HQ_OK) return cst;
  if (!workspace || workspace_bytes < hq_lutgemm_workspace_bytes(M)) return HQ_ERR_WORKSPACE;
  if (!aligned16(workspace)) return HQ_ERR_MISALIGNED;
  const int rpg = group_size / 32;
  const int reserved = reserved_smem_per_block();
  if (reserved < kDynBase || reserved > kDynBase + kSlack) return HQ_ERR_UNSUPPORTED;

  // Bulk-copy form: 64-input tiles, the whole column range of a CTA requested up
  // front.  Opt-in (environment HQ_LUT_BULK=1): on B200 it measured 37.1 us
  // against 29.7 us for the register form on a 12288 x 12288, 3-plane layer.
  if (env_flag("HQ_LUT_BULK") && M % 8 == 0 && rpg % 2 == 0 && aligned16(alpha_half) &&
      (!q_bias_half || aligned16(q_bias_half))) {
    const int tiles2 = (K / 32 + 1) / 2;
    const int max_cols = bulk_max_stages(std::min(nb, 3)) * kBulkCols;
    // balanced column ranges of at most max_cols columns, multiples of 512
    const int steps_total = (M + kBulkCols - 1) / kBulkCols;
    const int ranges = (steps_total * kBulkCols + max_cols - 1) / max_cols;
    const int steps_per_range = (steps_total + ranges - 1) / ranges;
    LaunchArgs a;
    a.cols_per_cta = steps_per_range * kBulkCols;
    const int mblocks = (M + a.cols_per_cta - 1) / a.cols_per_cta;
    a.grid = dim3(mblocks, tiles2);
    a.st = (cudaStream_t)stream;
    a.bW = bW;
    a.alpha = reinterpret_cast<const __half*>(alpha_half);
    a.q_bias = reinterpret_cast<const __half*>(q_bias_half);
    a.x = reinterpret_cast<const __half*>(x_half);
    a.out = reinterpret_cast<__half*>(out_half);
    a.ws = reinterpret_cast<float*>(workspace);
    a.counters = reinterpret_cast<unsigned*>(reinterpret_cast<char*>(workspace) +
                                             (hq_lutgemm_workspace_bytes(M) - 256));
    a.M = M;
    a.K = K;
    a.rows_per_group = rpg;
    a.nb_total = nb;
    a.per_range = mblocks <= kCounterWords - 1 ? 1 : 0;
    return launch_bulk_planes(a);
  }
  // K tile: 128 inputs wherever alpha groups do not straddle it; 64 inputs for
  // groups of 192, 320, ... inputs
  int tile_rows = (rpg % 4 == 0 || rpg <= 2) ? 4 : 2;
  const int tiles = (K / 32 + tile_rows - 1) / tile_rows;
  // columns per CTA: a multiple of 256 chosen so the grid is close to a
  // multiple of the resident CTA slots while the table build stays amortised.
  const int slots = sm_count() * (tile_rows == 2 ? 2 : 1);
  int best_cols = 256;
  double best_score = -1.0;
  const int max_chunks = (M + 255) / 256;
  for (int mb = 1; mb <= max_chunks; mb++) {
    const int chunk256 = (max_chunks + mb - 1) / mb;  // balanced ranges
    const long ctas = (long)((max_chunks + chunk256 - 1) / chunk256) * tiles;
    const long waves = (ctas + slots - 1) / slots;
    // efficiency = useful lookups / (lookups + table build), times wave balance
    const double amort = (double)(chunk256 * 256) / (chunk256 * 256 + 2000.0);
    const double balance = (double)ctas / (double)(waves * slots);
    const double score = amort * balance;
    if (score > best_score) { best_score = score; best_cols = chunk256 * 256; }
  }
  const int mblocks = (M + best_cols - 1) / best_cols;
  LaunchArgs a;
  a.grid = dim3(mblocks, tiles);
  a.st = (cudaStream_t)stream;
  a.bW = bW;
  a.alpha = reinterpret_cast<const __half*>(alpha_half);
  a.q_bias = reinterpret_cast<const __half*>(q_bias_half);
  a.x = reinterpret_cast<const __half*>(x_half);
  a.out = reinterpret_cast<__half*>(out_half);
  a.ws = reinterpret_cast<float*>(workspace);
  a.counters = reinterpret_cast<unsigned*>(reinterpret_cast<char*>(workspace) +
                                           (hq_lutgemm_workspace_bytes(M) - 256));
  a.M = M;
  a.K = K;
  a.rows_per_group = rpg;
  a.cols_per_cta = best_cols;
  a.nb_total = nb;
  a.per_range = mblocks <= kCounterWords ? 1 : 0;
  if (tile_rows == 4) {
    if (rpg % 4 == 0) return launch_planes<4, 4>(a);
    if (rpg == 2) return launch_planes<4, 2>(a);
    return launch_planes<4, 1>(a);
  }
  if (rpg % 2 == 0) return launch_planes<2, 2>(a);
  return launch_planes<2, 1>(a);
}

// ---- entry point that allocates nothing ----------------------------------

}  // extern "C"

namespace hq {
namespace {

// Scratch row of the allocation-free entry point: fp32 partial sums for up to
// HQ_LUTGEMM_NOALLOC_MAX_M outputs plus the completion counter.  Every GPU
// that loads the library holds these 257 KiB until the process exits.
static __device__ __align__(256) unsigned char g_noalloc_scratch[HQ_LUTGEMM_NOALLOC_MAX_M * 4 + 256];

std::mutex g_noalloc_mu;
void* g_noalloc_ptr[kMaxDevices];  // device address of the array, per device; null = not set up

// Device address of g_noalloc_scratch on the current device.  In host code the
// array's name is only a handle; the address a kernel can use comes from
// cudaGetSymbolAddress, asked once per device with that device current.
int noalloc_scratch(void** out) {
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return cuda_status(e);
  if (dev < 0 || dev >= kMaxDevices) return HQ_ERR_UNSUPPORTED;
  std::lock_guard<std::mutex> lock(g_noalloc_mu);
  if (g_noalloc_ptr[dev] == nullptr) {
    void* p = nullptr;
    e = cudaGetSymbolAddress((void**)&p, g_noalloc_scratch);
    if (e != cudaSuccess) return cuda_status(e);
    g_noalloc_ptr[dev] = p;
  }
  *out = g_noalloc_ptr[dev];
  return HQ_OK;
}

}  // namespace
}  // namespace hq

extern "C" int hq_lutgemm_nqmv_noalloc(void* out_half, const void* x_half, const uint32_t* bW,
                                       const void* alpha_half, const void* q_bias_half, int M,
                                       int K, int nb, int group_size, hq_stream_t stream) {
  using namespace hq;
  if (M > HQ_LUTGEMM_NOALLOC_MAX_M) return HQ_ERR_TOO_LARGE;
  // every argument rule is checked before the shared array is looked up or touched
  const int cst = check_args(out_half, x_half, bW, alpha_half, q_bias_half, M, K, nb, group_size);
  if (cst != HQ_OK) return cst;
  void* ws = nullptr;
  const int st = noalloc_scratch(&ws);
  if (st != HQ_OK) return st;
  const size_t bytes = hq_lutgemm_workspace_bytes(M);
  // The array keeps whatever the previous call (of any caller) left in it, and
  // the kernel needs partial sums and counter to start at zero.
  cudaError_t e = cudaMemsetAsync(ws, 0, bytes, (cudaStream_t)stream);
  if (e != cudaSuccess) return cuda_status(e);
  return hq_lutgemm_nqmv(out_half, x_half, bW, alpha_half, q_bias_half, M, K, nb, group_size, ws,
                         bytes, stream);
}
