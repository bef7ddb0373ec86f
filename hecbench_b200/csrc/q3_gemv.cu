// GPTQ 3-bit packed mat-vec for sm_100a.
//
// Packed layout (quant3MatMul-cuda/kernels.h:41-87): mat is int32[height][width];
// for output column c and K-group r (32 inputs) rows 3r..3r+2 of mat[:,c] form a
// 96-bit little-endian stream, code j at bits 3j..3j+2.
//
// Design.
//  * The products run on mma.sync m16n8k16 in bf16.  A 3-bit field left in place in the low eight bits
//    of a half of a word is the bf16 number q * 2^(p - 133) (the exponents 0 and 1 have one spacing), so
//    two weights of an A register cost one logic operation; a group's 16 pairs lie in three words
//    as they are and six windows of them (kPair).  Inputs are pre-scaled by the matching powers of two.
//  * An input is split into bf16 pieces by truncation, two for fp16, three for fp32, which hold it
//    exactly; piece i is column i of B, so both input types cost the same and every product is exact.
//    fp32 inputs are scaled by the largest exponent of their 128 (a quad of groups); their sums are held as
//    2^-8 of their value, so only what is below 2^-118 loses bits on the way.
//  * The affine part is factored: sum (s*q - z)*x = s*sum(q*x) - z*sum(x).
//  * A warp owns 32 columns and takes four groups (a quad) at a time: lane (g, t) multiplies
//    columns 4g .. 4g + 3 of group t.  NB warps side by side, W / NB in turn along K.
//  * One CTA per SM takes an equal range of (block of 32 NB columns, quads) steps; sums go to mul
//    (the reference API accumulates into it) once per range and block, an atomicAdd per column from each of
//    the W / NB warps along K.
//  * Words come by cp.async, two quads ahead per warp, eight lanes to a 128-byte line: with a quarter-warp
//    over four lines a read of 226 MB took 57 us, with whole lines 35 (the copy rate).
//
// What bounds it: the logic pipe (two cycles an operation, 22 of them for 32 weights), 56 %, and HBM.
// us in replayed graphs, sums of fp16 products in registers, a group ahead (before) -> this
// form, fp16 (fp32) inputs, words from HBM: 49152 x 12288 50.4 -> 40.6 (73.0 -> 41.7), 28672 x 8192 24.7 -> 18.2 (30.5 -> 18.6),
// 8192 x 8192 9.9 -> 7.4 (11.5 -> 7.7), 4096 x 4096 4.0 -> 3.8 (4.9 -> 3.8), 1024 x 4096 3.5 -> 2.7 (3.2 -> 2.7), 512 x
// 1024 2.3 -> 1.9 (2.3 -> 1.8); 499 layers of 512 to 32768 columns, 1024 to 16384 inputs 0.81, 8 of them above 1.02, worst 1.10
// (fp16 4644 x 1984 2.80 -> 3.08).
// Error against fp64 sums: 5e-4 to 1.1e-3 -> 1e-7 to 2.5e-7 (fp32 inputs 1e-7 to 5.7e-7 -> 1e-7 to 2.1e-7).
// Taken back: windows by multiplications on the other pipe (49152 x 12288 45.1 -> 54.6).
#include <limits.h>

#include <type_traits>
#include <utility>

#include "hq_common.cuh"

namespace hq {

namespace {

constexpr int kDepth = 3;                // quads of packed words per warp: one in use, the others on the way
constexpr int kSlot = 3 * 32 * 16;       // bytes of a warp's words of a quad
constexpr int kColsPerWarp = 32;
constexpr int kSliceQuads = 128;

__device__ __forceinline__ float pow2f(int e) { return __int_as_float((e + 127) << 23); }

constexpr int kPairs = 16;
struct Pair { int shift, lo, hi; };  // window's first bit in the group's stream; codes in its low and high half
constexpr Pair kPair[kPairs] = {{0, 0, 6},    {0, 1, 7},    {6, 2, 8},    {6, 3, 9},    {12, 4, 10},  {12, 5, 11},
                                {32, 12, 17}, {37, 13, 18}, {37, 14, 19}, {43, 15, 20}, {43, 16, 21}, {64, 22, 27},
                                {64, 23, 28}, {70, 24, 29}, {70, 25, 30}, {73, 26, 31}};
// bit positions of a pair's fields in the halves of its window
__host__ __device__ constexpr int field_lo(int j) { return 3 * kPair[j].lo - kPair[j].shift; }
__host__ __device__ constexpr int field_hi(int j) { return 3 * kPair[j].hi - kPair[j].shift - 16; }
constexpr bool pairs_cover() {
  unsigned seen = 0;
  for (int j = 0; j < kPairs; j++) {
    if (field_lo(j) < 0 || field_lo(j) > 5 || field_hi(j) < 0 || field_hi(j) > 5) return false;
    seen |= 1u << kPair[j].lo | 1u << kPair[j].hi;
  }
  return seen == 0xffffffffu;
}
static_assert(pairs_cover(), "every code once, its field in the low eight bits of a half");

// The same for a pair that is known at run time only: codes by their three runs, positions from
// nibbles.
__device__ __forceinline__ int code_lo(int j) { return j + (j >= 6 ? 6 : 0) + (j >= 11 ? 5 : 0); }
__device__ __forceinline__ int code_hi(int j) { return j + 6 + (j >= 6 ? 5 : 0) + (j >= 11 ? 5 : 0); }
constexpr uint64_t fields(bool high) {
  uint64_t v = 0;
  for (int j = 0; j < kPairs; j++) v |= (uint64_t)(high ? field_hi(j) : field_lo(j)) << (4 * j);
  return v;
}
constexpr uint64_t kFieldsLo = fields(false), kFieldsHi = fields(true);

template <int SHIFT>
__device__ __forceinline__ uint32_t window(const uint32_t (&w)[3]) {
  if constexpr (SHIFT % 32 == 0) return w[SHIFT / 32];
  else if constexpr (SHIFT / 32 == 2) return w[2] >> (SHIFT % 32);
  else return __funnelshift_r(w[SHIFT / 32], w[SHIFT / 32 + 1], SHIFT % 32);
}
template <int J>
__device__ __forceinline__ uint32_t pair_of(const uint32_t (&w)[3]) {
  return window<kPair[J].shift>(w) & (7u << field_lo(J) | 7u << (16 + field_hi(J)));
}

__device__ __forceinline__ void mma_bf16(float (&d)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3,
                                         uint32_t b0, uint32_t b1) {
  asm("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
      : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
      : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}
// sums of two columns' words (u: row of this lane, v: that row + 8) over the lane's group
template <int... J>
__device__ __forceinline__ void multiply(float (&d)[4], const uint32_t (&u)[3], const uint32_t (&v)[3],
                                         const uint32_t (&x)[kPairs], std::integer_sequence<int, J...>) {
  (mma_bf16(d, pair_of<2 * J>(u), pair_of<2 * J>(v), pair_of<2 * J + 1>(u), pair_of<2 * J + 1>(v), x[2 * J],
            x[2 * J + 1]),
   ...);
}

__device__ __forceinline__ uint32_t smem_at(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }
__device__ __forceinline__ void copy_16(uint32_t dst, const void* src) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst), "l"(src) : "memory");
}
__device__ __forceinline__ uint4 lds_u4(uint32_t at) {
  uint4 v;
  asm volatile("ld.shared.v4.u32 {%0,%1,%2,%3}, [%4];"
               : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w)
               : "r"(at)
               : "memory");
  return v;
}

template <bool F16IN>
constexpr int kPieces = F16IN ? 2 : 3;
// shared bytes of a quad's inputs
template <bool F16IN>
constexpr int kQuadBytes = kPairs * 4 * kPieces<F16IN> * 4;

struct Shape {
  int width, groups;  // columns; 32 inputs each
  int slice_quads;    // quads of a slice of K (blockIdx.y)
  int blocks, steps;  // blocks of 32 NB columns; steps of W / NB quads in each
  int share, over;    // steps of a CTA; the first `over` CTAs take one more
  int staged;         // steps whose inputs the fullest CTA holds
};

template <bool F16IN, int W, int NB>
__global__ void __launch_bounds__(W * 32, 1)
q3_gemv_kernel(const void* vec, const int32_t* mat, float* mul, const float* scales, const float* zeros,
               const Shape p) {
  constexpr int KW = W / NB, P = kPieces<F16IN>;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  // [ring W x kDepth slots][inputs staged x KW quads][their sums and scales, float2]
  const int tid = threadIdx.x, lane = tid & 31;
  const int warp = __shfl_sync(0xffffffffu, tid >> 5, 0);
  const int g = lane >> 2, t = lane & 3;
  const int kw = warp / NB, cw = warp % NB;
  const int q_lo = blockIdx.y * p.slice_quads;
  const int g_hi = min(p.groups, (q_lo + p.slice_quads) * 4);
  const int u0 = (int)blockIdx.x * p.share + min((int)blockIdx.x, p.over);
  const int u1 = u0 + p.share + ((int)blockIdx.x < p.over ? 1 : 0);
  const int staged = min(u1 - u0, p.steps);
  const int b0 = u0 / p.steps, k0 = u0 - b0 * p.steps;
  // eight lanes copy a line of a row (ct: group, cg: 16-byte piece); pieces of the four groups are turned
  // against one another, so that the lanes (g, t) of a quarter-warp read different banks
  const int ct = lane >> 3, cg = lane & 7;
  const uint32_t ring = smem_at(smem_raw) + (uint32_t)(warp * kDepth * kSlot);
  const uint32_t ring_in = ring + (uint32_t)((ct * 8 + ((cg + 2 * ct) & 7)) * 16);
  const uint32_t ring_out = ring + (uint32_t)((t * 8 + ((g + 2 * t) & 7)) * 16);
  unsigned char* const table = smem_raw + W * kDepth * kSlot;
  float2* const sums = reinterpret_cast<float2*>(table + (size_t)p.staged * KW * kQuadBytes<F16IN>);

  // extents of the caller's buffers, used only by the index-checked build
  const size_t mat_bytes = (size_t)p.groups * 3 * p.width * 4, vec_bytes = (size_t)p.groups * 32 * (F16IN ? 2 : 4);
  const size_t column_bytes = (size_t)p.width * 4;
  (void)mat_bytes; (void)vec_bytes; (void)column_bytes;

  pdl_launch_dependents();
  // The lines of the first steps on their way to L2 while the kernel before drains, where a CTA has three
  // steps or more (8192 x 8192 8.2 -> 7.4 us, 12288 x 16384 17.5 -> 16.3; one step, 1184 x 6976, 2.6 -> 3.0).
  if (u1 - u0 > 2) {
#pragma unroll
    for (int d = 0; d < kDepth - 1; d++) {
      const int row = (q_lo + (k0 + d) * KW) * 12 + tid, col = b0 * NB * kColsPerWarp;
      const uint32_t bytes = (uint32_t)min(NB * kColsPerWarp, p.width - col) * 4u;
      if (k0 + d < p.steps && tid < 12 * KW && row < g_hi * 3 &&
          HQ_IN_BOUNDS(mat + (size_t)row * p.width + col, bytes, mat, mat_bytes, 1101))
        prefetch_l2(mat + (size_t)row * p.width + col, bytes);
    }
  }
  pdl_wait();

  // ---- packed words: this lane's four columns of three rows, kDepth - 1 quads ahead ----
  // (rows past the slice and columns past the width are not copied: what the slot held is multiplied
  // by inputs of zero, or its sums go nowhere)
  const size_t row = (size_t)p.width, next = 12 * KW * row;
  int pk = k0, pb = b0, left = u1 - u0;  // of the next request
  int run = 0;    // requests until the block or the range ends
  int rows_left;  // groups of the slice from this lane's on
  const int32_t* src;
  auto aim = [&] {
    const int group = (q_lo + pk * KW + kw) * 4 + ct, col = (pb * NB + cw) * kColsPerWarp + cg * 4;
    src = mat + (size_t)group * 3 * row + col;
    rows_left = col < p.width && left > 0 ? g_hi - group : 0;
    run = left > 0 ? min(p.steps - pk, left) : INT_MAX;
    left -= run;
    pk = 0;
    pb++;
  };
  aim();
  auto request = [&](int slot) {
    const uint32_t dst = ring_in + slot * kSlot;
    if (rows_left > 0 && HQ_IN_BOUNDS(src, 16, mat, mat_bytes, 1102) &&
        HQ_IN_BOUNDS(src + 2 * row, 16, mat, mat_bytes, 1103)) {
      copy_16(dst, src);
      copy_16(dst + 512, src + row);
      copy_16(dst + 1024, src + 2 * row);
    }
    src += next;
    rows_left -= 4 * KW;
    if (--run == 0) aim();
    asm volatile("cp.async.commit_group;" ::: "memory");
  };

  // scale and zero of this lane's column in the block, and in the next one: asked for a block ahead, a
  // range of two or three steps would wait for them as long as for its words
  int block = b0;
  float2 par = make_float2(0.f, 0.f), par_next = par;
  auto parameters = [&](int of) {
    const int col = (of * NB + cw) * kColsPerWarp + lane;
    if (col >= p.width || !HQ_IN_BOUNDS(scales + col, 4, scales, column_bytes, 1104)) return make_float2(0.f, 0.f);
    const float s = ld_ordered_f32(scales + col);
    return make_float2(s, ld_ordered_f32(zeros + col));
  };

  // ---- inputs: a warp stages a quad at a time ----
  {
    // lane: pair j of the groups r0 and r0 + 2
    using In = typename std::conditional<F16IN, __half, float>::type;
    const int j = lane & 15, r0 = lane >> 4;
    const int plo = (int)(kFieldsLo >> (4 * j)) & 15, phi = (int)(kFieldsHi >> (4 * j)) & 15;
    const In* const mine_lo = reinterpret_cast<const In*>(vec) + code_lo(j);
    const In* const mine_hi = reinterpret_cast<const In*>(vec) + code_hi(j);
    In raw[4];
    auto load = [&](int i) {
      int st = k0 + i / KW;
      if (st >= p.steps) st -= p.steps;
      const int group = (q_lo + st * KW + i % KW) * 4 + r0;
#pragma unroll
      for (int h = 0; h < 2; h++) {
        raw[2 * h] = raw[2 * h + 1] = (In)0.f;
        if (i < staged * KW && group + 2 * h < g_hi) {
          const size_t at = (size_t)(group + 2 * h) * 32;
          if (!HQ_IN_BOUNDS(mine_lo + at, sizeof(In), vec, vec_bytes, 1105) ||
              !HQ_IN_BOUNDS(mine_hi + at, sizeof(In), vec, vec_bytes, 1106))
            continue;
          if constexpr (F16IN) {
            raw[2 * h] = ld_dependent_f16(mine_lo + at);
            raw[2 * h + 1] = ld_dependent_f16(mine_hi + at);
          } else {
            raw[2 * h] = ld_dependent_f32(mine_lo + at);
            raw[2 * h + 1] = ld_dependent_f32(mine_hi + at);
          }
        }
      }
    };
    load(warp);  // the inputs first: they would queue behind the packed words
#pragma unroll
    for (int d = 0; d < kDepth - 1; d++) request(d);
    par = parameters(b0);
    if ((b0 + 1) * p.steps < u1) par_next = parameters(b0 + 1);
    for (int i = warp; i < staged * KW; i += W) {
      const float x[4] = {(float)raw[0], (float)raw[1], (float)raw[2], (float)raw[3]};
      load(i + W);
      const float sum = warp_sum((x[0] + x[1]) + (x[2] + x[3]));
      int e = 0;
      if (!F16IN) {
        uint32_t m = 0;
#pragma unroll
        for (int r = 0; r < 4; r++) m = max(m, __float_as_uint(x[r]) & 0x7fffffffu);
        e = max(0, (int)(__reduce_max_sync(0xffffffffu, m) >> 23) - 126);  // all of them below 2^e
      }
      if (lane == 0) sums[i] = make_float2(sum, F16IN ? 1.f : pow2f(min(e, 128) - 1));  // (129: an infinity, or no number)
      const int top = F16IN ? 110 : 126 - e;
      const float slo = pow2f(top - plo), shi = pow2f(top - phi);
      unsigned char* const quad = table + (size_t)i * kQuadBytes<F16IN> + (j & 3) * 4;
#pragma unroll
      for (int h = 0; h < 2; h++) {
        float a = x[2 * h] * slo, b = x[2 * h + 1] * shi;
        const int r = 2 * h + r0;
#pragma unroll
        for (int q = 0; q < P; q++) {
          uint32_t ua = __float_as_uint(a), ub = __float_as_uint(b);
          *reinterpret_cast<uint32_t*>(quad + (((j >> 2) * 4 + r) * P + q) * 16) = __byte_perm(ua, ub, 0x7632);
          // an infinity has no rest
          a = isinf(a) ? 0.f : a - __uint_as_float(ua & 0xffff0000u);
          b = isinf(b) ? 0.f : b - __uint_as_float(ub & 0xffff0000u);
        }
      }
    }
  }
  __syncthreads();

  // ---- products ----
  const uint32_t xtab = smem_at(table) + (uint32_t)(kw * kQuadBytes<F16IN> + (t * P + min(g, P - 1)) * 16);
  const float2* const ktab = sums + kw;
  float acc0[4] = {0.f, 0.f, 0.f, 0.f}, acc1[4] = {0.f, 0.f, 0.f, 0.f};
  float sumx = 0.f;
  // a segment: steps of one block whose inputs lie in a row; u, k, at: where it begins
  int u = u0, k = k0, at = 0, seg = 0, todo = 0;
  uint32_t xat = xtab;
  const float2* sat = ktab;
  auto segment = [&] { seg = todo = min(min(p.steps - k, u1 - u), staged - at); };
  segment();
  for (;;) {
#pragma unroll
    for (int slot = 0; slot < kDepth; slot++) {
      asm volatile("cp.async.wait_group %0;" ::"n"(kDepth - 2) : "memory");
      __syncwarp();
      const uint4 w0 = lds_u4(ring_out + slot * kSlot), w1 = lds_u4(ring_out + slot * kSlot + 512),
                  w2 = lds_u4(ring_out + slot * kSlot + 1024);
      uint32_t x[kPairs];
#pragma unroll
      for (int q = 0; q < 4; q++) {
        const uint4 v = lds_u4(xat + (uint32_t)(q * 64 * P));
        x[4 * q] = v.x; x[4 * q + 1] = v.y; x[4 * q + 2] = v.z; x[4 * q + 3] = v.w;
      }
      const float2 sf = *sat;
      xat += KW * kQuadBytes<F16IN>;
      sat += KW;
      request((slot + kDepth - 1) % kDepth);
      const uint32_t c0[3] = {w0.x, w1.x, w2.x}, c1[3] = {w0.y, w1.y, w2.y}, c2[3] = {w0.z, w1.z, w2.z},
                     c3[3] = {w0.w, w1.w, w2.w};
      if constexpr (F16IN) {
        multiply(acc0, c0, c1, x, std::make_integer_sequence<int, kPairs / 2>());
        multiply(acc1, c2, c3, x, std::make_integer_sequence<int, kPairs / 2>());
      } else {
        float d0[4] = {0.f, 0.f, 0.f, 0.f}, d1[4] = {0.f, 0.f, 0.f, 0.f};
        multiply(d0, c0, c1, x, std::make_integer_sequence<int, kPairs / 2>());
        multiply(d1, c2, c3, x, std::make_integer_sequence<int, kPairs / 2>());
#pragma unroll
        for (int i = 0; i < 4; i++) {
          acc0[i] = fmaf(d0[i], sf.y, acc0[i]);
          acc1[i] = fmaf(d1[i], sf.y, acc1[i]);
        }
      }
      sumx += sf.x;
      if (--todo == 0) {
        u += seg;
        k += seg;
        at += seg;
        if (at == staged) {
          at = 0;
          xat = xtab;
          sat = ktab;
        }
        if (k == p.steps || u == u1) {
          // the pieces of the inputs are columns 0 .. P - 1 of the sums: lanes t = 0 and, of the third, t = 1
          const bool first = t == 0, any = P == 3 ? t < 2 : first;
          float s[4];
#pragma unroll
          for (int i = 0; i < 4; i++) {
            const float a = i < 2 ? acc0[2 * i] : acc1[2 * i - 4], b = i < 2 ? acc0[2 * i + 1] : acc1[2 * i - 3];
            s[i] = (any ? a : 0.f) + (first ? b : 0.f);
            s[i] += __shfl_xor_sync(0xffffffffu, s[i], 1);
            s[i] += __shfl_xor_sync(0xffffffffu, s[i], 2);
          }
          // lane = column of the warp
          float q = t == 0 ? s[0] : t == 1 ? s[1] : t == 2 ? s[2] : s[3];
          q *= F16IN ? pow2f(23) : pow2f(8);
          const int col = (block * NB + cw) * kColsPerWarp + lane;
          // (fp16 inputs: the reference rounds both parameters to fp16, kernels.h:121-122)
          const float sc = F16IN ? __half2float(__float2half_rn(par.x)) : par.x;
          const float nz = F16IN ? __half2float(__float2half_rn(-par.y)) : -par.y;
          if (col < p.width && HQ_IN_BOUNDS(mul + col, 4, mul, column_bytes, 1107)) atomicAdd(&mul[col], fmaf(sc, q, nz * sumx));
#pragma unroll
          for (int i = 0; i < 4; i++) acc0[i] = acc1[i] = 0.f;
          sumx = 0.f;
          if (u == u1) return;
          k = 0;
          block++;
          par = par_next;
          if ((block + 1) * p.steps < u1) par_next = parameters(block + 1);
        }
        segment();
      }
    }
  }
}

// W[k][c] for one (group, 4 columns) per thread; bit-exact dequant rules.
template <bool F16OUT>
__global__ void __launch_bounds__(256)
q3_dequant_kernel(const int32_t* __restrict__ mat, const float* __restrict__ scales,
                  const float* __restrict__ zeros, void* __restrict__ W_, int groups,
                  int width) {
  const int c = (blockIdx.x * 256 + threadIdx.x);
  const int r = blockIdx.y;
  if (c >= width) return;
  const uint32_t w0 = (uint32_t)mat[(size_t)(3 * r) * width + c];
  const uint32_t w1 = (uint32_t)mat[(size_t)(3 * r + 1) * width + c];
  const uint32_t w2 = (uint32_t)mat[(size_t)(3 * r + 2) * width + c];
  const float sc = scales[c], z = zeros[c];
  const __half sch = __float2half_rn(sc), nzh = __float2half_rn(-z);
#pragma unroll
  for (int j = 0; j < 32; j++) {
    const int bit = 3 * j;
    uint32_t q;
    if (bit + 3 <= 32) q = (w0 >> bit) & 7u;
    else if (bit < 32) q = __funnelshift_r(w0, w1, bit) & 7u;
    else if (bit + 3 <= 64) q = (w1 >> (bit - 32)) & 7u;
    else if (bit < 64) q = __funnelshift_r(w1, w2, bit - 32) & 7u;
    else q = (w2 >> (bit - 64)) & 7u;
    const size_t o = (size_t)(32 * r + j) * width + c;
    if (F16OUT) {
      reinterpret_cast<__half*>(W_)[o] = __hfma(__int2half_rn((int)q), sch, nzh);
    } else {
      reinterpret_cast<float*>(W_)[o] = fmaf(sc, (float)q, -z);
    }
  }
}

template <bool F16IN, int W, int NB>
int q3_gemv_go(const void* vec, const int32_t* mat, float* mul, const float* scales, const float* zeros,
               Shape p, int slices, hq_stream_t stream) {
  constexpr int KW = W / NB;
  p.blocks = (p.width + NB * kColsPerWarp - 1) / (NB * kColsPerWarp);
  p.steps = (p.slice_quads + KW - 1) / KW;
  const long long total = (long long)p.blocks * p.steps;
  const int grid = (int)min(total, (long long)max(1, sm_count() / slices));
  p.share = (int)(total / grid);
  p.over = (int)(total % grid);
  p.staged = min(p.steps, p.share + (p.over ? 1 : 0));
  const size_t smem = (size_t)W * kDepth * kSlot + (size_t)p.staged * KW * (kQuadBytes<F16IN> + sizeof(float2));
  constexpr auto kern = q3_gemv_kernel<F16IN, W, NB>;
  cudaError_t e = ensure_dynamic_smem<kern>(smem);
  if (e != cudaSuccess) return cuda_status(e);
  return cuda_status(launch_pdl(kern, dim3(grid, slices), dim3(W * 32), smem, (cudaStream_t)stream, vec, mat, mul,
                                scales, zeros, p));
}

template <bool F16IN>
int q3_gemv_launch(const void* vec, const int32_t* mat, float* mul, const float* scales,
                   const float* zeros, int height, int width, hq_stream_t stream) {
  if (!vec || !mat || !mul || !scales || !zeros) return HQ_ERR_NULL_POINTER;
  if (height <= 0 || width <= 0 || height % 3 != 0 || width % 4 != 0) return HQ_ERR_BAD_SHAPE;
  if (!aligned16(mat)) return HQ_ERR_MISALIGNED;
  if (!aligned4(vec) || !aligned4(mul)) return HQ_ERR_MISALIGNED;
  Shape p;
  p.width = width;
  p.groups = height / 3;
  // a CTA holds the inputs of a slice, 16384 of them at most (96 KB, fp32)
  const int quads = (p.groups + 3) / 4;
  const int slices = (quads + kSliceQuads - 1) / kSliceQuads;
  p.slice_quads = (quads + slices - 1) / slices;
  const int slots = max(1, sm_count() / slices);
  // Steps of the CTA that has most of them, W warps, NB side by side.  The widest block (whole
  // lines of DRAM pages, one set of inputs) unless a narrower one leaves less of its last block empty: 4100 columns
  // of 33 quads are 3 steps with 16 warps side by side and 2 with 8.
  auto longest = [&](int w, int nb) {
    const long long blocks = (width + nb * kColsPerWarp - 1) / (nb * kColsPerWarp);
    const long long steps = (p.slice_quads + w / nb - 1) / (w / nb);
    return (blocks * steps + slots - 1) / slots;
  };
  auto narrow = [&](int w) {  // log2 of W / NB
    int n = 0;
    for (int i = 1; i <= 2; i++)
      if (longest(w, w >> i) < longest(w, w >> n)) n = i;
    return n;
  };
  // 20 warps hide more of what a step waits for and take the same time for a warp's share of it: us in
  // graphs, 16 and 20 warps, at 20 l20 / 16 l16 of 0.62 (8804 x 1280) 3.5 and 2.9, 0.83 (5116 x 4288) 4.6 and 4.4, 0.95
  // (26236 x 7232) 17.1 and 16.3, 1 (36388 x 16128) 43.4 and 41.1, 1.04 (10012 x 5248) 7.6 and 7.9, 1.25 (11124 x
  // 1664) 4.1 and 4.6.
  const int n16 = narrow(16), n20 = narrow(20);
  const long long l16 = longest(16, 16 >> n16), l20 = longest(20, 20 >> n20);
  const bool wide = 20 * l20 <= 16 * l16;
  // 8 warps start sooner, and a layer of few steps, a step being W / 8 of theirs, wastes less of its last one: us
  // in graphs, words from HBM, 16 or 20 warps -> 8, at steps of 8 of 0.2 (512 x 1024) 2.5 -> 1.9, 1.7 (1408 x 5440,
  // fp32) 2.93 -> 2.89, 2.4 (4096 x 4096, fp32) 4.05 -> 3.80, 2.5 (11148 x 1088, fp32) 4.00 -> 3.57, 2.9 (1808 x 6784, fp32)
  // 4.00 -> 3.44, 4.5 (4096 x 5376) 4.76 -> 4.43.  One step of 20 warps is the better at 2 to 2.5 (1.05); with more than five
  // steps too few words are on their way (1.02 to 1.06 up to seven, then 1.2).
  const long long l8 = longest(8, 8);
  if (l8 <= 5 && 8 * l8 <= min(16 * l16, 20 * l20))
    return q3_gemv_go<F16IN, 8, 8>(vec, mat, mul, scales, zeros, p, slices, stream);
  switch (wide ? 3 + n20 : n16) {
    case 0: return q3_gemv_go<F16IN, 16, 16>(vec, mat, mul, scales, zeros, p, slices, stream);
    case 1: return q3_gemv_go<F16IN, 16, 8>(vec, mat, mul, scales, zeros, p, slices, stream);
    case 2: return q3_gemv_go<F16IN, 16, 4>(vec, mat, mul, scales, zeros, p, slices, stream);
    case 3: return q3_gemv_go<F16IN, 20, 20>(vec, mat, mul, scales, zeros, p, slices, stream);
    case 4: return q3_gemv_go<F16IN, 20, 10>(vec, mat, mul, scales, zeros, p, slices, stream);
    default: return q3_gemv_go<F16IN, 20, 5>(vec, mat, mul, scales, zeros, p, slices, stream);
  }
}

template <bool F16OUT>
int q3_dequant_launch(const int32_t* mat, const float* scales, const float* zeros, void* W,
                      int height, int width, hq_stream_t stream) {
  if (!mat || !scales || !zeros || !W) return HQ_ERR_NULL_POINTER;
  if (height <= 0 || width <= 0 || height % 3 != 0) return HQ_ERR_BAD_SHAPE;
  dim3 grid((width + 255) / 256, height / 3);
  q3_dequant_kernel<F16OUT><<<grid, 256, 0, (cudaStream_t)stream>>>(mat, scales, zeros, W,
                                                                  height / 3, width);
  return launch_status();
}

}  // namespace
}  // namespace hq

extern "C" {

int hq_q3_gemv_f32(const float* vec, const int32_t* mat, float* mul, const float* scales,
                   const float* zeros, int height, int width, hq_stream_t stream) {
  return hq::q3_gemv_launch<false>(vec, mat, mul, scales, zeros, height, width, stream);
}

int hq_q3_gemv_f16in(const void* vec_half, const int32_t* mat, float* mul, const float* scales,
                     const float* zeros, int height, int width, hq_stream_t stream) {
  return hq::q3_gemv_launch<true>(vec_half, mat, mul, scales, zeros, height, width, stream);
}

int hq_q3_dequant_f32(const int32_t* mat, const float* scales, const float* zeros, float* W,
                      int height, int width, hq_stream_t stream) {
  return hq::q3_dequant_launch<false>(mat, scales, zeros, W, height, width, stream);
}

int hq_q3_dequant_f16(const int32_t* mat, const float* scales, const float* zeros, void* W_half,
                      int height, int width, hq_stream_t stream) {
  return hq::q3_dequant_launch<true>(mat, scales, zeros, W_half, height, width, stream);
}

}  // extern "C"
