// AQLM additive-codebook mat-vec for sm_100a: 1x16 (one 65536-entry codebook,
// uint16 codes) and 2x8 (two 256-entry codebooks, uint8 codes).
//
// 1x16 follows the arithmetic of Code1x16MatVec (quantAQLM-cuda/main.cu:31-111)
// exactly - lane l of a row's warp takes the 16-byte code vectors l, l+32, ...;
// each code gathers a 16-byte codebook row, four hfma2 against the matching
// 8 inputs, the two halves are added to the lane's fp32 sum, lanes are combined
// with the shfl_down tree - so results are bit-identical to the reference
// kernel.  What changes is the memory behaviour: all code vectors of a row and
// all their 16-byte gathers are issued before any arithmetic (up to 16 gathers
// in flight per lane instead of 1), a warp walks several rows, and the 1 MiB
// codebook goes through L1 and stays L2-resident while the codes stream past it
// without allocating in L1.
//
// 2x8: both codebooks (8 KiB) live in shared memory, replicated 8 times with
// entry e of replica r at 16-byte slot 8*e + r, so the 8 lanes that a 128-bit
// shared load serves per cycle (r = lane % 8) always hit distinct bank groups.
#include <algorithm>

#include "hq_common.cuh"

namespace hq {
namespace {

constexpr int kWarps1x16 = 8;
constexpr int kWarps2x8 = 8;
// Rows per warp: 4 when that still gives every SM two CTAs, else 2 (a 4096-row
// layer is latency-bound: more resident warps pay more than the per-CTA staging
// of the inputs costs: 12.5 -> 11.0 us for 1x16, 11.5 -> 8.0 us for 2x8).
inline int rows_per_warp_for(int prob_m, int warps) {
  return prob_m / (warps * 4) >= 2 * sm_count() ? 4 : 2;
}
// How runs of rows_per_warp rows are divided: run warp * per_warp + CTA * per_cta goes to a warp.  Dealt one
// by one over as many CTAs for every SM (per_cta = 1) the SMs have the same number of rows: the
// gathers are bound by each SM's L1, and in blocks of a run for each warp the fullest SM has 32 rows of a 4096-row
// layer where 27.7 are even, and a 1024-row layer is on 64 SMs.  us of a call among others, blocks -> dealt:
// 1x16 300 x 4096 8.2 -> 3.7, 1024 x 8192 12.3 -> 6.9, 4096 x 4096 11.0 -> 10.0, 8192 x 4096 20.6 -> 18.4,
// 14336 x 4096 36.9 -> 30.8; 2x8 4096 x 4096 8.4 -> 6.6, 3000 x 2048 6.7 -> 4.5, 11008 x 4096 15.5 -> 14.5.  Blocks
// stay where they are nearly even (2x8 2368 x 4096 7.2, dealt 7.6), and where the CTAs per SM would leave
// a slot free for an uneven start of the next launch (1x16, three of four: 6144 x 4096 16.0 and 17.3) or not fit
// at once (2x8, more than three: 14336 x 4096 24.0 and 25.8).  fit: how many a 2x8 SM holds, three up to
// 4992 inputs and two beyond.  Where more are dealt each of them stages the codebooks again, for a last
// round that blocks may leave nearly empty: 4737 x 8192 14.2 us, dealt 20.8, 9473 x 5056 18.2 and 29.0, 6144 x
// 6144 17.4 and 17.3.  Only long rows pay for that, from a tenth of a round on (11008 x 8192 38.2, dealt
// 36.5, 6144 x 14336 35.5 and 34.4; rows of a CTA x inputs from some 150000 on, 5504 x 6144 15.7 and 16.4).
// 1x16, which stages nothing but its inputs, gains dealt whatever fits (14240 x 8192, one per SM, 72.6 -> 60.8).
// Lines: by CTAs per SM, one to four, how full blocks must be to stay (0: always).  2x8, blocks and dealt: 2048 x
// 4096 (0.86 of one) 7.2 and 7.2, 2240 x 4096 (0.95) 7.2 and 7.7; 4480 x 4096 (0.95 of two) 8.3 and 7.0; 6300 x 4096
// (0.89 of three) 9.03 and 8.87, 6656 x 4096 (0.94) 9.05 and 9.2, 13312 x 4096 (0.94) 15.6 and 15.9; where three
// do not fit 13400 x 8192 (0.94) 38.8 and 38.2.
using Lines = double[4];
constexpr Lines kDealt1x16 = {0.95, 0.95, 0, 0.95}, kDealt2x8 = {0.88, 0.95, 0.91, 0};
struct Runs {
  int ctas, per_warp, per_cta;
};
inline Runs divide_rows(int prob_m, int warps, int rows_per_warp, const Lines& dealt_below, int fit = 4,
                        bool long_rows = true) {
  const int sms = sm_count(), per_cta = warps * rows_per_warp;
  const int blocks = prob_m / per_cta + (prob_m % per_cta != 0), each = (blocks + sms - 1) / sms;
  if (each > 4 || dealt_below[each - 1] == 0) return {blocks, 1, warps};
  if (blocks >= (each > fit ? 0.95 : dealt_below[each - 1]) * each * sms) return {blocks, 1, warps};
  if (each > fit && (!long_rows || blocks < (each - 0.9) * sms)) return {blocks, 1, warps};
  const int ctas = std::min(prob_m / rows_per_warp + (prob_m % rows_per_warp != 0), each * sms);
  return {ctas, ctas, 1};
}
__device__ __forceinline__ int first_row(const Runs& r, int warp, int rows_per_warp) {
  return (warp * r.per_warp + (int)blockIdx.x * r.per_cta) * rows_per_warp;
}
constexpr int kPad = 9;  // input slots per 8 groups (one pad slot: conflict-free 128-bit reads)

__device__ __forceinline__ float dot8_ref_order(const uint4& a, const uint4& b) {
  // res2 = hfma2(a[j], b[j], res2), j = 0..3, from zero; float(res2.x) + float(res2.y)
  __half2 r = __float2half2_rn(0.f);
  r = __hfma2(u32_as_half2(a.x), u32_as_half2(b.x), r);
  r = __hfma2(u32_as_half2(a.y), u32_as_half2(b.y), r);
  r = __hfma2(u32_as_half2(a.z), u32_as_half2(b.z), r);
  r = __hfma2(u32_as_half2(a.w), u32_as_half2(b.w), r);
  return __half2float(__low2half(r)) + __half2float(__high2half(r));
}

constexpr int kMaxVpl1x16 = 4;  // code vectors per lane and row: up to 8192 inputs

// Four of a thread's 16-byte pieces of the inputs, g0, g0 + 256, ...: all loads in
// flight, then to shared memory.
struct InputPieces {
  uint4 v[4];
  __device__ __forceinline__ void load(const uint4* x, int groups, int g0) {
#pragma unroll
    for (int i = 0; i < 4; i++)
      if (g0 + i * 256 < groups) v[i] = ld_dependent_u4(x + g0 + i * 256);
  }
  __device__ __forceinline__ void store(uint4* sh_x, int groups, int g0) const {
#pragma unroll
    for (int i = 0; i < 4; i++) {
      const int g = g0 + i * 256;
      if (g < groups) sh_x[kPad * (g >> 3) + (g & 7)] = v[i];
    }
  }
};
static_assert(kWarps1x16 * 32 == 256 && kWarps2x8 * 32 == 256, "stride of InputPieces");
static_assert(kMaxVpl1x16 * 32 * 8 <= 4 * 256, "the 1x16 kernel stages its inputs in one turn");

// VPL = 16-byte code vectors per lane per row (prob_k / 64 / 32 rounded up),
// RPW = rows per warp.  The dependent chain code -> codebook row -> FMA is what
// bounds this kernel, so everything that does not depend on the input vector
// is issued early: the code vectors of ALL rows of the warp, the inputs, then,
// as the codes arrive, the gathers of the first vector; the inputs go to shared
// memory while those are under way, and afterwards the gathers of vector u + 1
// are in flight while vector u is multiplied.  The arithmetic (and its order) is
// the reference's.
template <int VPL, int RPW>
__global__ void __launch_bounds__(kWarps1x16 * 32)
aqlm_1x16_kernel(const uint4* codes, const uint4* x,
                 __half* __restrict__ out, const uint4* codebook, int prob_m,
                 int prob_k, int4 cb_sizes, int cb_stride, const __half* scales, const Runs runs) {
  extern __shared__ __align__(16) uint4 sh_x[];  // padded inputs: slot 9*(g/8) + g%8
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int groups = prob_k >> 3;    // 16-byte input groups
  const int vec_per_row = prob_k >> 6;
  const int row_begin = first_row(runs, warp, RPW);
  // the next kernel of the stream may become resident while this grid drains;
  // nothing is read or written before every earlier kernel has completed (codes,
  // codebook and scales may be their output: ordered loads below)
  pdl_launch_dependents();
  pdl_wait();
  constexpr int kUnits = RPW * VPL;  // unit u = (row u / VPL, vector u % VPL)

  uint4 cv[kUnits];
#pragma unroll
  for (int u = 0; u < kUnits; u++) {
    const int m = row_begin + u / VPL, idx = lane + 32 * (u % VPL);
    cv[u] = (m < prob_m && idx < vec_per_row)
                ? ld_ordered_stream_u4(codes + (size_t)m * vec_per_row + idx)
                : make_uint4(0, 0, 0, 0);
  }
  auto book = [&](int m) {
    const uint4* cb = codebook;
    if (m >= cb_sizes.x) cb += cb_stride;
    if (m >= cb_sizes.y) cb += cb_stride;
    if (m >= cb_sizes.z) cb += cb_stride;
    return cb;
  };
  auto gather = [&](int u, uint4 (&rows)[8]) {
    const int m = row_begin + u / VPL, idx = lane + 32 * (u % VPL);
    if (m < prob_m && idx < vec_per_row) {
      const uint4* cb = book(m);
      const uint32_t cw[4] = {cv[u].x, cv[u].y, cv[u].z, cv[u].w};
#pragma unroll
      for (int i = 0; i < 8; i++)
        rows[i] = ld_ordered_u4(cb + ((cw[i >> 1] >> (16 * (i & 1))) & 0xffffu));
    }
  };
  // at most 1024 pieces of inputs: four per thread, requested before the first
  // gather waits for its codes
  InputPieces xin;
  xin.load(x, groups, tid);
  uint4 rows[2][8];
  gather(0, rows[0]);

  xin.store(sh_x, groups, tid);
  __syncthreads();

  float res = 0.f;
#pragma unroll
  for (int u = 0; u < kUnits; u++) {
    if (u + 1 < kUnits) gather(u + 1, rows[(u + 1) & 1]);
    const int m = row_begin + u / VPL, idx = lane + 32 * (u % VPL);
    if (m < prob_m && idx < vec_per_row) {
#pragma unroll
      for (int i = 0; i < 8; i++) res += dot8_ref_order(rows[u & 1][i], sh_x[kPad * idx + i]);
    }
    if (u % VPL == VPL - 1) {  // the row is complete
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) res += __shfl_down_sync(0xffffffffu, res, o);
      if (lane == 0 && m < prob_m) {
        if (scales != nullptr) res *= __half2float(ld_ordered_f16(scales + m));
        out[m] = __float2half(res);
      }
      res = 0.f;
    }
  }
}

// DEALT: the division with per_cta = 1 (as launch parameters it took 2 to 8 % of a small layer's time)
template <bool DEALT>
__global__ void __launch_bounds__(kWarps2x8 * 32)
aqlm_2x8_kernel(const uint4* codes, const uint4* x,
                __half* __restrict__ out, const uint4* codebooks, int prob_m,
                int prob_k, const __half* scales, int rows_per_warp) {
  extern __shared__ __align__(16) uint4 smem4[];
  uint4* cbs = smem4;                  // [2][256][8 replicas]
  uint4* sh_x = smem4 + 2 * 256 * 8;   // padded inputs
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int groups = prob_k >> 3;
  const int vec_per_row = prob_k >> 6;  // 16 bytes = 8 groups x 2 codes
  pdl_launch_dependents();  // as in the 1x16 kernel
  pdl_wait();
  constexpr int kThreads2x8 = kWarps2x8 * 32, kBatch = 8;  // entries requested at a time
#pragma unroll
  for (int i0 = 0; i0 < 2 * 256 * 8; i0 += kBatch * kThreads2x8) {
    uint4 e[kBatch];
#pragma unroll
    for (int b = 0; b < kBatch; b++)
      e[b] = ld_ordered_u4(codebooks + ((i0 + b * kThreads2x8 + tid) >> 3));
#pragma unroll
    for (int b = 0; b < kBatch; b++) cbs[i0 + b * kThreads2x8 + tid] = e[b];
  }
  for (int g0 = tid; g0 < groups; g0 += 4 * 256) {
    InputPieces xin;
    xin.load(x, groups, g0);
    xin.store(sh_x, groups, g0);
  }
  __syncthreads();

  const uint4* cb0 = cbs + (lane & 7);
  const uint4* cb1 = cbs + 256 * 8 + (lane & 7);
  const int row_begin = (DEALT ? warp * (int)gridDim.x + (int)blockIdx.x : (int)blockIdx.x * kWarps2x8 + warp) * rows_per_warp;
  for (int rr = 0; rr < rows_per_warp; rr++) {
    const int m = row_begin + rr;
    if (m >= prob_m) break;
    const uint4* crow = codes + (size_t)m * vec_per_row;
    float res = 0.f;
    for (int idx = lane; idx < vec_per_row; idx += 32) {
      const uint4 cv = ld_ordered_stream_u4(crow + idx);
      const uint32_t cw[4] = {cv.x, cv.y, cv.z, cv.w};
#pragma unroll
      for (int i = 0; i < 8; i++) {
        const uint32_t pair = (cw[i >> 1] >> (16 * (i & 1))) & 0xffffu;
        const uint4 a0 = cb0[(pair & 0xffu) * 8];
        const uint4 a1 = cb1[(pair >> 8) * 8];
        const uint4 b = sh_x[kPad * idx + i];
        __half2 r = __float2half2_rn(0.f);
        r = __hfma2(u32_as_half2(a0.x), u32_as_half2(b.x), r);
        r = __hfma2(u32_as_half2(a0.y), u32_as_half2(b.y), r);
        r = __hfma2(u32_as_half2(a0.z), u32_as_half2(b.z), r);
        r = __hfma2(u32_as_half2(a0.w), u32_as_half2(b.w), r);
        r = __hfma2(u32_as_half2(a1.x), u32_as_half2(b.x), r);
        r = __hfma2(u32_as_half2(a1.y), u32_as_half2(b.y), r);
        r = __hfma2(u32_as_half2(a1.z), u32_as_half2(b.z), r);
        r = __hfma2(u32_as_half2(a1.w), u32_as_half2(b.w), r);
        res += __half2float(__low2half(r)) + __half2float(__high2half(r));
      }
    }
    res = warp_sum(res);
    if (lane == 0) {
      if (scales != nullptr) res *= __half2float(ld_ordered_f16(scales + m));
      out[m] = __float2half_rn(res);
    }
  }
}

template <auto Kern>
struct Form {
  static constexpr auto value = Kern;
};

}  // namespace
}  // namespace hq

extern "C" {

int hq_aqlm_1x16_matvec(const void* codes, const void* x_half, void* out_half, const void* codebook,
                        int prob_m, int prob_k, const int cb_sizes[4], int cb_stride_int4,
                        const void* scales_half, hq_stream_t stream) {
  using namespace hq;
  if (!codes || !x_half || !out_half || !codebook || !cb_sizes) return HQ_ERR_NULL_POINTER;
  if (prob_m <= 0 || prob_k <= 0 || prob_k % 64 != 0) return HQ_ERR_BAD_SHAPE;
  if (!aligned16(codes) || !aligned16(x_half) || !aligned16(codebook)) return HQ_ERR_MISALIGNED;
  const int vec_per_row = prob_k / 64;
  const int vpl = (vec_per_row + 31) / 32;
  if (vpl > kMaxVpl1x16) return HQ_ERR_TOO_LARGE;
  const int groups = prob_k / 8;
  const size_t smem = (size_t)kPad * ((groups + 7) / 8) * 16;
  const int rows_per_warp = rows_per_warp_for(prob_m, kWarps1x16);
  const Runs runs = divide_rows(prob_m, kWarps1x16, rows_per_warp, kDealt1x16);
  const int grid = runs.ctas;
  // A grid that fills the SMs starts while the one before it drains (4096 x 4096
  // back to back: 12.4 -> 11.0 us; in a replayed graph 10.7 -> 10.6, and 2368 x 4096,
  // 148 CTAs, 6.6 -> 6.4).  A smaller one does not: the CTAs of an early start are not
  // spread over all SMs, and the gathers are bound by each SM's L1 (1024 x 8192 in 64 CTAs: 13.2
  // us, 18.9 with the early start; 2048 x 4096 in 128, in a graph, 6.6 and 10.0).  Dealt over 148 it does: 1024
  // x 8192 6.9, in a graph 6.5 (in blocks 11.0), 2048 x 4096 6.6, in a graph 6.3 (7.0).
  const int4 sizes = make_int4(cb_sizes[0], cb_sizes[1], cb_sizes[2], cb_sizes[3]);
  cudaStream_t st = (cudaStream_t)stream;
#define HQ_AQLM_LAUNCH(VPL, RPW)                                                             \
  {                                                                                          \
    constexpr auto kern = aqlm_1x16_kernel<VPL, RPW>;                                        \
    if (smem > 48 * 1024) {                                                                  \
      cudaError_t e = ensure_dynamic_smem<kern>(smem);                                       \
      if (e != cudaSuccess) return cuda_status(e);                                           \
    }                                                                                        \
    const auto c = reinterpret_cast<const uint4*>(codes);                                    \
    const auto x = reinterpret_cast<const uint4*>(x_half);                                   \
    const auto o = reinterpret_cast<__half*>(out_half);                                      \
    const auto cb = reinterpret_cast<const uint4*>(codebook);                                \
    const auto sc = reinterpret_cast<const __half*>(scales_half);                            \
    if (grid >= sm_count())                                                                  \
      return cuda_status(launch_pdl(kern, dim3(grid), dim3(kWarps1x16 * 32), smem, st, c, x, o, \
                                    cb, prob_m, prob_k, sizes, cb_stride_int4, sc, runs));   \
    kern<<<grid, kWarps1x16 * 32, smem, st>>>(c, x, o, cb, prob_m, prob_k, sizes,            \
                                              cb_stride_int4, sc, runs);                     \
  }
#define HQ_AQLM_ROWS(VPL)                                \
  if (rows_per_warp == 4) HQ_AQLM_LAUNCH(VPL, 4)         \
  else HQ_AQLM_LAUNCH(VPL, 2)
  switch (vpl) {
    case 1: HQ_AQLM_ROWS(1) break;
    case 2: HQ_AQLM_ROWS(2) break;
    case 3: HQ_AQLM_ROWS(3) break;
    default: HQ_AQLM_ROWS(4) break;
  }
#undef HQ_AQLM_ROWS
#undef HQ_AQLM_LAUNCH
  return launch_status();
}

int hq_aqlm_2x8_matvec(const void* codes, const void* x_half, void* out_half, const void* codebooks,
                       int prob_m, int prob_k, const void* scales_half, hq_stream_t stream) {
  using namespace hq;
  if (!codes || !x_half || !out_half || !codebooks) return HQ_ERR_NULL_POINTER;
  if (prob_m <= 0 || prob_k <= 0 || prob_k % 64 != 0) return HQ_ERR_BAD_SHAPE;
  if (!aligned16(codes) || !aligned16(x_half) || !aligned16(codebooks)) return HQ_ERR_MISALIGNED;
  const int groups = prob_k / 8;
  const size_t smem = (size_t)2 * 256 * 8 * 16 + (size_t)kPad * ((groups + 7) / 8) * 16;
  if (smem > 220 * 1024) return HQ_ERR_TOO_LARGE;
  const int rows_per_warp = rows_per_warp_for(prob_m, kWarps2x8);
  const int fit = (int)((size_t)228 * 1024 / (smem + 1024));  // CTAs that an SM holds, 1 KiB of each reserved
  const bool long_rows = (long long)kWarps2x8 * rows_per_warp * prob_k >= 150000;
  const Runs runs = divide_rows(prob_m, kWarps2x8, rows_per_warp, kDealt2x8, fit, long_rows);
  const int grid = runs.ctas;
  const auto c = reinterpret_cast<const uint4*>(codes);
  const auto x = reinterpret_cast<const uint4*>(x_half);
  const auto o = reinterpret_cast<__half*>(out_half);
  const auto cb = reinterpret_cast<const uint4*>(codebooks);
  const auto sc = reinterpret_cast<const __half*>(scales_half);
  const cudaStream_t st = (cudaStream_t)stream;
  // Early start as for 1x16, from two CTAs per SM on.  The CTAs of an early start would
  // go wherever there is room; shared memory is asked for so that an SM holds no more of
  // them than the fullest SM takes anyway.  Three of up to 4992 inputs would fit: 296
  // CTAs (4736 x 4096) 7.6 us in a graph and 10.3 as calls without the early start, 9.2
  // and 9.3 with it, 7.5 and 7.8 held to two per SM; 9472 x 4096, 296 CTAs of 32 rows:
  // 12.6 and 14.5, 15.4 and 15.5, 12.5 and 12.7.
  const int per_sm = (grid + sm_count() - 1) / sm_count();
  const size_t share = (size_t)228 * 1024 / (per_sm + 1);  // 1 KiB of it is reserved per CTA
  const size_t request = std::max(smem, share > 1024 ? share - 1024 + 16 : 0);
  auto go = [&](auto form) {
    constexpr auto kern = decltype(form)::value;
    const cudaError_t e = ensure_dynamic_smem<kern>(request);
    if (e != cudaSuccess) return cuda_status(e);
    if (grid >= 2 * sm_count())
      return cuda_status(launch_pdl(kern, dim3(grid), dim3(kWarps2x8 * 32), request, st, c, x, o, cb, prob_m,
                                    prob_k, sc, rows_per_warp));
    kern<<<grid, kWarps2x8 * 32, smem, st>>>(c, x, o, cb, prob_m, prob_k, sc, rows_per_warp);
    return launch_status();
  };
  return runs.per_cta == 1 ? go(Form<aqlm_2x8_kernel<true>>()) : go(Form<aqlm_2x8_kernel<false>>());
}

}  // extern "C"
