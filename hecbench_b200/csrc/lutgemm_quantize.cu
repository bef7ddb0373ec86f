// Greedy binary-coding quantizer for sm_100a: fp16 / bf16 / fp32 weights W[K][M]
// -> the sign planes, scales and offsets that the LUT-GEMM mat-vec
// (hq_lutgemm_nqmv, the layouts of lut-gemm-cuda/main.cu:27-30,118-134) consumes.
// The reference tree holds only the consumer; the rule is the greedy
// binary-coding quantization the format comes from, per output column m and group
// g of group_size consecutive inputs, in fp32:
//   q_bias[g][m] = half(mean of the group)                  (when offsets are asked for)
//   r = w - q_bias;  for b = 0 .. nb - 1:
//     alpha[g][b][m] = half(mean |r|);  bit = r >= 0;  r -= +-alpha (the rounded value)
// and bit t of bW[k / 32][b][m] is the bit of input k = 32 (k / 32) + t.  A sum
// over a group is formed as one sum per 32 consecutive inputs (ascending k),
// and those partial sums are added in ascending order.
//
// Design: the summation order is the kernel's shape.  A thread holds 32
// consecutive inputs of two adjacent columns in registers - exactly the inputs of
// one output word per column and plane - warp w of a CTA the w-th run of 32 inputs
// of the group, the lanes 64 adjacent columns (one 32-bit load per lane and row,
// 128 contiguous bytes per warp).  Per plane the warps exchange their partial
// sums through shared memory (one barrier), every thread adds them in order,
// takes the signs of its residuals, updates them in registers and stores its two
// words.  The weights are read once; nothing else touches memory.
// The bound is instruction issue (20.2 per weight for three planes, 85 % of the
// slots busy): the bits come from the residual's sign (one funnel shift per weight
// instead of a comparison, a select and a merge), the update puts the sign on
// -alpha with one logic operation, and update, bits and the next plane's
// magnitudes share one pass.  12288 x 12288 fp16, three planes: 164 -> 101 us.
// Packed two-lane fp32 additions were no faster, neither were six CTAs per SM (spills).
// The kernel may become resident while the launch before it drains: 4096 x 4096 of a call
// among others 15.6 -> 13.6 us, 12288 x 12288 101.6 -> 100.0.
#include <cuda_bf16.h>

#include <algorithm>
#include <climits>

#include "hq_common.cuh"

namespace hq {
namespace {

constexpr int kColsPerCta = 64;   // two per lane
constexpr int kMaxRuns = 16;      // runs of 32 inputs per group = warps per CTA (group_size <= 512)

// Whether a row of the weights is less than 4 GiB, so that its length fits 32 bits (the
// 64-bit form of the addresses costs 1 to 4 %).
constexpr bool row_fits_32(int M, int bytes) { return (unsigned)M <= 0xffffffffu / bytes; }
static_assert(!row_fits_32(1 << 30, 4) && row_fits_32((1 << 30) - 2, 4) && row_fits_32(INT_MAX, 2),
              "fp32 rows of 2^30 columns on are longer");

// RUNS: runs of 32 inputs per group where it is a compile-time constant, else 0.
// Pitch: the type that holds the bytes of a row.
template <int DTYPE, int RUNS, typename Pitch>
__global__ void __launch_bounds__(RUNS ? RUNS * 32 : kMaxRuns * 32)
bcq_quantize_kernel(const void* W, int K, int M, int nb, int gs,
                    uint32_t* __restrict__ bW, __half* __restrict__ alpha,
                    __half* __restrict__ q_bias) {
  pdl_launch_dependents();
  pdl_wait();  // nothing is read or written before every earlier kernel has completed
  __shared__ float2 s_part[2][RUNS ? RUNS : kMaxRuns][kColsPerCta / 2];  // [parity][run][column pair]
  const int lane = threadIdx.x & 31, run = threadIdx.x >> 5, runs = RUNS ? RUNS : gs >> 5;
  const int g = blockIdx.y;
  const int m = blockIdx.x * kColsPerCta + 2 * lane;  // this thread's first column
  const bool live = m < M;                            // M is even: both columns or none
  const int k0 = g * gs + run * 32;                   // this thread's first input
  const size_t total = (size_t)K * M;
  (void)total;
  // the 32 inputs of the two columns; a lane beyond the last column reads the last pair again
  float2 r[32];
  {
    constexpr int kBytes = DTYPE == HQ_DTYPE_F32 ? 4 : 2;
    const char* p = reinterpret_cast<const char*>(W) + ((size_t)k0 * M + min(m, M - 2)) * kBytes;
    const Pitch step = (Pitch)(unsigned)M * kBytes;
#pragma unroll
    for (int t = 0; t < 32; t++) {
      const char* at = p + (unsigned long long)t * step;
      if (!HQ_IN_BOUNDS(at, 2 * kBytes, W, total * kBytes, 1001)) {
        r[t] = make_float2(0.f, 0.f);
      } else if (DTYPE == HQ_DTYPE_F32) {
        const uint2 a = ld_ordered_stream_u2(at);
        r[t] = make_float2(__uint_as_float(a.x), __uint_as_float(a.y));
      } else {
        const uint32_t u = ld_ordered_stream_u32(at);
        if (DTYPE == HQ_DTYPE_BF16) {
          r[t] = make_float2(__uint_as_float(u << 16), __uint_as_float(u & 0xffff0000u));
        } else {
          r[t] = __half22float2(u32_as_half2(u));
        }
      }
    }
  }
  const float fgs = (float)gs;
  const bool pow2 = (gs & (gs - 1)) == 0;  // then the product by 1 / gs is the same quotient
  const float inv_gs = 1.f / fgs;
  int parity = 0;
  // half(mean over the group), from what every thread holds as its run's partial sums
  auto group_mean = [&](float2 part) -> __half2 {
    s_part[parity][run][lane] = part;
    __syncthreads();
    float2 s = make_float2(0.f, 0.f);
#pragma unroll
    for (int w = 0; w < runs; w++) {
      const float2 p = s_part[parity][w][lane];
      s.x += p.x;
      s.y += p.y;
    }
    parity ^= 1;  // the next exchange uses the other half: no second barrier
    return pow2 ? __floats2half2_rn(s.x * inv_gs, s.y * inv_gs)
                : __floats2half2_rn(s.x / fgs, s.y / fgs);
  };
  // 0 - bias, +0 for a zero bias: the sums below then never leave a residual of -0,
  // so its sign bit alone says whether it is >= 0
  float2 nbias = make_float2(0.f, 0.f);
  if (q_bias != nullptr) {
    float2 part = make_float2(0.f, 0.f);
#pragma unroll
    for (int t = 0; t < 32; t++) {
      part.x += r[t].x;
      part.y += r[t].y;
    }
    const __half2 bh = group_mean(part);
    const float2 bias = __half22float2(bh);
    nbias = make_float2(0.f - bias.x, 0.f - bias.y);
    if (live && run == 0 &&
        HQ_IN_BOUNDS(q_bias + (size_t)g * M + m, 4, q_bias, (size_t)(K / gs) * M * 2, 1003))
      *reinterpret_cast<__half2*>(q_bias + (size_t)g * M + m) = bh;
  }
  // One pass per plane over the registers: the residual's sign bits go into the
  // words (most recent input lowest, reversed at the end), its magnitudes into the
  // partial sums; the update before it adds -alpha with the residual's sign on it.
  uint32_t w0 = 0, w1 = 0;
  float p0 = 0.f, p1 = 0.f;
  auto take = [&](float2 f) {
    p0 += fabsf(f.x);
    p1 += fabsf(f.y);
    w0 = __funnelshift_l(__float_as_uint(f.x), w0, 1);
    w1 = __funnelshift_l(__float_as_uint(f.y), w1, 1);
  };
#pragma unroll
  for (int t = 0; t < 32; t++) {
    r[t].x += nbias.x;
    r[t].y += nbias.y;
    take(r[t]);
  }
  __half* al = alpha + (size_t)g * nb * M + m;
  uint32_t* words = bW + (size_t)(k0 >> 5) * nb * M + m;
  for (int b = 0; b < nb; b++, al += M, words += M) {
    const __half2 ah = group_mean(make_float2(p0, p1));
    const float2 a = __half22float2(ah);
    const bool finite = a.x <= 65504.f && a.y <= 65504.f;
    if (!finite) {
      // overflowed or NaN scales: by comparison, where a NaN counts as negative
      w0 = w1 = 0xffffffffu;
#pragma unroll
      for (int t = 0; t < 32; t++) {
        const float2 f = r[t];
        w0 &= ~((f.x >= 0.f ? 0x80000000u : 0u) >> t);
        w1 &= ~((f.y >= 0.f ? 0x80000000u : 0u) >> t);
      }
    }
    if (live) {
      if (run == 0 && HQ_IN_BOUNDS(al, 4, alpha, (size_t)(K / gs) * nb * M * 2, 1004))
        *reinterpret_cast<__half2*>(al) = ah;
      if (HQ_IN_BOUNDS(words, 8, bW, (size_t)(K / 32) * nb * M * 4, 1005))
        *reinterpret_cast<uint2*>(words) = make_uint2(__brev(~w0), __brev(~w1));
    }
    if (b + 1 == nb) break;
    w0 = w1 = 0;
    p0 = p1 = 0.f;
    if (finite) {
      const uint32_t na0 = __float_as_uint(-a.x), na1 = __float_as_uint(-a.y);
#pragma unroll
      for (int t = 0; t < 32; t++) {
        r[t].x += __uint_as_float((__float_as_uint(r[t].x) & 0x80000000u) ^ na0);
        r[t].y += __uint_as_float((__float_as_uint(r[t].y) & 0x80000000u) ^ na1);
        take(r[t]);
      }
    } else {
#pragma unroll
      for (int t = 0; t < 32; t++) {
        const float2 f = r[t];
        r[t] = make_float2(f.x - (f.x >= 0.f ? a.x : -a.x), f.y - (f.y >= 0.f ? a.y : -a.y));
        take(r[t]);
      }
    }
  }
}

template <int DTYPE>
int run(const void* W, int K, int M, int nb, int gs, uint32_t* bW, void* alpha, void* q_bias,
        cudaStream_t st) {
  if (gs / 32 > kMaxRuns) return HQ_ERR_UNSUPPORTED;
  const dim3 grid((M + kColsPerCta - 1) / kColsPerCta, K / gs);
  __half* al = reinterpret_cast<__half*>(alpha);
  __half* qb = reinterpret_cast<__half*>(q_bias);
  // The early start from one CTA per SM on: the CTAs of a smaller grid would not be spread over
  // all SMs (1024 x 1024, 128 CTAs: 4.1 us, 4.8 with it; 4096 x 4096: 15.6 -> 13.7).
  const bool early = (long long)grid.x * grid.y >= sm_count();
  auto go = [&](auto kern) {
    if (early) return cuda_status(launch_pdl(kern, grid, dim3(gs), 0, st, W, K, M, nb, gs, bW, al, qb));
    kern<<<grid, gs, 0, st>>>(W, K, M, nb, gs, bW, al, qb);
    return launch_status();
  };
  if (DTYPE == HQ_DTYPE_F32 && !row_fits_32(M, 4))
    return go(bcq_quantize_kernel<HQ_DTYPE_F32, 0, unsigned long long>);
  // the usual group: its exchange is unrolled
  return gs == 128 ? go(bcq_quantize_kernel<DTYPE, 4, uint32_t>) : go(bcq_quantize_kernel<DTYPE, 0, uint32_t>);
}

}  // namespace
}  // namespace hq

extern "C" int hq_lutgemm_quantize(const void* W, int dtype, int K, int M, int nb, int group_size,
                                   uint32_t* bW, void* alpha_half, void* q_bias_half,
                                   hq_stream_t stream) {
  using namespace hq;
  if (K <= 0 || M <= 0 || nb < 1 || nb > 8 || group_size < 32 || group_size % 32 != 0 ||
      K % group_size != 0 || M % 8 != 0)
    return HQ_ERR_BAD_SHAPE;
  if (K / group_size > 65535) return HQ_ERR_TOO_LARGE;
  if (!W || !bW || !alpha_half) return HQ_ERR_NULL_POINTER;
  if (!aligned16(W) || !aligned16(bW) || !aligned4(alpha_half) ||
      (q_bias_half && !aligned4(q_bias_half)))
    return HQ_ERR_MISALIGNED;
  cudaStream_t st = (cudaStream_t)stream;
  switch (dtype) {
    case HQ_DTYPE_F16: return run<HQ_DTYPE_F16>(W, K, M, nb, group_size, bW, alpha_half, q_bias_half, st);
    case HQ_DTYPE_BF16: return run<HQ_DTYPE_BF16>(W, K, M, nb, group_size, bW, alpha_half, q_bias_half, st);
    case HQ_DTYPE_F32: return run<HQ_DTYPE_F32>(W, K, M, nb, group_size, bW, alpha_half, q_bias_half, st);
    default: return HQ_ERR_UNSUPPORTED;
  }
}
