// Decode-time MLP entry fused around the weight-only mat-vec, for sm_100a:
//   RMSNorm of the input vector  ->  mat-vec  ->  gated activation of row pairs
// in ONE kernel, for fp16 and uniform int8 / int4 weights (the NF4 form is a
// variant of the NF4 mat-vec kernel itself, nf4.cu).  At batch 1 the
// normalised vector (K halves) and the two projections (2 x N halves) otherwise
// make two round trips through memory and cost two more launches, each as long
// as the mat-vec of a small layer.
//
// Semantics (the host references of the stand-alone benchmarks):
//  * RMSNorm (rmsnorm-cuda/reference.h:4-25): xn[k] = x[k] * rsqrt(mean(x^2) +
//    eps) * gamma[k]; skipped when gamma is null.  Computed in fp32, rounded to
//    fp16 once.
//  * mat-vec: as hq_gemv_f16 / hq_gemv_int8_f16 / hq_gemv_int4_f16 (same
//    layouts, same scale / zero point rules), exact products, fp32 sums.
//  * gated activation: with act != 0 the matrix has 2 * rows_out rows, row 2m the
//    value row and row 2m + 1 the gate row of output m (the x / gate order of
//    geglu-cuda/reference.h:8-16, per output feature), and
//      out[m] = v * g / (1 + exp(-g))                (HQ_ACT_SWIGLU; swish-cuda/reference.h:4)
//      out[m] = v * 0.5 * g * (1 + erf(g / sqrt 2))  (HQ_ACT_GEGLU;  geglu-cuda/reference.h:1-5)
//    in fp32, rounded to fp16 once.  With act == 0 the kernel is the plain
//    mat-vec (plus the RMSNorm) and writes rows_out results.
//
// Design: the row-streaming form of gemv_uniform.cu (gemv_rows.cuh; two 512-thread CTAs per SM,
// a warp owns a PAIR of adjacent rows - here exactly a value / gate pair -, the
// input vector in shared memory).  The prologue reads the input vector there twice (sum of
// squares, then scale and round).
#include <algorithm>

#include "gemv_rows.cuh"

namespace hq {
namespace {

using namespace rows;

struct FusedParams {
  const unsigned char* mat;
  const __half* x;
  const __half* gamma;   // null: no RMSNorm
  __half* out;
  float eps, scale, zero_point;
  int rows_out, n, act;
};

// sum over the CTA (all threads get the result); buf holds kWarps floats and is used once
__device__ __forceinline__ float block_sum(float v, float* buf, int lane, int warp) {
  v = warp_sum(v);
  if (lane == 0) buf[warp] = v;
  __syncthreads();
  float t = 0.f;
#pragma unroll
  for (int w = 0; w < kWarps; w++) t += buf[w];
  return t;
}

template <int BITS, bool DEALT, bool RING>
__global__ void __launch_bounds__(kThreads, 2)
gemv_fused_kernel(const FusedParams p) {
  extern __shared__ __align__(16) unsigned char dsm_raw[];  // [ring] inputs
  __shared__ float s_squares[kWarps], s_part[kWarps];
  __half* xs = reinterpret_cast<__half*>(dsm_raw + (RING ? kRing : 0));
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int n = p.n;
  const size_t row_bytes = (size_t)n * BITS / 8;
  const int rows_mat = p.act ? 2 * p.rows_out : p.rows_out;

  // Programmatic dependent launch: nothing that earlier work of the stream may
  // have produced is read, and nothing is written, before the wait.
  pdl_launch_dependents();
  if (BITS == 4) prefetch_first_rows<DEALT>(p.mat, rows_mat, row_bytes, lane, warp);
  pdl_wait();
  PairStream<BITS, RING> stream(p.mat, first_row<DEALT>(warp), (int)gridDim.x * kWarps * kRows, rows_mat, n,
                                dsm_raw + warp * (kDepth * kSlot), lane, 504);
  const Inputs<BITS, RING> inputs = {p.x, xs, n, tid, 501};
  inputs.ask();
  auto gamma = [&](int i) {
    const uint4* at = reinterpret_cast<const uint4*>(p.gamma) + i;
    return p.gamma != nullptr && i < n / 8 && HQ_IN_BOUNDS(at, 16, p.gamma, (size_t)n * 2, 503) ? ld_ordered_u4(at)
                                                                                                : make_uint4(0, 0, 0, 0);
  };
  const uint4 first_gamma = gamma(tid);
  stream.begin();
  inputs.arrived();

  // ---- RMSNorm: sum of squares over the whole vector ----
  float norm = 1.f;
  if (p.gamma != nullptr) {
    float sq = 0.f;
    for (int i = tid; i < n / 8; i += kThreads) {
      const uint4 v = inputs.in(i);
      const uint32_t h[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
      for (int k = 0; k < 4; k++) {
        const float2 f = __half22float2(u32_as_half2(h[k]));
        sq = fmaf(f.x, f.x, fmaf(f.y, f.y, sq));
      }
    }
    sq = block_sum(sq, s_squares, lane, warp);
    norm = rsqrtf(sq / (float)n + p.eps);
  }
  // ---- scale, round to fp16; sum of the inputs ----
  float part = 0.f;
  for (int i = tid; i < n / 8; i += kThreads) {
    uint4 v = inputs.in(i);
    if (p.gamma != nullptr) {
      const uint4 g = i == tid ? first_gamma : gamma(i);
      uint32_t h[4] = {v.x, v.y, v.z, v.w};
      const uint32_t gh[4] = {g.x, g.y, g.z, g.w};
#pragma unroll
      for (int k = 0; k < 4; k++) {
        const float2 f = __half22float2(u32_as_half2(h[k]));
        const float2 w = __half22float2(u32_as_half2(gh[k]));
        h[k] = half2_as_u32(__floats2half2_rn(f.x * norm * w.x, f.y * norm * w.y));
      }
      v = make_uint4(h[0], h[1], h[2], h[3]);
    }
    inputs.out(i, v, part);
  }
  const float sumx = block_sum(part, s_part, lane, warp);  // also: inputs complete

  // ---- row pairs of this warp ----
  stream.run_rows(xs, [&](uint32_t row0, float total) {
    const float v = BITS == 16 ? total : p.scale * (total - p.zero_point * sumx);
    if (p.act) {
      const float gate = __shfl_down_sync(0xffffffffu, v, 4);
      const uint32_t m = row0 >> 1;  // row0 is even: the value row; row0 + 1 the gate row
      if (lane == 0 && HQ_IN_BOUNDS(p.out + m, 2, p.out, (size_t)p.rows_out * 2, 506))
        p.out[m] = __float2half_rn(v * gate_act(gate, p.act));
    } else {
      const uint32_t row = row0 + (lane >> 2);
      if ((lane == 0 || (lane == 4 && row < (uint32_t)rows_mat)) &&
          HQ_IN_BOUNDS(p.out + row, 2, p.out, (size_t)p.rows_out * 2, 507))
        p.out[row] = __float2half_rn(v);
    }
  });
}

template <int BITS>
int launch(const FusedParams& prm, hq_stream_t stream) {
  if (!prm.mat || !prm.x || !prm.out) return HQ_ERR_NULL_POINTER;
  if (prm.rows_out <= 0 || prm.n <= 0 || prm.n % (128 / BITS) != 0) return HQ_ERR_BAD_SHAPE;
  if (prm.act != HQ_ACT_NONE && prm.act != HQ_ACT_SWIGLU && prm.act != HQ_ACT_GEGLU)
    return HQ_ERR_BAD_SHAPE;
  if (!aligned16(prm.mat) || !aligned16(prm.x) || (prm.gamma && !aligned16(prm.gamma)))
    return HQ_ERR_MISALIGNED;
  // beyond 113 KiB only one CTA fits an SM
  if ((size_t)prm.n * 2 > 226 * 1024) return HQ_ERR_TOO_LARGE;
  const int rows_mat = prm.act ? 2 * prm.rows_out : prm.rows_out;
  Share share = share_rows(rows_mat, (size_t)prm.n * BITS / 8, BITS, false);
  const bool ring = takes_ring(rows_mat, input_steps<BITS>(prm.n), BITS, input_bytes<BITS>(prm.n), false, &share);
  const int grid = share.ctas;
  const size_t smem = smem_request((ring ? kRing : 0) + input_bytes<BITS>(prm.n), grid);
  auto go = [&](auto dealt, auto by_ring) {
    constexpr auto kern = gemv_fused_kernel<BITS, decltype(dealt)::value, decltype(by_ring)::value>;
    const cudaError_t e = ensure_dynamic_smem<kern>(smem);
    if (e != cudaSuccess) return cuda_status(e);
    return cuda_status(launch_pdl(kern, dim3(grid), dim3(kThreads), smem, (cudaStream_t)stream, prm));
  };
  auto by_ring = [&](auto dealt) { return ring ? go(dealt, std::true_type()) : go(dealt, std::false_type()); };
  return share.dealt ? by_ring(std::true_type()) : by_ring(std::false_type());
}

FusedParams base_params(const void* mat, const void* x_half, const void* gamma_half, float eps,
                        void* out_half, int rows_out, int n, int act) {
  FusedParams prm = {};
  prm.mat = reinterpret_cast<const unsigned char*>(mat);
  prm.x = reinterpret_cast<const __half*>(x_half);
  prm.gamma = reinterpret_cast<const __half*>(gamma_half);
  prm.out = reinterpret_cast<__half*>(out_half);
  prm.eps = eps;
  prm.scale = 1.f;
  prm.rows_out = rows_out;
  prm.n = n;
  prm.act = act;
  return prm;
}

}  // namespace
}  // namespace hq

extern "C" {

int hq_gemv_fused_f16(const void* x_half, const void* gamma_half, float eps, const void* mat_half,
                      void* out_half, int rows_out, int n, int act, hq_stream_t stream) {
  using namespace hq;
  return launch<16>(base_params(mat_half, x_half, gamma_half, eps, out_half, rows_out, n, act),
                      stream);
}

int hq_gemv_fused_int8_f16(const void* x_half, const void* gamma_half, float eps, const int8_t* mat,
                           void* out_half, int rows_out, int n, float scale, float zero_point,
                           int act, hq_stream_t stream) {
  using namespace hq;
  FusedParams prm = base_params(mat, x_half, gamma_half, eps, out_half, rows_out, n, act);
  prm.scale = __half2float(__float2half_rn(scale));  // as the reference launchers (gemv.cu:21-22)
  prm.zero_point = __half2float(__float2half_rn(zero_point));
  return launch<8>(prm, stream);
}

int hq_gemv_fused_int4_f16(const void* x_half, const void* gamma_half, float eps,
                           const uint8_t* mat, void* out_half, int rows_out, int n, float scale,
                           float zero_point, int act, hq_stream_t stream) {
  using namespace hq;
  FusedParams prm = base_params(mat, x_half, gamma_half, eps, out_half, rows_out, n, act);
  prm.scale = __half2float(__float2half_rn(scale));
  prm.zero_point = __half2float(__float2half_rn(zero_point));
  return launch<4>(prm, stream);
}

}  // extern "C"
