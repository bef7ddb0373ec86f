// Uniformly quantized weight-only mat-vec (gemv-cuda) for sm_100a: fp16, int8
// and packed int4 weights with ONE scale and zero point per tensor.
//
// Reference semantics (gemv-cuda/kernels.h:64-123 fp16, :127-200 int8, :205-307
// int4; launchers gemv.cu:15-81): mat is row-major [rows][n] (int4: n/2 bytes
// per row, element 2j in the LOW nibble of byte j, 2j+1 in the high nibble);
// scale and zero point are rounded to fp16 by the launcher and used as fp32;
//   res[row] = half( scale * sum_j float(vec[j]) * (float(w[row][j]) - zero_point) )
// with fp32 accumulation.  Here the affine part is factored,
//   scale * ( sum_j w*x  -  zero_point * sum_j x ),
// the products are exact (fp16 on the matrix pipe) and summed in fp32.
//
// Design.  HBM-bound (2, 1 or 0.5 bytes per weight).  Two 512-thread CTAs per
// SM; the input vector is staged once per CTA in shared memory (fp16) and its
// sum reduced there; a warp owns whole rows, two adjacent ones at a time (a
// piece of the input vector read from shared memory then serves both), which it streams
// through a ring in shared memory or into registers (gemv_rows.cuh).
//  * int8 -> fp16: one XOR flips the sign bits of four bytes (b + 128), a byte
//    permute places two of them under the exponent byte 0x64 (1024 + b + 128,
//    exact), one half2 subtract of 1152 leaves the integers: 5 instructions per 4 weights.
//  * int4: codes masked in place are fp16 numbers below the normal range: 5 instructions per 8
//    weights, no table.  The inputs are staged in the
//    matching order (x0, x4)(x1, x5)(x2, x6)(x3, x7).
#include <algorithm>

#include "gemv_rows.cuh"

namespace hq {
namespace {

using namespace rows;

// n: inputs per row; row_bytes = n * BITS / 8 (a multiple of 16).  DEALT: the division of the rows; 8 bits take
// it from per_warp and per_cta (gemv_rows.cuh).
template <int BITS, bool DEALT, bool RING>
__global__ void __launch_bounds__(kThreads, 2)
gemv_uniform_kernel(const unsigned char* mat, const __half* vec,
                    __half* __restrict__ res, int rows, int n, float scale, float zero_point, int per_warp,
                    int per_cta) {
  extern __shared__ __align__(16) unsigned char dsm_raw[];  // [ring] inputs
  __shared__ float s_part[kWarps];
  __half* xs = reinterpret_cast<__half*>(dsm_raw + (RING ? kRing : 0));
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const size_t row_bytes = (size_t)n * BITS / 8;

  // Programmatic dependent launch: the next kernel of the stream may become
  // resident while this grid drains; nothing is read before the wait (the matrix
  // may be an earlier kernel's output like the input vector), and nothing is
  // written before it.
  pdl_launch_dependents();
  if (BITS == 4) prefetch_first_rows<DEALT>(mat, rows, row_bytes, lane, warp);
  pdl_wait();
  const long long first = BITS == 8 ? (warp * per_warp + (int)blockIdx.x * per_cta) * kRows : first_row<DEALT>(warp);
  PairStream<BITS, RING> stream(mat, first, (int)gridDim.x * kWarps * kRows, rows, n,
                                dsm_raw + warp * (kDepth * kSlot), lane, 402);
  // ---- prologue: inputs to shared memory and their sum ----
  const Inputs<BITS, RING> inputs = {vec, xs, n, tid, 401};
  inputs.ask();
  stream.begin();
  inputs.arrived();
  float part = 0.f;
  for (int i = tid; i < n / 8; i += kThreads) inputs.out(i, inputs.in(i), part);
  part = warp_sum(part);
  if (lane == 0) s_part[warp] = part;
  __syncthreads();
  float sumx = 0.f;
#pragma unroll
  for (int w = 0; w < kWarps; w++) sumx += s_part[w];

  // ---- rows of this warp: kRows adjacent rows at a time, so that a piece of the
  // input vector read from shared memory serves kRows rows ----
  stream.run_rows(xs, [&](uint32_t row0, float total) {
    const uint32_t row = row0 + (lane >> 2);
    if ((lane == 0 || (lane == 4 && row < (uint32_t)rows)) && HQ_IN_BOUNDS(res + row, 2, res, (size_t)rows * 2, 403))
      res[row] = __float2half_rn(BITS == 16 ? total : scale * (total - zero_point * sumx));
  });
}

template <int BITS>
int launch(const void* mat, const void* vec_half, void* res_half, int rows, int n, float scale,
           float zero_point, hq_stream_t stream) {
  if (!mat || !vec_half || !res_half) return HQ_ERR_NULL_POINTER;
  // a row is a whole number of 16-byte chunks and the inputs a whole number of
  // 16-byte groups: n a multiple of 8 (fp16), 16 (int8), 32 (int4)
  if (rows <= 0 || n <= 0 || n % (128 / BITS) != 0) return HQ_ERR_BAD_SHAPE;
  if (!aligned16(mat) || !aligned16(vec_half)) return HQ_ERR_MISALIGNED;
  if ((size_t)n * 2 > 226 * 1024) return HQ_ERR_TOO_LARGE;  // beyond 113 KiB only one CTA fits an SM
  Share share = share_rows(rows, (size_t)n * BITS / 8, BITS, true);
  const bool ring = takes_ring(rows, input_steps<BITS>(n), BITS, input_bytes<BITS>(n), true, &share);
  const int grid = share.ctas;
  const size_t smem = smem_request((ring ? kRing : 0) + input_bytes<BITS>(n), grid);
  // the launcher of the reference rounds both parameters to fp16 (gemv.cu:21-22)
  const float s = __half2float(__float2half_rn(scale));
  const float z = __half2float(__float2half_rn(zero_point));
  auto go = [&](auto dealt, auto by_ring) {
    constexpr auto kern = gemv_uniform_kernel<BITS, decltype(dealt)::value, decltype(by_ring)::value>;
    const cudaError_t e = ensure_dynamic_smem<kern>(smem);
    if (e != cudaSuccess) return cuda_status(e);
    return cuda_status(launch_pdl(kern, dim3(grid), dim3(kThreads), smem, (cudaStream_t)stream,
                                  reinterpret_cast<const unsigned char*>(mat),
                                  reinterpret_cast<const __half*>(vec_half),
                                  reinterpret_cast<__half*>(res_half), rows, n, s, z, share.dealt ? grid : 1,
                                  share.dealt ? 1 : kWarps));
  };
  auto by_ring = [&](auto dealt) { return ring ? go(dealt, std::true_type()) : go(dealt, std::false_type()); };
  return share.dealt && BITS != 8 ? by_ring(std::bool_constant<BITS != 8>()) : by_ring(std::false_type());
}

}  // namespace
}  // namespace hq

extern "C" {

int hq_gemv_f16(const void* mat_half, const void* vec_half, void* res_half, int rows, int n,
                hq_stream_t stream) {
  return hq::launch<16>(mat_half, vec_half, res_half, rows, n, 1.f, 0.f, stream);
}

int hq_gemv_int8_f16(const int8_t* mat, const void* vec_half, void* res_half, int rows, int n,
                     float scale, float zero_point, hq_stream_t stream) {
  return hq::launch<8>(mat, vec_half, res_half, rows, n, scale, zero_point, stream);
}

int hq_gemv_int4_f16(const uint8_t* mat, const void* vec_half, void* res_half, int rows, int n,
                     float scale, float zero_point, hq_stream_t stream) {
  return hq::launch<4>(mat, vec_half, res_half, rows, n, scale, zero_point, stream);
}

}  // extern "C"
