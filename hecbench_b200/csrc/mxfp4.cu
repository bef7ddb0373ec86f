// MXFP4 (OCP microscaling: 32 elements share one power-of-two scale, each
// element is a 4-bit e2m1 float) for sm_100a: quantize-dequantize in place of
// the reference kernel, plus the packer and the unpacker that the simulation
// stands for.
//
// Reference semantics (mxfp4-cuda/main.cu:112-150, qdq_mxfp4_kernel; constants
// common.h:12-34), per group of 32 consecutive elements of an fp16 or bf16 tensor:
//   m  = max |x|, its mantissa rounded to a power of two: bits + (quarter of the
//        mantissa range), mantissa cleared - so 1.75 * 2^e and above become 2^(e+1)
//   k  = clamp(floor(log2 m) - 2, -127, 127)      (e2m1's largest binade is 2^2)
//   q  = x / 2^k rounded to the e2m1 grid {0, .5, 1, 1.5, 2, 3, 4, 6}, ties to the
//        even mantissa (main.cu:21-109: .25 -> 0, .75 -> 1, 1.25 -> 1, 1.75 -> 2,
//        2.5 -> 2, 3.5 -> 4, 5 -> 4), magnitudes above 6 saturate, sign kept
//   y  = q * 2^k
// The reference computes in the input type.  Every step is a scaling by a power
// of two or a rounding to a grid coarser than the input's, so the same values
// come out of fp32 arithmetic, which is what the kernels below use; fp32 also
// makes the extension to what the reference leaves undefined harmless: a group
// whose maximum rounds to a zero exponent field (zero, small denormals: the
// reference takes log2 of 0 and overflows an int) here gets the smallest scale
// the reference's expression can produce, and a zero group gives zeros.
// NaN and infinity are not treated specially in either.
//
// Packed form (hq_mxfp4_quantize / hq_mxfp4_dequantize): one byte per two
// elements, element 2j in the LOW nibble, nibble = sign << 3 | index into the
// grid above; one E8M0 byte (k + 127) per group.
//
// Design.  HBM-bound streaming kernels (4 bytes per element for the
// quantize-dequantize, 2.53 for the packer and the unpacker).  A thread owns one
// group: 64 bytes in two 256-bit loads, so the group maximum needs no shuffle
// (SIMD maxima of the magnitudes), the codes leave as one 16-byte store and the
// scales of a warp as 32 adjacent bytes.  Rounding to the grid is the hardware's
// e2m1 conversion (round to nearest even, saturating at 6, sign kept: the rule
// above) of x * 2^-k in fp32, decoding the conversion back to fp16 pairs and one
// exact product by 2^k.  Warp instructions per 32 values: 4.9 packing (14.1 with binade
// compares, magic additions and index arithmetic), 4.6 unpacking, 6.3 for the
// quantize-dequantize (16.9).  Packing and unpacking 32 Mi bf16 values took 69.6 us and
// took 31.6 after that; 64 Mi fp16 packed 37.7 -> 26.1, quantized and dequantized 54.5 -> 41.5.
// The kernels may become resident while the launch before them drains: packed and
// unpacked, of a pair of calls among others, 32 Mi bf16 values 29.9 -> 26.4 us, 64 Mi fp16
// 55.8 -> 52.4, 1 Mi 8.2 -> 4.4.
// Groups that hold an
// infinity or a NaN, and scales whose power of two is no number of the type, go
// through plain fp32 arithmetic.
#include <cuda_bf16.h>

#include "hq_common.cuh"

namespace hq {
namespace {

constexpr int kThreads = 256;

template <bool BF16>
__device__ __forceinline__ float2 to_float2(uint32_t w) {
  if (BF16) return make_float2(__uint_as_float(w << 16), __uint_as_float(w & 0xffff0000u));
  return __half22float2(u32_as_half2(w));
}
template <bool BF16>
__device__ __forceinline__ uint32_t from_float2(float a, float b) {
  if (BF16) {
    const __nv_bfloat162 h = __floats2bfloat162_rn(a, b);
    return *reinterpret_cast<const uint32_t*>(&h);
  }
  return half2_as_u32(__floats2half2_rn(a, b));
}

// exponent k of the group's scale from the largest magnitude (16 bits of T, sign
// clear): a quarter of the mantissa range added, the exponent field kept; a field
// of 0 (zero or small denormal maximum: undefined in the reference) counts as 1
template <bool BF16>
__device__ __forceinline__ int scale_exponent(uint32_t max_bits) {
  constexpr int M = BF16 ? 7 : 10, B = BF16 ? 127 : 15;
  const int field = max((int)((max_bits + (1u << (M - 2))) >> M), 1);
  return max(-127, min(field - B - 2, 127));
}
// 2^k for k in [-127, 127] (2^-127 is an fp32 denormal)
__device__ __forceinline__ float pow2i(int k) {
  return k > -127 ? __uint_as_float((uint32_t)(k + 127) << 23) : __uint_as_float(0x00400000u);
}

// |v| scaled into the e2m1 range -> the grid value, ties to even, saturating at 6
__device__ __forceinline__ float to_grid(float a) {
  // grid step .5 below 2, 1 below 4, 2 above: adding 1.5 * 2^(23 + log2 step) and
  // taking it away again rounds to that step, ties to even
  const float c = a < 2.f ? 6291456.f : (a < 4.f ? 12582912.f : 25165824.f);
  return fminf((a + c) - c, 6.f);
}
// grid value -> index 0..7 into {0, .5, 1, 1.5, 2, 3, 4, 6}: from 1 on the index
// is (exponent - 126) * 2 + mantissa bit = the fp32 pattern >> 22, less 252; .5 is
// e2m1's one denormal (index 1) and 0 is 0
__device__ __forceinline__ uint32_t grid_index(float q) {
  const uint32_t b = __float_as_uint(q);
  return (uint32_t)max((int)(b >> 22) - 252, (int)min(b, 1u));
}

// 8 values times inv -> four bytes of codes, by the hardware conversion: byte j holds
// element 2j in the low nibble
template <bool BF16>
__device__ __forceinline__ uint32_t encode8(const uint32_t* w, float inv) {
  float2 f[4];
#pragma unroll
  for (int j = 0; j < 4; j++) {
    f[j] = to_float2<BF16>(w[j]);
    f[j].x *= inv;
    f[j].y *= inv;
  }
  uint32_t r;
  asm("{\n .reg .b8 b0, b1, b2, b3;\n"
      " cvt.rn.satfinite.e2m1x2.f32 b0, %2, %1;\n"
      " cvt.rn.satfinite.e2m1x2.f32 b1, %4, %3;\n"
      " cvt.rn.satfinite.e2m1x2.f32 b2, %6, %5;\n"
      " cvt.rn.satfinite.e2m1x2.f32 b3, %8, %7;\n"
      " mov.b32 %0, {b0, b1, b2, b3};\n}"
      : "=r"(r)
      : "f"(f[0].x), "f"(f[0].y), "f"(f[1].x), "f"(f[1].y), "f"(f[2].x), "f"(f[2].y), "f"(f[3].x),
        "f"(f[3].y));
  return r;
}
// the same by plain arithmetic (infinities and NaN count as 6); the values of a
// quantize-dequantize take their signs after the conversion to fp32, which drops a NaN's
template <bool BF16, bool VALUES>
__device__ uint32_t encode8_plain(const uint32_t* w, float inv) {
  uint32_t r = 0;
  for (int j = 0; j < 4; j++) {
    const float2 f = to_float2<BF16>(w[j]);
    const uint32_t s0 = (VALUES ? __float_as_uint(f.x) >> 28 : w[j] >> 12) & 8u;  // the sign bits
    const uint32_t s1 = (VALUES ? __float_as_uint(f.y) : w[j]) >> 28 & 8u;
    const uint32_t i0 = grid_index(to_grid(fabsf(f.x) * inv)), i1 = grid_index(to_grid(fabsf(f.y) * inv));
    r |= ((i0 | s0) | ((i1 | s1) << 4)) << (8 * j);
  }
  return r;
}

// four bytes of codes -> 8 values of T, times 2^k
template <bool BF16>
__device__ __forceinline__ void decode8(uint32_t c, int k, uint32_t* o) {
  uint32_t h[4];  // fp16 pairs of grid values
  asm("{\n .reg .b8 b0, b1, b2, b3;\n mov.b32 {b0, b1, b2, b3}, %4;\n"
      " cvt.rn.f16x2.e2m1x2 %0, b0;\n cvt.rn.f16x2.e2m1x2 %1, b1;\n"
      " cvt.rn.f16x2.e2m1x2 %2, b2;\n cvt.rn.f16x2.e2m1x2 %3, b3;\n}"
      : "=r"(h[0]), "=r"(h[1]), "=r"(h[2]), "=r"(h[3])
      : "r"(c));
  if (BF16 && k <= 15) {
    // the fp16 pattern moved three bits down is the bf16 pattern of value * 2^-112
    // (15 - 127), zero included; one product by 2^(k + 112) restores both
    const uint32_t sb = (uint32_t)(k + 112 + 127) << 7, s2 = sb | (sb << 16);
#pragma unroll
    for (int j = 0; j < 4; j++) {
      const uint32_t b = ((h[j] >> 3) & 0x0fff0fffu) | (h[j] & 0x80008000u);
      const __nv_bfloat162 v = __hmul2(*reinterpret_cast<const __nv_bfloat162*>(&b),
                                       *reinterpret_cast<const __nv_bfloat162*>(&s2));
      o[j] = *reinterpret_cast<const uint32_t*>(&v);
    }
  } else if (!BF16 && k >= -24 && k <= 15) {
    const __half2 s2 = __float2half2_rn(pow2i(k));  // a number of the type, denormal below -14
#pragma unroll
    for (int j = 0; j < 4; j++) o[j] = half2_as_u32(__hmul2(u32_as_half2(h[j]), s2));
  } else {
    const float scale = k > 127 ? __uint_as_float(0x7f800000u) : pow2i(k);
#pragma unroll
    for (int j = 0; j < 4; j++) {
      const float2 f = __half22float2(u32_as_half2(h[j]));
      o[j] = from_float2<BF16>(f.x * scale, f.y * scale);
    }
  }
}

// the 64 bytes of a group; wide: the address is 32-byte aligned
__device__ __forceinline__ void load_group(uint32_t (&w)[16], const char* p, bool wide) {
  if (wide) {
#pragma unroll
    for (int h = 0; h < 2; h++)
      asm volatile("ld.global.L1::no_allocate.v8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
                   : "=r"(w[8 * h]), "=r"(w[8 * h + 1]), "=r"(w[8 * h + 2]), "=r"(w[8 * h + 3]),
                     "=r"(w[8 * h + 4]), "=r"(w[8 * h + 5]), "=r"(w[8 * h + 6]), "=r"(w[8 * h + 7])
                   : "l"(p + 32 * h));
  } else {
#pragma unroll
    for (int h = 0; h < 4; h++) {
      const uint4 v = ld_ordered_stream_u4(p + 16 * h);
      w[4 * h] = v.x, w[4 * h + 1] = v.y, w[4 * h + 2] = v.z, w[4 * h + 3] = v.w;
    }
  }
}
__device__ __forceinline__ void store_group(const uint32_t (&w)[16], char* p, bool wide) {
  if (wide) {
#pragma unroll
    for (int h = 0; h < 2; h++)
      asm volatile("st.global.v8.b32 [%8], {%0,%1,%2,%3,%4,%5,%6,%7};" ::"r"(w[8 * h]),
                   "r"(w[8 * h + 1]), "r"(w[8 * h + 2]), "r"(w[8 * h + 3]), "r"(w[8 * h + 4]),
                   "r"(w[8 * h + 5]), "r"(w[8 * h + 6]), "r"(w[8 * h + 7]), "l"(p + 32 * h)
                   : "memory");
  } else {
#pragma unroll
    for (int h = 0; h < 4; h++)
      *reinterpret_cast<uint4*>(p + 16 * h) = make_uint4(w[4 * h], w[4 * h + 1], w[4 * h + 2], w[4 * h + 3]);
  }
}

// MODE 0: out = quantize-dequantize of in (type T); MODE 1: codes + scales
template <bool BF16, int MODE>
__global__ void __launch_bounds__(kThreads)
mxfp4_kernel(const char* in, char* __restrict__ out, uint32_t* __restrict__ codes,
             uint8_t* __restrict__ scales, size_t groups, bool wide, bool wide_codes) {
  pdl_launch_dependents();
  pdl_wait();  // nothing is read or written before every earlier kernel has completed
  const size_t g = (size_t)blockIdx.x * kThreads + threadIdx.x;
  if (g >= groups || !HQ_IN_BOUNDS(in + g * 64, 64, in, groups * 64, 601)) return;
  uint32_t w[16];
  load_group(w, in + g * 64, wide);
  uint32_t m = 0;
#pragma unroll
  for (int j = 0; j < 16; j++) m = __vmaxu2(m, w[j] & 0x7fff7fffu);
  const uint32_t mx = max(m & 0xffffu, m >> 16);
  const int k = scale_exponent<BF16>(mx);
  const float inv = pow2i(-k);
  uint32_t c[4];
  if (mx < (BF16 ? 0x7f80u : 0x7c00u)) {
#pragma unroll
    for (int j = 0; j < 4; j++) c[j] = encode8<BF16>(w + 4 * j, inv);
  } else {
#pragma unroll
    for (int j = 0; j < 4; j++) c[j] = encode8_plain<BF16, MODE == 0>(w + 4 * j, inv);
  }
  if (MODE == 0) {
#pragma unroll
    for (int j = 0; j < 4; j++) decode8<BF16>(c[j], k, w + 4 * j);
    if (HQ_IN_BOUNDS(out + g * 64, 64, out, groups * 64, 602)) store_group(w, out + g * 64, wide);
  } else {
    if (!HQ_IN_BOUNDS(codes + 4 * g, 16, codes, groups * 16, 603) ||
        !HQ_IN_BOUNDS(scales + g, 1, scales, groups, 604))
      return;
    if (wide_codes) {
      *reinterpret_cast<uint4*>(codes + 4 * g) = make_uint4(c[0], c[1], c[2], c[3]);
    } else {
#pragma unroll
      for (int j = 0; j < 4; j++) codes[4 * g + j] = c[j];
    }
    scales[g] = (uint8_t)(k + 127);
  }
}

// codes + scales -> T
template <bool BF16>
__global__ void __launch_bounds__(kThreads)
mxfp4_dequant_kernel(const uint32_t* codes, const uint8_t* scales, char* __restrict__ out,
                     size_t groups, bool wide, bool wide_codes) {
  pdl_launch_dependents();
  pdl_wait();  // nothing is read or written before every earlier kernel has completed
  const size_t g = (size_t)blockIdx.x * kThreads + threadIdx.x;
  if (g >= groups || !HQ_IN_BOUNDS(codes + 4 * g, 16, codes, groups * 16, 605) ||
      !HQ_IN_BOUNDS(scales + g, 1, scales, groups, 606))
    return;
  uint32_t c[4];
  if (wide_codes) {
    const uint4 v = ld_ordered_stream_u4(codes + 4 * g);
    c[0] = v.x, c[1] = v.y, c[2] = v.z, c[3] = v.w;
  } else {
#pragma unroll
    for (int j = 0; j < 4; j++) c[j] = ld_ordered_stream_u32(codes + 4 * g + j);
  }
  const int k = (int)ld_ordered_u8(scales + g) - 127;
  uint32_t w[16];
#pragma unroll
  for (int j = 0; j < 4; j++) decode8<BF16>(c[j], k, w + 4 * j);
  if (HQ_IN_BOUNDS(out + g * 64, 64, out, groups * 64, 607)) store_group(w, out + g * 64, wide);
}

bool aligned32(const void* p) { return (reinterpret_cast<uintptr_t>(p) & 31u) == 0; }

unsigned grid_for(size_t groups) { return (unsigned)((groups + kThreads - 1) / kThreads); }

int check_args(const void* a, const void* b, size_t numel, int dtype) {
  if (dtype != HQ_DTYPE_F16 && dtype != HQ_DTYPE_BF16) return HQ_ERR_UNSUPPORTED;
  if (numel % 32 != 0) return HQ_ERR_BAD_SHAPE;
  if (numel && (!a || !b)) return HQ_ERR_NULL_POINTER;
  return HQ_OK;
}

}  // namespace
}  // namespace hq

extern "C" {

int hq_mxfp4_qdq(const void* in, void* out, size_t numel, int dtype, hq_stream_t stream) {
  using namespace hq;
  const int rc = check_args(in, out, numel, dtype);
  if (rc != HQ_OK || numel == 0) return rc;
  if (!aligned16(in) || !aligned16(out)) return HQ_ERR_MISALIGNED;
  const size_t groups = numel / 32;
  const auto kern = dtype == HQ_DTYPE_BF16 ? mxfp4_kernel<true, 0> : mxfp4_kernel<false, 0>;
  return cuda_status(launch_pdl(kern, dim3(grid_for(groups)), dim3(kThreads), 0, (cudaStream_t)stream,
                                (const char*)in, (char*)out, nullptr, nullptr, groups,
                                aligned32(in) && aligned32(out), false));
}

int hq_mxfp4_quantize(const void* in, uint8_t* codes, uint8_t* scales_e8m0, size_t numel, int dtype,
                      hq_stream_t stream) {
  using namespace hq;
  const int rc = check_args(in, codes, numel, dtype);
  if (rc != HQ_OK || numel == 0) return rc;
  if (!scales_e8m0) return HQ_ERR_NULL_POINTER;
  if (!aligned16(in) || !aligned4(codes)) return HQ_ERR_MISALIGNED;
  const size_t groups = numel / 32;
  const auto kern = dtype == HQ_DTYPE_BF16 ? mxfp4_kernel<true, 1> : mxfp4_kernel<false, 1>;
  return cuda_status(launch_pdl(kern, dim3(grid_for(groups)), dim3(kThreads), 0, (cudaStream_t)stream,
                                (const char*)in, nullptr, reinterpret_cast<uint32_t*>(codes), scales_e8m0,
                                groups, aligned32(in), aligned16(codes)));
}

int hq_mxfp4_dequantize(const uint8_t* codes, const uint8_t* scales_e8m0, void* out, size_t numel,
                        int dtype, hq_stream_t stream) {
  using namespace hq;
  const int rc = check_args(codes, out, numel, dtype);
  if (rc != HQ_OK || numel == 0) return rc;
  if (!scales_e8m0) return HQ_ERR_NULL_POINTER;
  if (!aligned4(codes) || !aligned16(out)) return HQ_ERR_MISALIGNED;
  const size_t groups = numel / 32;
  const auto kern = dtype == HQ_DTYPE_BF16 ? mxfp4_dequant_kernel<true> : mxfp4_dequant_kernel<false>;
  return cuda_status(launch_pdl(kern, dim3(grid_for(groups)), dim3(kThreads), 0, (cudaStream_t)stream,
                                reinterpret_cast<const uint32_t*>(codes), scales_e8m0, (char*)out, groups,
                                aligned32(out), aligned16(codes)));
}

}  // extern "C"
