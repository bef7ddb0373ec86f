// Per-token int8 activation quantization (quantVLLM) for sm_100a: the step in
// front of a W8A8 linear layer.
//
// Replaces the launchers static_scaled_int8_quant / dynamic_scaled_int8_quant
// of quantVLLM-cuda/main.cu:137-172 and their four kernels (main.cu:12-134):
//   static            out = sat8(rint(x / scale))
//   static + azp      out = sat8(sat32(rint(x / scale)) + azp)
//   dynamic           scale[t] = absmax_t / 127, out = sat8(rint(x * (127 / absmax_t)))
//   dynamic + azp     scale[t] = (max_t - min_t) / 255, azp[t] = rint(-128 - min_t / scale[t]),
//                     out = sat8(sat32(rint(x / scale[t])) + azp[t])
// for fp16, bf16 or fp32 inputs x[num_tokens][hidden_size].  Every arithmetic
// step is the reference's (IEEE division, round-half-even, the same order of
// saturations; the running maximum of the azp form starts at FLT_MIN like
// utils.h / reference.h:66), so the outputs are byte-exact.
//
// Design.  Pure streaming, 2-4 bytes in and 1 byte out per element; the bound is
// memory, the second wall instruction issue:
//  * static forms have no per-token state: the tensor is processed flat, 16
//    elements per thread and turn (16-byte loads, one 16-byte store);
//  * dynamic forms: one CTA per token row; the row is read ONCE, kept in
//    registers as it is (packed), reduced with packed maxima, warp shuffles and
//    one shared-memory exchange, and quantized from the registers - the
//    reference reads every row twice.  Rows are contiguous but start at any
//    element (the reference's own run uses hidden_size = 5137), so the CTA
//    works on the aligned 16-byte chunks that overlap its row and masks the
//    neighbours' elements: full-width loads and 8-byte stores at any row
//    offset, all loads of a row in flight together.  Block size and chunks per
//    thread follow the row length (dynamic_launch_ept).  An element-wise form
//    covers unaligned buffers and rows beyond the register cache.
//  * per element a conversion, a product, a rounding to int (saturating), half a
//    saturating pack (cvt.pack.sat.s8), half a packed maximum.  The divisions of the
//    other forms are a product by the rounded reciprocal and one fused residual
//    correction (exact_quotient).  4096 x 5137 fp16: dynamic 24.1 -> 11.7 us, 13.4 warp
//    instructions per 32 elements with addresses, masks and stores (22.0 before), issue
//    slots 75 % busy; with zero point 33.3 -> 18.4; static 18.4 -> 11.3;
//  * every kernel may become resident while the launch before it drains: of a call
//    among others the launch and the last wave of the one before cost 1.7 to 2.4 us
//    (device time per call, dynamic: 1 x 4096 fp16 4.1 -> 1.75 us, 300 x 1025 4.1 -> 2.4,
//    4096 x 5137 14.4 -> 12.7, 8192 x 16384 63.6 -> 61.7; static 2048 x 8192 bf16 12.3 ->
//    10.3; with zero point 2048 x 4096 fp32 13.7 -> 11.7).
#include <cuda_bf16.h>

#include <cfloat>
#include <type_traits>

#include "hq_common.cuh"

namespace hq {
namespace {

constexpr int kThreads = 256;
constexpr int kWarps = kThreads / 32;

template <typename T>
__device__ __forceinline__ float to_float(T v);
template <>
__device__ __forceinline__ float to_float<__half>(__half v) { return __half2float(v); }
template <>
__device__ __forceinline__ float to_float<__nv_bfloat16>(__nv_bfloat16 v) {
  return __bfloat162float(v);
}
template <>
__device__ __forceinline__ float to_float<float>(float v) { return v; }

// utils.h:9-28: nearbyint, clamp to [-128, 127], convert (NaN gives 0)
__device__ __forceinline__ int f2i8_rn(float x) {
  return max(-128, min(127, __float2int_rn(x)));  // the conversion saturates at int32 first
}
// utils.h:30-63: sat32(rint(x)) + azp (wrapping, as two's complement does), clamp
__device__ __forceinline__ int f2i8_azp(float x, int azp) {
  const int q = (int)((unsigned)__float2int_rn(x) + (unsigned)azp);
  return max(-128, min(127, q));
}

// Four int32 -> four int8 with saturation, element 0 lowest: two instructions
__device__ __forceinline__ uint32_t pack_sat8(int a, int b, int c, int d) {
  uint32_t hi, r;
  asm("cvt.pack.sat.s8.s32.b32 %0, %1, %2, %3;" : "=r"(hi) : "r"(d), "r"(c), "r"(0));
  asm("cvt.pack.sat.s8.s32.b32 %0, %1, %2, %3;" : "=r"(r) : "r"(b), "r"(a), "r"(hi));
  return r;
}

// x / s from y = 1 / s rounded to nearest: the residual of the product is exact, and
// q + residual * y rounds to the IEEE quotient (Markstein) as long as nothing over-
// or underflows on the way, which the callers see to (divides_fast and finite x; a
// NaN stays a NaN).
__device__ __forceinline__ float exact_quotient(float x, float s, float y) {
  const float q = __fmul_rn(x, y);
  return __fmaf_rn(__fmaf_rn(-q, s, x), y, q);
}
__device__ __forceinline__ bool divides_fast(float s) {
  return fabsf(s) >= 8.6736174e-19f && fabsf(s) <= 1.1529215e18f;  // 2^-60 .. 2^60
}

// 16 bytes of T as floats
template <typename T>
__device__ __forceinline__ void unpack16(const uint4& v, float (&f)[16 / sizeof(T)]) {
  const T* e = reinterpret_cast<const T*>(&v);
#pragma unroll
  for (int k = 0; k < 16 / (int)sizeof(T); k++) f[k] = to_float<T>(e[k]);
}

// ---- static forms: flat over num_tokens * hidden_size elements ----
template <typename T, bool AZP>
__global__ void __launch_bounds__(kThreads)
vllm_static_kernel(const T* in, int8_t* __restrict__ out, size_t n, float scale,
                   int azp, int vec_ok) {
  pdl_launch_dependents();
  pdl_wait();  // nothing is read or written before every earlier kernel has completed
  constexpr int kPerLoad = 16 / sizeof(T);  // elements per 16-byte load
  constexpr int kLoads = 16 / kPerLoad;     // loads per 16 outputs
  const size_t stride = (size_t)gridDim.x * kThreads;
  const size_t nvec = vec_ok ? n / 16 : 0;
  const bool fast = divides_fast(scale);
  const float inv = __frcp_rn(scale), limit = fabsf(scale) * 1073741824.f;
  for (size_t v = (size_t)blockIdx.x * kThreads + threadIdx.x; v < nvec; v += stride) {
    if (!HQ_IN_BOUNDS(reinterpret_cast<const uint4*>(in) + v * kLoads, 16 * kLoads, in,
                      n * sizeof(T), 401) ||
        !HQ_IN_BOUNDS(reinterpret_cast<uint4*>(out) + v, 16, out, n, 402))
      continue;
    uint4 raw[kLoads];
#pragma unroll
    for (int l = 0; l < kLoads; l++)
      raw[l] = ld_ordered_stream_u4(reinterpret_cast<const uint4*>(in) + v * kLoads + l);
    float f[16], big = 0.f;
#pragma unroll
    for (int l = 0; l < kLoads; l++) {
      float g[kPerLoad];
      unpack16<T>(raw[l], g);
#pragma unroll
      for (int k = 0; k < kPerLoad; k++) {
        f[l * kPerLoad + k] = g[k];
        big = fmaxf(big, fabsf(g[k]));
      }
    }
    int q[16];
    if (fast && big < limit) {  // limit: quotients far inside int32, no infinity
#pragma unroll
      for (int k = 0; k < 16; k++) q[k] = __float2int_rn(exact_quotient(f[k], scale, inv));
    } else {
#pragma unroll
      for (int k = 0; k < 16; k++) q[k] = __float2int_rn(__fdiv_rn(f[k], scale));
    }
    uint32_t o[4];
#pragma unroll
    for (int w = 0; w < 4; w++) {
      if (AZP) {
#pragma unroll
        for (int b = 0; b < 4; b++) q[4 * w + b] = (int)((unsigned)q[4 * w + b] + (unsigned)azp);
      }
      o[w] = pack_sat8(q[4 * w], q[4 * w + 1], q[4 * w + 2], q[4 * w + 3]);
    }
    reinterpret_cast<uint4*>(out)[v] = make_uint4(o[0], o[1], o[2], o[3]);
  }
  // tail (and everything, when the buffers are not 16-byte aligned)
  for (size_t i = nvec * 16 + (size_t)blockIdx.x * kThreads + threadIdx.x; i < n; i += stride) {
    const float q = __fdiv_rn(to_float<T>(in[i]), scale);
    out[i] = (int8_t)(AZP ? f2i8_azp(q, azp) : f2i8_rn(q));
  }
}

// Running extremes of packed elements (a NaN never wins); Extremes<T>::type holds
// them as T pairs, or as floats for fp32.
template <typename T>
struct Extremes {
  uint32_t mx, mn;  // two T each
  __device__ __forceinline__ static uint32_t neutral(bool max_side) {
    const uint32_t inf = sizeof(T) == 2 && std::is_same<T, __half>::value ? 0x7c007c00u : 0x7f807f80u;
    return max_side ? inf | 0x80008000u : inf;
  }
  __device__ __forceinline__ Extremes() : mx(neutral(true)), mn(neutral(false)) {}
  template <bool ABS>
  __device__ __forceinline__ void take(uint32_t w) {
    using T2 = typename std::conditional<std::is_same<T, __half>::value, __half2, __nv_bfloat162>::type;
    T2 x = *reinterpret_cast<const T2*>(&w), a = *reinterpret_cast<const T2*>(&mx),
       b = *reinterpret_cast<const T2*>(&mn);
    a = __hmax2(a, ABS ? __habs2(x) : x);
    mx = *reinterpret_cast<const uint32_t*>(&a);
    if (!ABS) {
      b = __hmin2(b, x);
      mn = *reinterpret_cast<const uint32_t*>(&b);
    }
  }
  __device__ __forceinline__ float high() const {
    const T* e = reinterpret_cast<const T*>(&mx);
    return fmaxf(to_float<T>(e[0]), to_float<T>(e[1]));
  }
  __device__ __forceinline__ float low() const {
    const T* e = reinterpret_cast<const T*>(&mn);
    return fminf(to_float<T>(e[0]), to_float<T>(e[1]));
  }
};
template <>
struct Extremes<float> {
  float mx, mn;
  __device__ __forceinline__ Extremes() : mx(-INFINITY), mn(INFINITY) {}
  template <bool ABS>
  __device__ __forceinline__ void take(uint32_t w) {
    const float x = __uint_as_float(w);
    mx = fmaxf(mx, ABS ? fabsf(x) : x);
    if (!ABS) mn = fminf(mn, x);
  }
  __device__ __forceinline__ float high() const { return mx; }
  __device__ __forceinline__ float low() const { return mn; }
};

// ---- dynamic forms: one CTA per token row ----
// Vector form.  The tensor is viewed as aligned 16-byte chunks (EPC = 8 or 4
// elements); the CTA of row t takes the chunks that overlap [t*hidden,
// (t+1)*hidden) - a chunk on a row boundary is read by both rows' CTAs and each
// masks the elements of the other row.  A thread keeps CPT chunks in registers
// (chunks tid, tid + blockDim, ...), so the row is read once, with full-width
// loads whatever the row's starting address is.  The eight (four) results of a
// chunk inside the row leave as one 8-byte (4-byte) store; a boundary chunk
// stores its in-row bytes one by one.
template <typename T, bool AZP, int CPT>
__global__ void __launch_bounds__(1024)
vllm_dynamic_vec_kernel(const T* in, int8_t* __restrict__ out,
                        float* __restrict__ scale_out, int* __restrict__ azp_out, int num_tokens,
                        int hidden) {
  pdl_launch_dependents();
  pdl_wait();  // nothing is read or written before every earlier kernel has completed
  constexpr int EPC = 16 / sizeof(T);
  constexpr int EPW = 4 / sizeof(T);  // elements per 32-bit word
  __shared__ float2 sh[32];  // a warp's maximum and minimum
  const int tid = threadIdx.x, threads = blockDim.x;
  const size_t total = (size_t)num_tokens * hidden;
  const int t = blockIdx.x;
  const size_t e0 = (size_t)t * hidden;  // the row's elements start here, flat
  const size_t c0 = e0 / EPC;            // first chunk that overlaps the row
  const int skip = (int)(e0 - c0 * EPC); // its elements that belong to the row before
  const int end = skip + hidden;         // the row in elements counted from chunk c0
  const uint4* src = reinterpret_cast<const uint4*>(in) + c0;
  uint4 raw[CPT];
#pragma unroll
  for (int j = 0; j < CPT; j++) {
    const int c = tid + j * threads, first = c * EPC;
    raw[j] = make_uint4(0, 0, 0, 0);
    if (first >= end) continue;
    if ((c0 + c) * EPC + EPC <= total) {
      if (HQ_IN_BOUNDS(src + c, 16, in, total * sizeof(T), 403)) raw[j] = ld_ordered_stream_u4(src + c);
    } else {  // the last chunk of the tensor may be partial: it is fetched element-wise
      T* r = reinterpret_cast<T*>(&raw[j]);
      for (int k = 0; k < EPC; k++)
        if ((c0 + c) * EPC + k < total) r[k] = in[(c0 + c) * EPC + k];
    }
  }
  Extremes<T> ext;
#pragma unroll
  for (int j = 0; j < CPT; j++) {
    const int first = (tid + j * threads) * EPC;
    const uint32_t w[4] = {raw[j].x, raw[j].y, raw[j].z, raw[j].w};
    if (first >= skip && first + EPC <= end) {  // wholly inside the row: no masks
#pragma unroll
      for (int k = 0; k < 4; k++) ext.template take<!AZP>(w[k]);
    } else if (first < end) {
      // a row boundary: the neighbour's elements are replaced by zeros for the largest
      // magnitude, else by one of this row (the chunk's first or last, whichever end of
      // the row it holds)
      const int own = max(skip - first, 0);
      const T* e = reinterpret_cast<const T*>(&raw[j]);
#pragma unroll
      for (int k = 0; k < 4; k++) {
        uint32_t u = 0;
#pragma unroll
        for (int h = 0; h < EPW; h++) {
          const int i = EPW * k + h, at = first + i;
          T x = e[i];
          if (at < skip || at >= end) {
            x = AZP ? e[0] : T(0.f);
#pragma unroll
            for (int o = 1; o < EPC; o++) x = AZP && o == own ? e[o] : x;
          }
          if (EPW == 2) u |= (uint32_t)*reinterpret_cast<const unsigned short*>(&x) << (16 * h);
          else u = *reinterpret_cast<const uint32_t*>(&x);
        }
        ext.template take<!AZP>(u);
      }
    }
  }
  // reference.h:40-46 / :66-72: NaN inputs never win a compare, the running maximum of
  // the zero-point form starts at FLT_MIN
  float mx = fmaxf(AZP ? FLT_MIN : 0.f, ext.high()), mn = AZP ? fminf(FLT_MAX, ext.low()) : 0.f;
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, o));
    if (AZP) mn = fminf(mn, __shfl_xor_sync(0xffffffffu, mn, o));
  }
  if ((tid & 31) == 0) sh[tid >> 5] = make_float2(mx, mn);
  __syncthreads();
  for (int w = 0; w < threads >> 5; w++) {
    const float2 e = sh[w];
    mx = fmaxf(mx, e.x);
    if (AZP) mn = fminf(mn, e.y);
  }
  float scale, mul = 0.f;
  int azp = 0;
  bool fast = false;
  if (AZP) {
    scale = __fdiv_rn(__fsub_rn(mx, mn), 255.0f);
    azp = __float2int_rz(rintf(__fsub_rn(-128.0f, __fdiv_rn(mn, scale))));
    mul = __frcp_rn(scale);
    fast = divides_fast(scale) && fmaxf(mx, fabsf(mn)) < scale * 1073741824.f;
  } else {
    scale = __fdiv_rn(mx, 127.0f);
    mul = __fdiv_rn(127.0f, mx);
  }
  if (tid == 0) {
    scale_out[t] = scale;
    if (AZP) azp_out[t] = azp;
  }
  int8_t* dst = out + c0 * EPC;
  // quantizes and stores the thread's chunks; value() is the scaled element
  auto finish = [&](auto value) {
#pragma unroll
    for (int j = 0; j < CPT; j++) {
      const int first = (tid + j * threads) * EPC;
      if (first >= end) continue;
      float f[EPC];
      unpack16<T>(raw[j], f);
      int q[EPC];
#pragma unroll
      for (int k = 0; k < EPC; k++) {
        q[k] = __float2int_rn(value(f[k]));
        if (AZP) q[k] = (int)((unsigned)q[k] + (unsigned)azp);
      }
      uint32_t o[EPC / 4];
#pragma unroll
      for (int k = 0; k < EPC / 4; k++)
        o[k] = pack_sat8(q[4 * k], q[4 * k + 1], q[4 * k + 2], q[4 * k + 3]);
      if (first >= skip && first + EPC <= end) {  // wholly inside the row: one aligned store
        if (HQ_IN_BOUNDS(dst + first, EPC, out, total, 404)) {
          if (EPC == 8) *reinterpret_cast<uint2*>(dst + first) = make_uint2(o[0], o[EPC / 4 - 1]);
          else *reinterpret_cast<uint32_t*>(dst + first) = o[0];
        }
      } else {
#pragma unroll
        for (int k = 0; k < EPC; k++)
          if (first + k >= skip && first + k < end)
            dst[first + k] = (int8_t)((o[k / 4] >> (8 * (k & 3))) & 0xff);
      }
    }
  };
  if (!AZP) finish([&](float x) { return __fmul_rn(x, mul); });
  else if (fast) finish([&](float x) { return exact_quotient(x, scale, mul); });
  else finish([&](float x) { return __fdiv_rn(x, scale); });
}

__device__ __forceinline__ float block_reduce(float v, bool is_max, float* sh) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    const float u = __shfl_xor_sync(0xffffffffu, v, o);
    v = is_max ? fmaxf(v, u) : fminf(v, u);
  }
  __syncthreads();  // sh may still be read from an earlier reduction
  if (lane == 0) sh[warp] = v;
  __syncthreads();
  float r = sh[0];
#pragma unroll
  for (int w = 1; w < kWarps; w++) r = is_max ? fmaxf(r, sh[w]) : fminf(r, sh[w]);
  return r;
}

// Element-wise form for buffers that are not 16 / 8-byte aligned and for rows
// longer than the register cache.  EPT: elements per thread kept in registers;
// EPT == 0 re-reads the row.
template <typename T, bool AZP, int EPT>
__global__ void __launch_bounds__(kThreads)
vllm_dynamic_kernel(const T* in, int8_t* __restrict__ out,
                    float* __restrict__ scale_out, int* __restrict__ azp_out, int num_tokens,
                    int hidden) {
  pdl_launch_dependents();
  pdl_wait();  // nothing is read or written before every earlier kernel has completed
  __shared__ float sh[kWarps];
  const int tid = threadIdx.x;
  for (int t = blockIdx.x; t < num_tokens; t += gridDim.x) {
    const T* row = in + (size_t)t * hidden;
    int8_t* orow = out + (size_t)t * hidden;
    float v[EPT > 0 ? EPT : 1];
    // reference.h:40-46 / :66-72: NaN inputs never win a compare
    float mx = AZP ? FLT_MIN : 0.f, mn = FLT_MAX;
    if (EPT > 0) {
#pragma unroll
      for (int j = 0; j < EPT; j++) {
        const int i = tid + j * kThreads;
        v[j] = i < hidden ? to_float<T>(row[i]) : (AZP ? FLT_MIN : 0.f);
      }
#pragma unroll
      for (int j = 0; j < EPT; j++) {
        if (AZP) {
          mx = fmaxf(mx, v[j]);
          if (tid + j * kThreads < hidden) mn = fminf(mn, v[j]);
        } else {
          mx = fmaxf(mx, fabsf(v[j]));
        }
      }
    } else {
      for (int i = tid; i < hidden; i += kThreads) {
        const float x = to_float<T>(row[i]);
        if (AZP) { mx = fmaxf(mx, x); mn = fminf(mn, x); }
        else mx = fmaxf(mx, fabsf(x));
      }
    }
    mx = block_reduce(mx, true, sh);
    float scale, mul = 0.f;
    int azp = 0;
    if (AZP) {
      mn = block_reduce(mn, false, sh);
      scale = __fdiv_rn(__fsub_rn(mx, mn), 255.0f);
      azp = __float2int_rz(rintf(__fsub_rn(-128.0f, __fdiv_rn(mn, scale))));
    } else {
      scale = __fdiv_rn(mx, 127.0f);
      mul = __fdiv_rn(127.0f, mx);
    }
    if (tid == 0) {
      scale_out[t] = scale;
      if (AZP) azp_out[t] = azp;
    }
    if (EPT > 0) {
#pragma unroll
      for (int j = 0; j < EPT; j++) {
        const int i = tid + j * kThreads;
        if (i < hidden)
          orow[i] = (int8_t)(AZP ? f2i8_azp(__fdiv_rn(v[j], scale), azp)
                                 : f2i8_rn(__fmul_rn(v[j], mul)));
      }
    } else {
      for (int i = tid; i < hidden; i += kThreads) {
        const float x = to_float<T>(row[i]);
        orow[i] = (int8_t)(AZP ? f2i8_azp(__fdiv_rn(x, scale), azp) : f2i8_rn(__fmul_rn(x, mul)));
      }
    }
  }
}

template <typename T>
int static_launch(int8_t* out, const void* in, size_t n, float scale, int azp, cudaStream_t st) {
  const int vec_ok = aligned16(in) && aligned16(out);
  const size_t want = (n / 16 + kThreads - 1) / kThreads;
  const size_t cap = (size_t)sm_count() * 16;
  const unsigned grid = (unsigned)(want < 1 ? 1 : (want < cap ? want : cap));
  const T* x = reinterpret_cast<const T*>(in);
  if (azp == 0)  // the launcher's choice, main.cu:147-152
    return cuda_status(launch_pdl(vllm_static_kernel<T, false>, dim3(grid), dim3(kThreads), 0, st, x, out,
                                  n, scale, azp, vec_ok));
  return cuda_status(launch_pdl(vllm_static_kernel<T, true>, dim3(grid), dim3(kThreads), 0, st, x, out, n,
                                scale, azp, vec_ok));
}

template <typename T, bool AZP>
int dynamic_launch_ept(int8_t* out, const T* x, float* scales, int* azp, int tokens, int hidden,
                       cudaStream_t st) {
  const unsigned grid = (unsigned)std::min(tokens, sm_count() * 32);
  constexpr int EPC = 16 / sizeof(T);
  // chunks a row can overlap: exactly its own where rows start on chunk boundaries
  const long chunks = hidden % EPC == 0 ? hidden / EPC : ((long)hidden + EPC - 2) / EPC + 1;
  // Chunks per thread: with rows for every SM the count that leaves the fewest thread
  // slots of its whole-warp block without a chunk (a row of 644 chunks: 3 x 224
  // threads) among blocks of at most 256 threads, so that some of an SM's blocks
  // load while others store (8192 x 16384 fp16: 62 us, with blocks of 512 and 1024
  // threads 79 and 91), larger blocks where the row needs them.  One chunk per thread
  // where a warp covers the row and where there are too few rows to fill the SMs: below
  // two per SM, or 24 warps per SM in all (300 x 1025 fp16, 10 warps per SM: 1.83 us,
  // with two chunks per thread 2.46; 900 x 1025, 30: 2.21 and 2.62; 1800 x 1025, 61:
  // 3.62 and 3.23; 900 x 2049, 55: 3.03 and 2.86).
  int cpt = 0, threads = 0;
  if (aligned16(x) && aligned8(out) && chunks <= 8L * 1024) {
    const long sms = sm_count(), warps = (chunks + 31) / 32;
    const int lo = warps == 1 || tokens < 2 * sms || tokens * warps <= 24 * sms ? 1 : 2;
    long best = 0;
    for (int c = lo; c <= 8; c++) {
      const long th = (chunks + c - 1) / c, w = (th + 31) / 32 * 32;
      if (w > (lo == 1 || c == 8 ? 1024 : 256)) continue;
      if (cpt && (lo == 1 || w * c >= best)) continue;
      cpt = c, threads = (int)w, best = w * c;
    }
  }
  auto go = [&](auto kern, unsigned blocks, int block) {
    return cuda_status(launch_pdl(kern, dim3(blocks), dim3(block), 0, st, x, out, scales, azp, tokens, hidden));
  };
  switch (cpt) {
    case 1: return go(vllm_dynamic_vec_kernel<T, AZP, 1>, tokens, threads);
    case 2: return go(vllm_dynamic_vec_kernel<T, AZP, 2>, tokens, threads);
    case 3: return go(vllm_dynamic_vec_kernel<T, AZP, 3>, tokens, threads);
    case 4: return go(vllm_dynamic_vec_kernel<T, AZP, 4>, tokens, threads);
    case 5: return go(vllm_dynamic_vec_kernel<T, AZP, 5>, tokens, threads);
    case 6: return go(vllm_dynamic_vec_kernel<T, AZP, 6>, tokens, threads);
    case 7: return go(vllm_dynamic_vec_kernel<T, AZP, 7>, tokens, threads);
    case 8: return go(vllm_dynamic_vec_kernel<T, AZP, 8>, tokens, threads);
  }
  if (hidden <= 8 * kThreads) return go(vllm_dynamic_kernel<T, AZP, 8>, grid, kThreads);
  if (hidden <= 16 * kThreads) return go(vllm_dynamic_kernel<T, AZP, 16>, grid, kThreads);
  if (hidden <= 32 * kThreads) return go(vllm_dynamic_kernel<T, AZP, 32>, grid, kThreads);
  return go(vllm_dynamic_kernel<T, AZP, 0>, grid, kThreads);
}

template <typename T>
int dynamic_launch(int8_t* out, const void* in, float* scales, int* azp, int tokens, int hidden,
                   cudaStream_t st) {
  const T* x = reinterpret_cast<const T*>(in);
  return azp == nullptr ? dynamic_launch_ept<T, false>(out, x, scales, nullptr, tokens, hidden, st)
                        : dynamic_launch_ept<T, true>(out, x, scales, azp, tokens, hidden, st);
}

int check_common(const void* out, const void* in, int dtype, int hidden, int tokens) {
  if (!out || !in) return HQ_ERR_NULL_POINTER;
  if (hidden <= 0 || tokens <= 0) return HQ_ERR_BAD_SHAPE;
  if (dtype != HQ_DTYPE_F16 && dtype != HQ_DTYPE_BF16 && dtype != HQ_DTYPE_F32)
    return HQ_ERR_UNSUPPORTED;
  const uintptr_t a = reinterpret_cast<uintptr_t>(in);
  if (a & (dtype == HQ_DTYPE_F32 ? 3u : 1u)) return HQ_ERR_MISALIGNED;
  return HQ_OK;
}

}  // namespace
}  // namespace hq

extern "C" {

int hq_vllm_static_scaled_int8_quant(int8_t* out, const void* input, int dtype, int hidden_size,
                                     int num_tokens, float scale, int32_t azp,
                                     hq_stream_t stream) {
  using namespace hq;
  const int st = check_common(out, input, dtype, hidden_size, num_tokens);
  if (st != HQ_OK) return st;
  const size_t n = (size_t)num_tokens * (size_t)hidden_size;
  cudaStream_t s = (cudaStream_t)stream;
  if (dtype == HQ_DTYPE_F16) return static_launch<__half>(out, input, n, scale, azp, s);
  if (dtype == HQ_DTYPE_BF16) return static_launch<__nv_bfloat16>(out, input, n, scale, azp, s);
  return static_launch<float>(out, input, n, scale, azp, s);
}

int hq_vllm_dynamic_scaled_int8_quant(int8_t* out, const void* input, int dtype, int hidden_size,
                                      int num_tokens, float* scales, int32_t* azp,
                                      hq_stream_t stream) {
  using namespace hq;
  const int st = check_common(out, input, dtype, hidden_size, num_tokens);
  if (st != HQ_OK) return st;
  if (!scales) return HQ_ERR_NULL_POINTER;
  cudaStream_t s = (cudaStream_t)stream;
  if (dtype == HQ_DTYPE_F16)
    return dynamic_launch<__half>(out, input, scales, azp, num_tokens, hidden_size, s);
  if (dtype == HQ_DTYPE_BF16)
    return dynamic_launch<__nv_bfloat16>(out, input, scales, azp, num_tokens, hidden_size, s);
  return dynamic_launch<float>(out, input, scales, azp, num_tokens, hidden_size, s);
}

}  // extern "C"
