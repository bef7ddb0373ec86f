// The streamed form of the batched product (formats, helpers and the rule that chooses it:
// qgemm.cu), for long layers: some 16 steps of 128 inputs x 256 features per SM for 3-bit, 10 for
// NF4.
//
// One CTA of 608 threads per SM takes a contiguous range of (tile, step) units, so that
// every SM has the same work whatever the number of tiles; a tile is 256 output features
// (two UMMA M = 128 subtiles that share the X tile of a step), a tile that a range cuts
// meets the rest of its parts in the fp32 scratch.
//   warps 0-15  unpack: four groups of four warps = (subtile, every other step), beyond 64 tokens
//               (subtile, half of every step); thread = one output feature; 64 weights of a half
//               go to 32 columns of the stage in tensor memory, eight columns at a time;
//   warp 16     MMA issuer: 16 tcgen05.mma (K = 16) and one commit per step;
//   warp 17     packed words of a step by TMA into a ring (3-bit 12 rows x 256 words and the
//               scales and zeros, NF4 256 rows x 64 bytes and their absmax values);
//   warp 18     X by TMA into the stages, 64 inputs x all tokens per half.
//
// What bounds it.  3-bit, up to 64 tokens: issue slots, 3360 instructions a step with all
// roles and the ends (4175 before the two changes below), 1630 of them the unpacking (a byte
// permute, a look-up, an fp16 fma per pair), and the ends of the ranges (15 of 41 us at 64 x 8192 x 28672).  NF4: the shared-memory pipe, two wavefronts
// for every look-up of a byte, 1024 of a step's 1430 cycles.  Beyond 64 tokens: the two stages that
// tensor memory leaves.
//  * A table row is a byte and a lane's copy, one byte permute, for both formats: four 3-bit pairs lie in
//    three bytes, and with the stream shifted by four bits each of them is the high or the low part
//    of one byte (shift and mask per pair before: 3-bit 64 x 8192 x 28672 46.4 -> 43.6 us, NF4 37 x 28672
//    x 8192 66.1 -> 64.8);
//  * up to 64 tokens a warp unpacks both halves of every other step, so that barriers, rings and waits
//    are paid once for 128 weights of a thread (43.6 -> 42.1, 64.8 -> 61; beyond 64 tokens, on two
//    stages, no gain for 3-bit and 5 % more for NF4: there a warp takes one half of every step);
//  * NF4's absmax values, 4 bytes from each of 32 rows per warp and half step, were 32 wavefronts
//    of the load pipe; the TMA unit brings them with the words (57.8 -> 48.7; 100 x 28672 x 8192 72.6 ->
//    64.7).
// The tables and slots take 217 to 230 KB of shared memory (172 and 180 before): no neighbour in the stream
// becomes resident beside this kernel any more.  In chains the gain is larger than that: 64 tokens int8-quantized,
// then x 8192 x 28672, 3-bit 50.8 -> 47.8 us (the quantizer's share 4.6 -> 5.8; in a graph 52.3 -> 48.3), NF4 74.4 ->
// 59.5; followed by an int4 mat-vec of 4096 x 4096 51.3 -> 47.9 and 76.6 -> 59.6.
// Of what the other form spent:
//  * tcgen05.mma takes N / 2 cycles on the tensor pipe, but issuing one took 64 (a commit 95)
//    where its addresses come from registers, 26 (15) where they are constants: the CTA
//    takes all 512 columns of tensor memory, which start at 0, and the only shared memory
//    is the dynamic region at a checked, fixed address;
//  * a wait for a barrier that is over costs 100 to 250 cycles among other warps: there is one
//    stage barrier per step for A, X and all groups, the unpack warps ask about the next
//    step's barriers before their arithmetic and read its words while their stores are under
//    way, and waiting warps sleep in try_wait instead of polling;
//  * 224 tiles of 128 features left 72 of 148 SMs half empty.
// us of a call among some hundreds at 1965 MHz (over a second the power cap takes the clock to some
// 1700 MHz: 3-bit 64 x 8192 x 28672 49.5, NF4 37 x 28672 x 8192 56.1), the other form -> this one, 3-bit (NF4): 64
// x 8192 x 28672 56.3 -> 41 (89.6 -> 53), 128 x 8192 x 28672 82.6 -> 57.6 (116.6 -> 70.5), 64 x 28672 x 8192
// 45 -> 40.7 (80 -> 52.2), 32 x 8192 x 14336 31.8 -> 26.7 (48.6 -> 32.5), 64 x 4096 x 28672 31 -> 28.3 (46 ->
// 35.2).  On short layers the ends of the ranges outweigh the rest: 64 x 8192 x 8192, 14 steps, 20.4 and 22.1
// (29.2 and 27), 64 x 4096 x 6144 12.1 and 17.1.  Unpacking 3-bit pairs by byte permutes and magic numbers
// instead of the table takes more slots: 51.6 for 46.4 at 64 x 8192 x 28672 (half of the pairs: 48.1).
// Taken back: reading a tile's accumulators one step into the next, and settling the parts of
// a cut tile warp by warp without a barrier of the CTA, are shorter at the ends of ranges but
// cost the inner loop its registers (96 of 96, spills): 3-bit 64 x 8192 x 28672 55.6 and 49.5 for 46.4.  A tile's
// last part taking the others' sum from the scratch instead of adding its own there: 40.9 -> 42.3,
// NF4 48.7 -> 51.2.
#ifndef HQ_QGEMM_STREAM_CUH_
#define HQ_QGEMM_STREAM_CUH_
namespace hq {
namespace {
namespace streamed {

constexpr int kBlockK = 64;                 // inputs of half a step: 128 bytes of an X row
constexpr int kTileN = 256;                 // output features per tile: two UMMA M = 128 subtiles
constexpr int kAColumns = kBlockK / 2;      // tensor-memory columns of one A tile (2 halves each)
constexpr int kUnpackWarps = 16;
constexpr int kIssueWarp = kUnpackWarps;
constexpr int kThreads = (kUnpackWarps + 3) * 32;  // + MMA issuer, word TMA, X TMA
constexpr uint32_t kBase = 1024;            // shared-window address of the dynamic region

// Depths and layout of a CTA; WIDE: more than 64 tokens.
//   tensor memory: accumulators of the two subtiles, then kStages stages of four A tiles
//   shared memory: X [stage][half][tokens x 128 bytes], word ring, lookup table, barriers, one
//   word of notes
//   word slot: 3-bit 12 rows x 256 words, then scales and zeros [half][256];
//   NF4 256 rows x 64 bytes (64-byte swizzle), then (AM) 16 bytes of absmax for each row
//   table, by byte value: 3-bit [256][2][32 copies] of half2, the pair in the byte's low six bits and
//   the one in its high six; NF4 [256][32 or 16 copies] of float2 (the two levels of the byte's
//   codes).  A lane reads a copy of its own (16: the lanes of a half-warp do), so 16 or 32 lanes read
//   different banks whatever their bytes are
//   AM: NF4 whose absmax values come with the words (else the unpack warps load them)
template <int FMT, bool WIDE, bool AM>
struct Shape {
  static constexpr int kTokens = WIDE ? 128 : 64;
  static constexpr int kStages = WIDE ? 2 : 3;
  // Unpack warps 0-7 and 8-15 take every other step, both halves of it, where there are stages enough
  // (WIDE: every step, one half each): what a step costs besides its unpacking is then paid for 128
  // weights of a thread at a time, not 64.
  static constexpr bool kAlternate = !WIDE && (FMT == kFmtQ3 || AM);
  static constexpr int kHalves = kAlternate ? 2 : 1;          // halves of a step that a warp unpacks
  static constexpr int kStepWarps = kAlternate ? 8 : 16;      // unpack warps of a step
  static constexpr uint32_t kACol = 2 * kTokens;
  static_assert(kACol + 4 * kStages * kAColumns <= 512, "tensor memory");
  static constexpr int kXHalf = kTokens * 128;
  static constexpr int kXRing = kStages * 2 * kXHalf;
  static constexpr int kWordSlots = FMT == kFmtQ3 ? (WIDE ? 7 : 8) : (WIDE || !AM ? 6 : 5);
  static constexpr int kWordBytes = FMT == kFmtQ3 ? 14 * 1024 : AM ? 20 * 1024 : 16 * 1024;
  // Rows of the table: 256 bytes, whose address is one byte permute, where shared memory allows;
  // without AM the rest is left to L1, which holds the absmax lines (64 x 28608 x 8192 61.4 us, with
  // 256-byte rows and slots of 20 KB 66.7; 100 tokens 68.6 and 74.1).
  static constexpr int kTabRow = FMT == kFmtNf4 && (WIDE || !AM) ? 128 : 256;
  static constexpr int kLut = kXRing + kWordSlots * kWordBytes;
  static constexpr int kBars = kLut + 256 * kTabRow;
  static constexpr int kBarBytes = 8 * (2 * kStages + 2 * kWordSlots + 2);
  static constexpr int kSmem = kBars + kBarBytes + 16;
  static_assert(kSmem <= 227 * 1024, "shared memory");
};

struct Params {
  __half* Y;
  float* ws;            // fp32 [Mb][N] scratch + per-tile counters
  unsigned* counters;
  int* status;
  int Mb, N, K, group_size, tokens_padded;
  int tiles, steps;     // 256-feature tiles, 128-input steps of a tile
  int ordered;          // the parts of a tile add to the scratch in a fixed order
  int one_group;        // 3-bit: both halves of a step lie in one scale group
  int am_shift;         // NF4: log2 of the 64-input blocks per absmax value, or -1
  // NF4 only (group_size is the absmax block size there)
  const float* absmax;
  const float* lut16;
  int low_first;
};

// Bounded wait like the other form's; a poll may sleep, so that the warps that wait leave
// the issue slots to those that unpack.
constexpr uint32_t kSuspendNs = 20000;
constexpr uint32_t kWaits = 1u << 16;  // about a second
__device__ __forceinline__ bool mbar_wait(uint32_t bar, uint32_t parity, bool healthy) {
  if (!healthy) return false;
  for (uint32_t i = 0; i < kWaits; i++) {
    uint32_t done;
    asm volatile(
        "{\n .reg .pred p;\n"
        " mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2, %3;\n"
        " selp.u32 %0, 1, 0, p;\n}\n"
        : "=r"(done)
        : "r"(bar), "r"(parity), "r"(kSuspendNs)
        : "memory");
    if (done) return true;
  }
  return false;
}

__device__ __forceinline__ void tmem_store(uint32_t taddr, const uint32_t (&v)[8]) {
  asm volatile("tcgen05.st.sync.aligned.32x32b.x8.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8};" ::"r"(taddr), "r"(v[0]), "r"(v[1]), "r"(v[2]), "r"(v[3]), "r"(v[4]), "r"(v[5]), "r"(v[6]), "r"(v[7])
               : "memory");
}

// whether the phase with the given parity is over, without waiting: this lane's answer, the
// caller brings the warp together
__device__ __forceinline__ bool mbar_test(uint32_t bar, uint32_t parity) {
  uint32_t done;
  asm volatile(
      "{\n .reg .pred p;\n"
      " mbarrier.test_wait.parity.shared::cta.b64 p, [%1], %2;\n"
      " selp.u32 %0, 1, 0, p;\n}\n"
      : "=r"(done)
      : "r"(bar), "r"(parity)
      : "memory");
  return done != 0;
}

// A ring position and the parity of its current round.
template <int N>
struct Ring {
  uint32_t at = 0, parity = 0;
  __device__ __forceinline__ void next() {
    if (++at == N) { at = 0; parity ^= 1u; }
  }
  template <int D>
  __device__ __forceinline__ void skip() {
    static_assert(D <= N, "one turn at most");
    if (D == 1) return next();
    at += D;
    if (at >= N) { at -= N; parity ^= 1u; }
  }
};

// Byte B of the words next to this lane's place in a table row: row and copy in one byte permute
// (the byte in bits 8 to 15, the lane's place in bits 0 to 7).
template <int B>
__device__ __forceinline__ uint32_t table_at(uint32_t word, uint32_t place) {
  return __byte_perm(word, place, 0x7604u | (uint32_t)(B << 4));
}
// Pair E (codes 2E, 2E + 1) of the 32 in three words w of the 96-bit stream to half2 weights.  Four
// pairs are three bytes.  The first is the low six bits of the first byte and the last the high
// six bits of the third; with the stream shifted by four bits (v) the second is the high part of
// the first byte and the third the low part of the second: a byte and one of two tables for each.
template <int E, int LUT>
__device__ __forceinline__ uint32_t q3_pair(const uint32_t (&w)[3], const uint32_t (&v)[3], __half2 sc2,
                                            __half2 nz2, uint32_t lane4) {
  constexpr int i = E % 4, byte = E / 4 * 3 + (i == 3 ? 2 : i == 2 ? 1 : 0);
  constexpr bool high = i & 1;
  const uint32_t at = table_at<byte % 4>(i == 0 || i == 3 ? w[byte / 4] : v[byte / 4], lane4);
  uint32_t q2;
  asm("ld.shared.u32 %0, [%1+%2];" : "=r"(q2) : "r"(at), "n"(LUT + (high ? 128 : 0)));
  return half2_as_u32(__hfma2(u32_as_half2(q2), sc2, nz2));
}
// pairs E0 .. E0 + N - 1 of three words
template <int E0, int LUT, int N, int... E>
__device__ __forceinline__ void q3_pairs(const uint32_t (&w)[3], const uint32_t (&v)[3], __half2 sc2, __half2 nz2,
                                         uint32_t lane4, uint32_t (&o)[N], std::integer_sequence<int, E...>) {
  ((o[E] = q3_pair<E0 + E, LUT>(w, v, sc2, nz2, lane4)), ...);
}
template <int E0, int LUT, int N>
__device__ __forceinline__ void q3_words(const uint32_t (&w)[3], const uint32_t (&v)[3], __half2 sc2, __half2 nz2,
                                         uint32_t lane4, uint32_t (&o)[N]) {
  q3_pairs<E0, LUT>(w, v, sc2, nz2, lane4, o, std::make_integer_sequence<int, N>());
}

// The units of work are (tile, step) pairs, numbered tile by tile.  CTA c takes units
// first_unit(r) .. first_unit(r + 1) - 1 of place r = gridDim.x - 1 - c, so that the parts of a
// tile that an ordered sum waits for belong to CTAs that started earlier.
__device__ __forceinline__ int first_unit(const Params& p, int r) {
  return (int)((long long)p.tiles * p.steps * r / (int)gridDim.x);
}
// the place whose range holds unit u
__device__ __forceinline__ int owner(const Params& p, int u) {
  return (int)((((long long)u + 1) * gridDim.x - 1) / ((long long)p.tiles * p.steps));
}

template <int FMT, bool WIDE, bool AM>
__global__ void __launch_bounds__(kThreads, 1)
qgemm_stream_kernel(const __grid_constant__ CUtensorMap map_x, const __grid_constant__ CUtensorMap map_w,
                    const __grid_constant__ CUtensorMap map_s, const __grid_constant__ CUtensorMap map_z,
                    const Params p) {
  using S = Shape<FMT, WIDE, AM>;
  extern __shared__ __align__(1024) unsigned char dsm_raw[];
  // The kernel has no static shared memory, so the dynamic region starts behind the KiB that
  // the system reserves: every address below is a constant.  (The swizzle pattern of the
  // tiles repeats every 1024 bytes.)  The host has checked it; never taken.
  if (smem_u32(dsm_raw) != kBase) {
    if (p.status != nullptr) atomicExch(p.status, 1);
    return;
  }
  unsigned char* const sm = dsm_raw;
  constexpr uint32_t x_ring = kBase, w_ring = kBase + S::kXRing, bars = kBase + S::kBars;
  // full[stage]: its kStepWarps unpack warps have written their rows of the stage's A tiles and its X
  //              tile has landed;  empty[stage]: the MMAs that read them have completed
  // wfull / wempty: the packed words of a step have landed / its unpack warps read them
  // done: accumulators complete (and, ordered, it is this part's turn)
  // taken: accumulators read, the next segment may overwrite them
  constexpr uint32_t full = bars, empty = full + 8 * S::kStages;
  constexpr uint32_t wfull = empty + 8 * S::kStages, wempty = wfull + 8 * S::kWordSlots;
  constexpr uint32_t done = wempty + 8 * S::kWordSlots, taken = done + 8;
  volatile uint32_t* note = reinterpret_cast<uint32_t*>(sm + S::kBars + S::kBarBytes);

  const int tid = threadIdx.x, lane = tid & 31;
  const int warp = __shfl_sync(0xffffffffu, tid >> 5, 0);  // uniform for the compiler
  const int r = (int)(gridDim.x - 1 - blockIdx.x);
  const int u0 = first_unit(p, r), u1 = first_unit(p, r + 1);
  bool ok = true;

  if (tid == 0) {
    for (int i = 0; i < S::kStages; i++) {
      mbar_init(full + 8 * i, S::kStepWarps + 1);
      mbar_init(empty + 8 * i, 1);
    }
    for (int i = 0; i < S::kWordSlots; i++) {
      mbar_init(wfull + 8 * i, 1);
      mbar_init(wempty + 8 * i, S::kStepWarps);
    }
    mbar_init(done, 2);
    mbar_init(taken, kUnpackWarps);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (FMT == kFmtQ3) {
    uint32_t* lut = reinterpret_cast<uint32_t*>(sm + S::kLut);
    for (int i = tid; i < 256 * 16; i += kThreads) {  // 16 bytes: four copies
      const int v = (i & 8) ? i >> 6 : (i >> 4) & 63;
      const uint32_t e = half2_as_u32(__halves2half2(__int2half_rn(v & 7), __int2half_rn(v >> 3)));
      reinterpret_cast<uint4*>(lut)[i] = make_uint4(e, e, e, e);
    }
  }
  // Everything up to here needs no earlier kernel's results.  The wait stands before the
  // tensor-memory allocation, and the next kernel is let in after it: a CTA never holds
  // columns that an unfinished kernel still asks for.
  pdl_wait();
  if (FMT == kFmtNf4) {
    uint32_t* lut = reinterpret_cast<uint32_t*>(sm + S::kLut);
    for (int i = tid; i < 16 * S::kTabRow; i += kThreads) {  // 16 bytes: two copies
      const int b = i / (S::kTabRow / 16), hi = b >> 4, lo = b & 15;
      // even element = high nibble unless the low-nibble-first flag is given
      const uint32_t e0 = __float_as_uint(p.lut16[p.low_first ? lo : hi]);
      const uint32_t e1 = __float_as_uint(p.lut16[p.low_first ? hi : lo]);
      reinterpret_cast<uint4*>(lut)[i] = make_uint4(e0, e1, e0, e1);
    }
  }
  if (warp == kIssueWarp) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;"
                 ::"r"(bars + S::kBarBytes), "r"(512u)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  pdl_launch_dependents();
  // All 512 columns are this CTA's, so they start at column 0: every address below is a
  // constant, which the issuing thread needs in uniform registers (see the top).
  const uint32_t tmem_base = note[0];
  __syncthreads();  // note[0] is used again below

  if (warp < kUnpackWarps) {
    // ------------------------------ unpack warps ------------------------------
    // Four warps = the 128 rows of subtile s; a thread owns one output feature and unpacks its
    // weights.  grp: the steps of that parity of the CTA's range (alternate), or the half of every step.
    const int s = (warp >> 2) & 1, grp = warp >> 3;
    const int row = tid & 127, col = s * 128 + row;
    const uint32_t lanes = (uint32_t)((warp & 3) * 32) << 16;
    const uint32_t a_lane = lanes + S::kACol + (uint32_t)(((S::kAlternate ? 0 : grp * 2) + s) * kAColumns);
    constexpr int kEvery = S::kAlternate ? 2 : 1;
    Ring<S::kStages> a;
    Ring<S::kWordSlots> w;
    if (S::kAlternate) {
      a.at = (uint32_t)grp;
      w.at = (uint32_t)grp;
    }
    uint32_t segment = 0;
    // The words of a half are in registers before its arithmetic begins: those of a step's first
    // are read while the stores of the step before are under way, and both barriers that a step
    // needs are asked about ahead of its arithmetic.  Waited for one after the other
    // (words, stage, stores) the four warps of a scheduler met at the waits and again
    // at the arithmetic: 2300 cycles a step for 1000 of arithmetic, 3-bit.
    uint32_t nw[8];
    auto read_words = [&](int h) {
      const uint32_t slot = w_ring + w.at * S::kWordBytes;
      if constexpr (FMT == kFmtQ3) {
        const uint32_t src = slot + (uint32_t)(h * 6 * 1024 + col * 4);
        asm volatile("ld.shared.u32 %0, [%1];" : "=r"(nw[0]) : "r"(src));
        asm volatile("ld.shared.u32 %0, [%1+1024];" : "=r"(nw[1]) : "r"(src));
        asm volatile("ld.shared.u32 %0, [%1+2048];" : "=r"(nw[2]) : "r"(src));
        asm volatile("ld.shared.u32 %0, [%1+3072];" : "=r"(nw[3]) : "r"(src));
        asm volatile("ld.shared.u32 %0, [%1+4096];" : "=r"(nw[4]) : "r"(src));
        asm volatile("ld.shared.u32 %0, [%1+5120];" : "=r"(nw[5]) : "r"(src));
        const uint32_t par = slot + 12 * 1024 + (uint32_t)((p.one_group ? 0 : h * 512) + col * 2);
        uint16_t sc_bits, z_bits;
        asm volatile("ld.shared.u16 %0, [%1];" : "=h"(sc_bits) : "r"(par));
        asm volatile("ld.shared.u16 %0, [%1+1024];" : "=h"(z_bits) : "r"(par));
        nw[6] = sc_bits;
        nw[7] = z_bits;
      } else {
        // row `col` of the box: 64 bytes, its 16-byte pieces swizzled (64-byte pattern)
        const uint32_t src = slot + (uint32_t)(col * 64);
        const uint32_t x0 = (uint32_t)((2 * h) ^ ((col >> 1) & 3)) * 16u;
        asm volatile("ld.shared.v4.u32 {%0,%1,%2,%3}, [%4];"
                     : "=r"(nw[0]), "=r"(nw[1]), "=r"(nw[2]), "=r"(nw[3])
                     : "r"(src + x0));
        asm volatile("ld.shared.v4.u32 {%0,%1,%2,%3}, [%4];"
                     : "=r"(nw[4]), "=r"(nw[5]), "=r"(nw[6]), "=r"(nw[7])
                     : "r"(src + (x0 ^ 16u)));
      }
    };
    const int first_half = S::kAlternate ? 0 : grp;
    auto take_words = [&](bool ready) {
      if (!ready) {
        if (!mbar_wait(wfull + 8 * w.at, w.parity, ok)) ok = false;
        __syncwarp();
      }
      read_words(first_half);
    };
    int left = S::kAlternate ? (u1 - u0 + 1 - grp) >> 1 : u1 - u0;  // steps of this warp
    if (left > 0) take_words(false);

    for (int u = u0; u < u1;) {
      const int tile = u / p.steps, k0 = u - tile * p.steps;
      const int k1 = min(p.steps, k0 + (u1 - u));
      const int n = tile * kTileN + col;
      const int ka = S::kAlternate ? k0 + ((grp ^ (u - u0)) & 1) : k0;  // this warp's first step
      u += k1 - k0;

      // NF4, absmax: with the words (AM), else straight from global memory, one step ahead, where the 32
      // rows of a warp are 32 wavefronts of the load pipe.  Rows past N and a half step past K have none.
      [[maybe_unused]] const float* am_row = nullptr;
      [[maybe_unused]] auto absmax_at = [&](int k) {
        const int kb = 2 * k + grp;
        if (n >= p.N || kb * kBlockK >= p.K) return 0.f;
        return ld_ordered_f32(am_row + (p.am_shift >= 0 ? kb >> p.am_shift : kb * kBlockK / p.group_size));
      };
      [[maybe_unused]] float am_next = 0.f;
      if constexpr (FMT == kFmtNf4 && !AM) {
        am_row = p.absmax + ((size_t)n * p.K) / p.group_size;
        am_next = absmax_at(k0);
      }

      for (int k = ka; k < k1; k += kEvery) {
        const bool stage_free = mbar_test(empty + 8 * a.at, a.parity ^ 1u);
        const uint32_t slot_done = wempty + 8 * w.at;
        [[maybe_unused]] const uint32_t slot_now = w_ring + w.at * S::kWordBytes;
        bool words_ready = false;
        auto ask_words = [&] {  // those of the warp's next step, if it has one
          w.template skip<kEvery>();
          words_ready = --left > 0 && mbar_over(wfull + 8 * w.at, w.parity);
        };
        if (!S::kAlternate) ask_words();
        // the A stage must have been released by the tensor core
        if (!stage_free && !mbar_wait(empty + 8 * a.at, a.parity ^ 1u, ok)) ok = false;
        __syncwarp();
        tc_fence_after();  // orders the stores after the tensor core's reads of the stage
        // kPiece columns at a time: the stores of one piece are under way while the next is
        // unpacked, and no more than that many results are held
        constexpr int kPiece = 8;
        [[maybe_unused]] float am_now[2];  // of the halves that this warp unpacks
        if constexpr (FMT == kFmtNf4 && AM) {
          // four values of this row, two of them of step k
          const uint32_t pair = (uint32_t)(((col & 1) * (p.K / kBlockK) + 2 * k) & 2);
          const uint32_t at = slot_now + 16 * 1024 + (uint32_t)((col & 1) * 2048 + (col >> 1) * 16) + 4 * pair;
          if constexpr (S::kAlternate)
            asm volatile("ld.shared.v2.f32 {%0,%1}, [%2];" : "=f"(am_now[0]), "=f"(am_now[1]) : "r"(at));
          else
            asm volatile("ld.shared.f32 %0, [%1];" : "=f"(am_now[0]) : "r"(at + 4 * grp));
        } else if constexpr (FMT == kFmtNf4) {
          am_now[0] = am_next;
          if (k + 1 < k1) am_next = absmax_at(k + 1);
        }
#pragma unroll
        for (int hh = 0; hh < S::kHalves; hh++) {
          const uint32_t a_at = a_lane + a.at * (uint32_t)(4 * kAColumns) + (uint32_t)(hh * 2 * kAColumns);
          if (S::kAlternate && hh == 1) ask_words();
          if constexpr (FMT == kFmtQ3) {
            const uint32_t lo[3] = {nw[0], nw[1], nw[2]}, hi[3] = {nw[3], nw[4], nw[5]};
            // the streams shifted by four bits
            const uint32_t lo4[3] = {__funnelshift_r(lo[0], lo[1], 4), __funnelshift_r(lo[1], lo[2], 4), lo[2] >> 4};
            const uint32_t hi4[3] = {__funnelshift_r(hi[0], hi[1], 4), __funnelshift_r(hi[1], hi[2], 4), hi[2] >> 4};
            const __half2 sc2 = __half2half2(__ushort_as_half((unsigned short)nw[6]));
            const __half2 nz2 = __half2half2(__hneg(__ushort_as_half((unsigned short)nw[7])));
            const uint32_t lane4 = (uint32_t)lane * 4u;
            constexpr int kTab = kBase + S::kLut;
            if (hh + 1 < S::kHalves) read_words(hh + 1);
            uint32_t o[kPiece];
            q3_words<0, kTab>(lo, lo4, sc2, nz2, lane4, o);
            tmem_store(a_at, o);
            q3_words<8, kTab>(lo, lo4, sc2, nz2, lane4, o);
            tmem_store(a_at + 8, o);
            q3_words<0, kTab>(hi, hi4, sc2, nz2, lane4, o);
            tmem_store(a_at + 16, o);
            q3_words<8, kTab>(hi, hi4, sc2, nz2, lane4, o);
            tmem_store(a_at + 24, o);
          } else {
            const float am = am_now[hh];
            const uint32_t lane8 = (uint32_t)(lane & (S::kTabRow / 8 - 1)) * 8u;  // this lane's copy of a table row
            const bool past = !AM && (2 * k + (S::kAlternate ? hh : grp)) * kBlockK >= p.K;  // half a step past K: zero weights
            const uint32_t cw[8] = {nw[0], nw[1], nw[2], nw[3], nw[4], nw[5], nw[6], nw[7]};
            if (hh + 1 < S::kHalves) read_words(hh + 1);
#pragma unroll
            for (int q0 = 0; q0 < 8; q0 += kPiece / 4) {
              uint32_t o[kPiece];
#pragma unroll
              for (int q = 0; q < kPiece / 4; q++) {
#pragma unroll
                for (int t = 0; t < 4; t++) {
                  // byte t of the word is the table row
                  const uint32_t b = cw[q0 + q];
                  const uint32_t off = S::kTabRow == 256 ? __byte_perm(b, lane8, 0x7604u | (uint32_t)(t << 4))
                                                         : ((t == 0 ? b << 7 : b >> (8 * t - 7)) & 0x7f80u) | lane8;
                  float2 lv;
                  asm("ld.shared.v2.f32 {%0,%1}, [%2+%3];"
                      : "=f"(lv.x), "=f"(lv.y)
                      : "r"(off), "n"(kBase + S::kLut));
                  const float2 w2 = mul_f32x2(lv, am);
                  o[4 * q + t] = half2_as_u32(__floats2half2_rn(w2.x, w2.y));
                }
              }
              if (past) {
#pragma unroll
                for (int e = 0; e < kPiece; e++) o[e] = 0u;
              }
              tmem_store(a_at + 4 * q0, o);
            }
          }
        }
        __syncwarp();
        mbar_arrive_lane0(slot_done, lane);  // the words were consumed, so their loads have returned
        if (left > 0) take_words(words_ready);
        asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(full + 8 * a.at);
        a.template skip<kEvery>();
      }

      // ------------------------------ epilogue of the segment ------------------------------
      const bool whole = k0 == 0 && k1 == p.steps;
      if (!mbar_wait(done, segment & 1u, ok)) ok = false;
      segment++;
      __syncwarp();
      tc_fence_after();
      const uint32_t taddr = lanes + (uint32_t)(s * S::kTokens);
      const bool live = n < p.N;  // all or none of a warp: N is a multiple of 128
      // warps 0-7 take the even 16-token chunks, warps 8-15 the odd ones
      for (int j0 = grp * 16; j0 < p.tokens_padded; j0 += 32) {
        uint32_t v[16];
        asm volatile(
            "tcgen05.ld.sync.aligned.32x32b.x16.b32 "
            "{%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
            : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]),
              "=r"(v[7]), "=r"(v[8]), "=r"(v[9]), "=r"(v[10]), "=r"(v[11]), "=r"(v[12]), "=r"(v[13]),
              "=r"(v[14]), "=r"(v[15])
            : "r"(taddr + (uint32_t)j0));
        asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
        if (!live) continue;
        if (whole) {
#pragma unroll
          for (int j = 0; j < 16; j++)
            if (j0 + j < p.Mb) p.Y[(size_t)(j0 + j) * p.N + n] = __float2half_rn(__uint_as_float(v[j]));
        } else {
#pragma unroll
          for (int j = 0; j < 16; j++)
            if (j0 + j < p.Mb)
              asm volatile("red.global.add.f32 [%0], %1;" ::"l"(p.ws + (size_t)(j0 + j) * p.N + n),
                           "f"(__uint_as_float(v[j]))
                           : "memory");
        }
      }
      __syncwarp();
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(taken);

      if (!whole) {
        // the last part of the tile to arrive converts the scratch to fp16 and re-zeroes it
        __threadfence();
        asm volatile("bar.sync 1, 512;" ::: "memory");
        if (tid == 0) {
          const int parts = owner(p, (tile + 1) * p.steps - 1) - owner(p, tile * p.steps) + 1;
          const unsigned prev = atomicAdd(p.counters + tile, 1u);
          note[0] = prev == (unsigned)parts - 1u ? 1u : 0u;
        }
        asm volatile("bar.sync 1, 512;" ::: "memory");
        const bool last = note[0] != 0u;
        if (last) {
          __threadfence();
          // Mb x 64 groups of four features; four groups per thread and turn, all loads of
          // a turn issued before the first is used (one L2 round trip per turn)
          constexpr int kTurn = 4;
          const int groups = p.Mb * (kTileN / 4);
          for (int g0 = tid; g0 < groups; g0 += kUnpackWarps * 32 * kTurn) {
            float4 v[kTurn];
#pragma unroll
            for (int i = 0; i < kTurn; i++) {
              const int gi = g0 + i * kUnpackWarps * 32;
              const int j = gi / (kTileN / 4), c = tile * kTileN + (gi % (kTileN / 4)) * 4;
              if (gi < groups && c < p.N)
                v[i] = __ldcg(reinterpret_cast<const float4*>(p.ws + (size_t)j * p.N + c));
            }
#pragma unroll
            for (int i = 0; i < kTurn; i++) {
              const int gi = g0 + i * kUnpackWarps * 32;
              const int j = gi / (kTileN / 4), c = tile * kTileN + (gi % (kTileN / 4)) * 4;
              if (gi < groups && c < p.N) {
                const size_t at = (size_t)j * p.N + c;
                const __half2 lo = __floats2half2_rn(v[i].x, v[i].y), hi = __floats2half2_rn(v[i].z, v[i].w);
                const uint2 packed = make_uint2(half2_as_u32(lo), half2_as_u32(hi));
                if ((reinterpret_cast<uintptr_t>(p.Y + at) & 7u) == 0) {
                  *reinterpret_cast<uint2*>(p.Y + at) = packed;
                } else {
                  p.Y[at] = __low2half(lo); p.Y[at + 1] = __high2half(lo);
                  p.Y[at + 2] = __low2half(hi); p.Y[at + 3] = __high2half(hi);
                }
                *reinterpret_cast<float4*>(p.ws + at) = make_float4(0.f, 0.f, 0.f, 0.f);
              }
            }
          }
          if (tid == 0) p.counters[tile] = 0u;
        }
      }
    }
  } else if (warp == kIssueWarp) {
    // ------------------------------ MMA issuer ------------------------------
    // One warp for both subtiles, four MMAs (K = 16) per half and subtile: one wait and one
    // commit per step.
    // instruction descriptor: D fp32, A/B fp16, both K-major, N = tokens_padded, M = 128
    const uint32_t idesc = (1u << 4) | ((uint32_t)(p.tokens_padded >> 3) << 17) | ((uint32_t)(128 >> 4) << 24);
    Ring<S::kStages> a;
    uint32_t segment = 0;
    for (int u = u0; u < u1;) {
      const int tile = u / p.steps, k0 = u - tile * p.steps;
      const int k1 = min(p.steps, k0 + (u1 - u));
      u += k1 - k0;
      // the accumulators of the segment before must have been read
      if (segment != 0 && !mbar_wait(taken, (segment - 1u) & 1u, ok)) ok = false;
      segment++;
      uint32_t accumulate = 0;
      for (int k = k0; k < k1; k++) {
        if (!mbar_wait(full + 8 * a.at, a.parity, ok)) ok = false;
        __syncwarp();
        tc_fence_after();
        if (elect_one()) {
          const uint32_t a_tmem = S::kACol + a.at * (4 * kAColumns);
#pragma unroll
          for (int h = 0; h < 2; h++) {
            const uint64_t bdesc = smem_desc(x_ring + (2 * a.at + h) * S::kXHalf);
#pragma unroll
            for (int q = 0; q < kBlockK / 16; q++)
#pragma unroll
              for (int s = 0; s < 2; s++)
                umma_f16_ts(s * S::kTokens, a_tmem + (h * 2 + s) * kAColumns + 8 * q, bdesc + 2 * q, idesc,
                            h || q ? 1u : accumulate);
          }
          umma_commit(empty + 8 * a.at);
        }
        __syncwarp();
        accumulate = 1u;
        a.next();
      }
      // the commit covers the MMAs of the thread that executes it: elect.sync names
      // the same lane of the full warp every time
      if (elect_one()) {
        umma_commit(done);
        // sums in a fixed order: the epilogue starts when it is this part's turn as well
        if (p.ordered && !(k0 == 0 && k1 == p.steps))
          await_turn(p.counters + tile, (unsigned)(owner(p, (tile + 1) * p.steps - 1) - r));
        mbar_arrive(done);
      }
      __syncwarp();
    }
  } else if (warp == kIssueWarp + 1) {
    // ------------------------------ packed-word TMA ------------------------------
    Ring<S::kWordSlots> w;
    const uint32_t bytes = FMT == kFmtQ3 ? (p.one_group ? 12 * 1024 + 2 * 512 : 12 * 1024 + 4 * 512)
                                         : 16 * 1024 + (AM ? 4 * 1024 : 0);
    for (int u = u0; u < u1;) {
      const int tile = u / p.steps, k0 = u - tile * p.steps;
      const int k1 = min(p.steps, k0 + (u1 - u)), n0 = tile * kTileN;
      u += k1 - k0;
      for (int k = k0; k < k1; k++) {
        if (!mbar_wait(wempty + 8 * w.at, w.parity ^ 1u, ok)) ok = false;
        __syncwarp();
        if (elect_one()) {
          const uint32_t dst = w_ring + w.at * S::kWordBytes, bar = wfull + 8 * w.at;
          mbar_expect_tx(bar, bytes);
          if constexpr (FMT == kFmtQ3) {
            tma_load_2d(dst, &map_w, n0, 12 * k, bar);
            for (int h = 0; h < (p.one_group ? 1 : 2); h++) {
              const int g = (2 * k + h) * kBlockK / p.group_size;
              tma_load_2d(dst + 12 * 1024 + h * 512, &map_s, n0, g, bar);
              tma_load_2d(dst + 13 * 1024 + h * 512, &map_z, n0, g, bar);
            }
          } else {
            tma_load_2d(dst, &map_w, 64 * k, n0, bar);
            if constexpr (AM) {
              // map_s has two rows as one, which begins on 16 bytes: the aligned four values that hold
              // those of step k, for the 128 even rows of the tile and then for the odd ones
              tma_load_2d(dst + 16 * 1024, &map_s, (2 * k) & ~3, n0 / 2, bar);
              tma_load_2d(dst + 18 * 1024, &map_s, (p.K / kBlockK + 2 * k) & ~3, n0 / 2, bar);
            }
          }
        }
        __syncwarp();
        w.next();
      }
    }
  } else {
    // ------------------------------ X TMA ------------------------------
    Ring<S::kStages> x;
    const uint32_t bytes = (uint32_t)p.tokens_padded * 256u;
    int k = u0 % p.steps;
    for (int u = u0; u < u1; u++) {
      if (!mbar_wait(empty + 8 * x.at, x.parity ^ 1u, ok)) ok = false;
      __syncwarp();
      if (elect_one()) {
        const uint32_t bar = full + 8 * x.at, dst = x_ring + 2 * x.at * S::kXHalf;
        mbar_expect_tx(bar, bytes);
        tma_load_2d(dst, &map_x, 2 * k * kBlockK, 0, bar);
        tma_load_2d(dst + S::kXHalf, &map_x, (2 * k + 1) * kBlockK, 0, bar);
      }
      __syncwarp();
      x.next();
      if (++k == p.steps) k = 0;
    }
  }

  if ((!ok || tmem_base != 0u) && p.status != nullptr) atomicExch(p.status, 1);
  tc_fence_before();
  __syncthreads();
  if (warp == kIssueWarp) {
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(512u)
                 : "memory");
  }
}

template <int FMT, bool WIDE, bool AM>
int launch_shape(const CUtensorMap& map_x, const CUtensorMap& map_w, const CUtensorMap& map_s,
                 const CUtensorMap& map_z, const Params& prm, hq_stream_t stream) {
  constexpr auto kern = qgemm_stream_kernel<FMT, WIDE, AM>;
  constexpr size_t smem = Shape<FMT, WIDE, AM>::kSmem;
  cudaError_t e = ensure_dynamic_smem<kern>(smem);
  if (e != cudaSuccess) return cuda_status(e);
  return cuda_status(launch_pdl(kern, dim3(sm_count()), dim3(kThreads), smem, (cudaStream_t)stream, map_x,
                                map_w, map_s, map_z, prm));
}

template <int FMT>
int launch(const CUtensorMap& map_x, const CUtensorMap& map_w, const CUtensorMap& map_s,
           const CUtensorMap& map_z, const QgemmParams& q, bool ordered, bool am_tma, hq_stream_t stream) {
  Params prm;
  prm.Y = q.Y;
  prm.ws = q.ws;
  prm.counters = q.counters;
  prm.status = q.status;
  prm.Mb = q.Mb;
  prm.N = q.N;
  prm.K = q.K;
  prm.group_size = q.group_size;
  prm.tokens_padded = q.tokens_padded;
  prm.tiles = (q.N + kTileN - 1) / kTileN;
  prm.steps = (q.K + 2 * kBlockK - 1) / (2 * kBlockK);
  prm.ordered = ordered ? 1 : 0;
  prm.one_group = q.group_size % (2 * kBlockK) == 0 ? 1 : 0;
  prm.absmax = q.absmax;
  prm.lut16 = q.lut16;
  prm.low_first = q.low_first;
  prm.am_shift = -1;
  for (int i = 0; i < 25; i++)
    if (q.group_size == kBlockK << i) prm.am_shift = i;
  auto go = [&](auto am) {
    constexpr bool kAm = decltype(am)::value;
    return q.Mb > 64 ? launch_shape<FMT, true, kAm>(map_x, map_w, map_s, map_z, prm, stream)
                     : launch_shape<FMT, false, kAm>(map_x, map_w, map_s, map_z, prm, stream);
  };
  if constexpr (FMT == kFmtNf4)
    if (am_tma) return go(std::true_type());
  return go(std::false_type());
}

}  // namespace streamed
}  // namespace
}  // namespace hq
#endif  // HQ_QGEMM_STREAM_CUH_
