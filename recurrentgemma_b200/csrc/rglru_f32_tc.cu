// RG-LRU forward in float32 as ONE kernel: the block-diagonal gate projections, the gate arithmetic, the linear
// recurrence and the join with the other branch (recurrentgemma torch/layers.py:127-137, 313-365, 140-191; join of
// torch/modules.py:627-628, 646), heads of width 256.  a and the normalised input never reach memory.
//
// The contraction runs on the tensor cores as three products of float16 halves: with x scaled by a power of two
// of its token (over the 256 channels of the head) and w by one of its output channel, so that the largest
// magnitude lies in [2^14, 2^15),
//     x w  ~  x1 w1 + x2 w1 + x1 w2,      v1 = fp16(v),  v2 = fp16(v - v1)
// with float32 accumulation.  What is dropped is 2^-22 of a product, and 2^-39 of the row's largest factor where a
// factor is below 2^-17 of that; the scales are exact and undone in the epilogue.  As three TF32 products
// (gates_tf32.cu) the dropped part is up to 2^-20, an operand twice the bytes, and an instruction half as fast.
// TF32 keeps an exponent for each value, though, and halves under a common scale do not.  Where what they drop beyond
// 2^-22 could move the argument of any gate of the head by more than 2^-23, and by more than 2^-22 of the sum of its
// terms' magnitudes, the token's gates are float32 dot products on the CUDA cores instead (wide_tokens, exact_tokens).
// With N(0, 1/256) weights no token is looked at below a magnitude of some thousand, and normal data of any magnitude
// stay on the tensor cores: 2 x 1024 tokens of width 2560 33 us, 43 where all are looked at.  Where all are recomputed,
// one input channel 1e8 times the others and its weights as much smaller, they take 1.2 ms.
//
// Accumulators are channel-major, D[channel, token] = W[channel, k] . X[token, k]^T: a TMEM lane is a channel, its
// columns are tokens, and a thread walks its channel's tokens in time order.  A global access of a warp is one
// token of 32 consecutive channels: 128 contiguous bytes.
//
// Work: 128 tokens of one sequence x one head, as two units of 128 channels each that share the split activations;
// jobs are numbered time-major, for persistent CTAs, one per SM.  A last round that leaves half of the CTAs without a
// job goes as units.  A tile waits for the state of earlier ones, so no CTA may wait for one that work of other streams
// keeps off the device:
//   - the first round is dealt out by the CTAs' numbers.  Grids are placed in that order (what any look-back by block
//     number rests on), so a CTA waits for ones that have started;
//   - where there is more than a round, and tiles that wait (kDrawn), the rest is drawn by an atomic ticket, and only
//     once all CTAs have started: what a tile waits for was drawn before it, by a CTA that runs.  A CTA that finds some
//     missing for 20 us leaves when its job is done, which makes room; the last one to start finds none missing.
// All dealt out / drawn, us, inputs from memory: 2 x 1024 tokens 33.2 / 34.6, 5001 60.4 / 60.7 (coordinates that do not
// come from the CTA's number are in no uniform registers), 3 x 2000 of width 4096 99.1 / 96.5, with Conv1D and join 2 x
// 1024 48.7 / 48.8, 4 x 4000 302 / 280.  A cooperative launch of all dealt out: as that in a graph, 2 us more elsewhere.
//
// Roles in a CTA (24 warps, one or two of them idle):
//   tickets   one warp, if jobs are drawn: the next one as the tensor core begins the one before (with a join its last
//             unit: 3 x 2000 tokens of width 4096 169 -> 166 us, without 96.5 -> 98.1);
//   split     4 warps: the scale of each token (a pass over the head's 256 channels), then per K-slice of 64 the two
//             halves of the activations into the operand tiles (128-byte swizzle), as the tensor core releases them, and
//             ahead of the last slice's release the gates of tokens that are not left to the halves;
//   producer  one warp, an elected lane of which issues: packed weights, per K-slice and gate the two halves (128
//             rows x 64, 16 KiB each) by TMA through a ring of five;
//   MMA       one warp, an elected lane of which issues tcgen05.mma kind::f16 M128 N128 into one of two accumulator
//             sets (x-gate and a-gate columns, 2 x 128 each);
//   epilogue  two groups of 8 warps, a group an accumulator set, so that one's waits lie under the other's arithmetic;
//             8 warps = 4 channel quarters (TMEM lane quarters) x 2 token halves.  Pass one: gates, (a, x) of each
//             token back into the accumulator's own columns, the map (P, H): h -> P h + H of the thread's 64
//             tokens.  Then the state that enters the tile, by look-back over the maps of earlier tiles (records of
//             64-bit words {value, token}: no flags, no fences).  Pass two: the recurrence from tensor memory, join,
//             stores.
//
// What bounds it: an accumulator set belongs to the tensor core for 11,000 cycles (6,144 of instructions: operands,
// weights and halves share the shared memory's bandwidth) and then to its epilogue group for 18,000 (12,500 in pass one,
// 2,500 to 4,000 until the state is there, 3,500 in pass two), and there is room for two sets: 15,500 a unit.  67 warp
// instructions for 32 elements without a join, 54 % of the issue slots.  (Cycles and instructions before the warp's
// number was uniform, which took 5 to 7 % off the calls up to 5001 tokens.)  Width 2560, float32, us as gate and
// scan kernels with a and the normalised input through memory / this, in a loop: 2 x 1024 tokens 64 / 32, 5001 tokens
// 150 / 60, 8 x 4096 730 / 340, 16 tokens 19 / 11; with Conv1D and join 1500 tokens 64 / 35, 4 x 4000 458 / 281.  With one
// epilogue group of eight warps 2 x 1024 tokens took 42.  Distance of the 2-norm from a 64-bit evaluation: 9.5e-7 /
// 5.6e-7 at 2 x 1024 tokens, and the smaller one at every size and scale of normal data compared.
//
// All waits are bounded; on expiry WsHeader::status is raised, the affected values are taken as zero and the
// kernel runs to completion.
#include <cuda.h>
#include <cuda_fp16.h>
#include <limits.h>

#include "rgk_common.cuh"
#include "rgk_internal.h"
#include "tc_common.cuh"

namespace rgk {
namespace {

constexpr int kHW = 256;                 // head width = K
constexpr int kUT = 128;                 // tokens of a unit (MMA N)
constexpr int kUC = 128;                 // channels of a unit (MMA M)
constexpr int kKB = 64;                  // K of a slice: 128-byte rows of float16
constexpr int kKBlocks = kHW / kKB;
constexpr int kRing = 5;
constexpr int kXPart = kUT * kKB * 2;    // 16 KiB: one half of the activations of a slice
constexpr int kWPart = kUC * kKB * 2;    // 16 KiB: one half of one gate's weights of a slice
constexpr int kGroup = 8, kEpi = 2 * kGroup, kSplit = 4;
// Six warpgroups: four of epilogue warps, one of split warps, one of the producer, MMA and two idle warps, which
// hands registers to the split warps (loads in flight).  setmaxnreg.inc waits, without a limit, until the CTA has
// that many to give: no variant is launched that was compiled to fewer (set_attributes).
constexpr int kThreads = (kEpi + kSplit + 4) * 32;
constexpr int kRegsEpilogue = 80, kRegsSplit = 120, kRegsOther = 40;
constexpr bool registers_suffice(int per_thread) {
  return 6 * per_thread >= 4 * kRegsEpilogue + kRegsSplit + kRegsOther;
}
static_assert(kThreads == 6 * 128, "six warpgroups, four of them epilogue");
static_assert(registers_suffice(80) && !registers_suffice(79), "the hand-over takes all of 80 a thread");
constexpr int kTokHalf = kUT / 2;        // tokens of an epilogue thread
constexpr int kBarFirst = 9;             // named barrier behind the first job's activations (1-8: the epilogue's)
constexpr int kBatch = 8;                // tokens between two loads from tensor memory
constexpr int kOffX = 0;                                         // [slice][half]
constexpr int kOffRing = kOffX + kKBlocks * 2 * kXPart;
constexpr int kScaleBufs = 4;
constexpr int kOffScale = kOffRing + kRing * kWPart;             // float [job & 3][token]: 1 / scale, < 0: not trusted
constexpr int kOffWide = kOffScale + kScaleBufs * kUT * 4;       // bit [job & 3][token]: gates not left to the halves
constexpr int kOffMap = kOffWide + kScaleBufs * kUT / 8;         // float2 [group][channel]: map of the first half
constexpr int kDraws = 4;                                        // jobs between their draw and the last warp that reads it
constexpr int kDrawReaders = kEpi + kSplit + 2;                  // warps
constexpr int kOffBar = kOffMap + 2 * kUC * 8;  // ring full, empty; slice full, empty; sets full, empty; draw full, empty; go
constexpr int kNumBar = 2 * kRing + 2 * kKBlocks + 4 + 2 * kDraws + 1;
constexpr int kOffDraw = kOffBar + kNumBar * 8;
constexpr int kOffTmem = kOffDraw + kDraws * 4;
constexpr int kOffAbort = kOffTmem + 4;                          // two: the second of the waits for draws
constexpr int kSmem = kOffAbort + 8 + 1024;
static_assert(kSmem <= 232448, "exceeds the 227 KiB of shared memory a CTA may use");

// kind::f16, D float32, A and B float16, both K-major
constexpr uint32_t kIdesc = (1u << 4) | ((uint32_t)(kUT >> 3) << 17) | ((uint32_t)(kUC >> 4) << 24);

constexpr unsigned kLookbackSpins = 1u << 20;
constexpr int kStartPolls = 40;          // looks at how many CTAs have started, half a microsecond apart
constexpr int kLookback = 2;             // earlier tiles asked for per round trip (four: 8 x 4096 tokens 4 % slower)
constexpr unsigned long long kToken = 1ull << 32;

__device__ __forceinline__ unsigned long long ld_word(const unsigned long long* p) {
  unsigned long long v;
  asm volatile("ld.relaxed.gpu.global.u64 %0, [%1];" : "=l"(v) : "l"(p) : "memory");
  return v;
}
__device__ __forceinline__ void st_word(unsigned long long* p, float v) {
  asm volatile("st.relaxed.gpu.global.u64 [%0], %1;" :: "l"(p), "l"(kToken | (unsigned long long)__float_as_uint(v))
               : "memory");
}

// The power of two that brings a largest magnitude (its bits) into [2^14, 2^15), and its inverse, both normal.
// (Infinity and NaN: any power, the halves carry them on.)
__device__ __forceinline__ float scale_of(uint32_t max_bits) {
  const int e = max((int)(max_bits >> 23), 15);
  return __uint_as_float((uint32_t)(268 - e) << 23);
}
__device__ __forceinline__ float inverse_scale_of(uint32_t max_bits) {
  const int e = max((int)(max_bits >> 23), 15);
  return __uint_as_float((uint32_t)(e - 14) << 23);
}

// Two scaled values -> their float16 halves, packed.
__device__ __forceinline__ void split_pair(float v0, float v1, uint32_t& hi, uint32_t& lo) {
  const __half2 h = __floats2half2_rn(v0, v1);
  const float2 f = __half22float2(h);
  const __half2 l = __floats2half2_rn(v0 - f.x, v1 - f.y);
  hi = *reinterpret_cast<const uint32_t*>(&h);
  lo = *reinterpret_cast<const uint32_t*>(&l);
}

// Bits of the largest magnitude among the 256 values that a warp holds, 8 a lane.  (A value that is no number does
// not count: it reaches the products whatever the scale.)
__device__ __forceinline__ uint32_t largest(const float4& a, const float4& b) {
  const float m = fmaxf(fmaxf(fmaxf(fabsf(a.x), fabsf(a.y)), fmaxf(fabsf(a.z), fabsf(a.w))),
                        fmaxf(fmaxf(fabsf(b.x), fabsf(b.y)), fmaxf(fabsf(b.z), fabsf(b.w))));
  return __reduce_max_sync(0xffffffffu, __float_as_uint(m));
}

// How far the halves of activations and weights may move a gate's argument, beyond 2^-22 of its terms.
constexpr float kAllowed = 0x1p-23f;

// What the halves of a value under its row's scale drop, beyond 2^-22 of it.
__device__ __forceinline__ float dropped(float v) {
  const float hi = __half2float(__float2half_rn(v));
  const float rest = v - hi;
  return fmaxf(fabsf(rest - __half2float(__float2half_rn(rest))) - 0x1p-22f * fabsf(v), 0.0f);
}

// What the packing kernel says of 32 rows of weights, as bits.
struct WeightRange {
  uint32_t limit;                          // smallest over the rows: a token's largest magnitude up to which it is trusted
  uint32_t lost;                           // largest over the rows: sum of what the halves drop
  uint32_t largest;
  uint32_t pad;
};
constexpr int kRangesHead = 2 * 2 * kUC / 32;
// (from 2^113 on the products overflow before the scales are undone)
constexpr float kTopLimit = 0x1p100f;

// Which of the tokens in `tokens` (bit i: token i behind x0, of stride E) really lose too much, by themselves and against
// the least that |x| . |w| can be.  x0: the lane's first four values of the first token, the other four 128 behind;
// least: the smallest weight of each of these channels, by blocks of 32 rows.
__device__ __forceinline__ uint32_t wide_tokens(const float* x0, int E, uint32_t tokens, const WeightRange* range,
                                                const float* least, int lane) {
  const WeightRange r = range[lane & (kRangesHead - 1)];
  const float lost = __uint_as_float(__reduce_max_sync(0xffffffffu, r.lost));
  const float weight = __uint_as_float(__reduce_max_sync(0xffffffffu, r.largest));
  float4 m[2];
#pragma unroll
  for (int q = 0; q < 2; ++q) {
    m[q] = *reinterpret_cast<const float4*>(least + q * 128);
#pragma unroll 5
    for (int i = 1; i < kRangesHead; ++i) {
      const float4 v = *reinterpret_cast<const float4*>(least + i * kHW + q * 128);
      m[q] = make_float4(fminf(m[q].x, v.x), fminf(m[q].y, v.y), fminf(m[q].z, v.z), fminf(m[q].w, v.w));
    }
  }
  uint32_t wide = 0u;
#pragma unroll 1
  while (tokens != 0u) {
    int at[4];                                           // (the last one again where fewer are left)
    float moved[4], product[4], top[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      at[i] = tokens != 0u ? __ffs(tokens) - 1 : at[i > 0 ? i - 1 : 0];
      tokens &= tokens - 1u;
      const float* p = x0 + (int64_t)at[i] * E;
      const float4 v[2] = {*reinterpret_cast<const float4*>(p), *reinterpret_cast<const float4*>(p + 128)};
      const uint32_t t = largest(v[0], v[1]);
      const float s = scale_of(t);
      top[i] = __uint_as_float(t);
      moved[i] = product[i] = 0.0f;
#pragma unroll
      for (int q = 0; q < 2; ++q) {
        moved[i] += dropped(v[q].x * s) + dropped(v[q].y * s) + dropped(v[q].z * s) + dropped(v[q].w * s);
        product[i] += fabsf(v[q].x) * m[q].x + fabsf(v[q].y) * m[q].y + fabsf(v[q].z) * m[q].z + fabsf(v[q].w) * m[q].w;
      }
      moved[i] *= inverse_scale_of(t) * weight;
    }
#pragma unroll
    for (int j = 16; j > 0; j >>= 1)
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        moved[i] += __shfl_xor_sync(0xffffffffu, moved[i], j);
        product[i] += __shfl_xor_sync(0xffffffffu, product[i], j);
      }
#pragma unroll
    for (int i = 0; i < 4; ++i)
      if (!(fmaf(top[i], lost, moved[i]) <= fmaxf(kAllowed, 0x1p-22f * product[i])) || !(top[i] <= kTopLimit))
        wide |= 1u << at[i];
  }
  return wide;
}

__device__ __forceinline__ float2 fma2(const float2& a, const float2& b, const float2& c) {
  float2 d;
  asm("{\n\t.reg .b64 a, b, c;\n\t"
      "mov.b64 a, {%2, %3};\n\tmov.b64 b, {%4, %5};\n\tmov.b64 c, {%6, %7};\n\t"
      "fma.rn.f32x2 c, a, b, c;\n\t"
      "mov.b64 {%0, %1}, c;\n\t}"
      : "=f"(d.x), "=f"(d.y) : "f"(a.x), "f"(a.y), "f"(b.x), "f"(b.y), "f"(c.x), "f"(c.y));
  return d;
}

// The gates' arguments (without bias) of the tokens of `wide`, as float32 dot products with the weights as they are
// given, to zx and za (stride E as x; all three at token 0's values of the head).  A lane has eight channels of a gate at
// a time, four tokens share the weights' loads, and sums are added up by quarters, which rounds less.  (mine: of a head
// that two CTAs share, the lanes of each with its own channels write.)  A call, and with the roles in the order in
// which a short call needs their instructions: inlined between them 16 tokens with Conv1D took 15.0 us, not 13.9.
__device__ __noinline__ void exact_tokens(const float* x, int E, uint32_t wide, const float* wx, const float* wa,
                                          float* zx, float* za, bool mine, int lane) {
  constexpr int kTokens = 4, kQuarter = kHW / 4;
#pragma unroll 1
  while (wide != 0u) {
    int at[kTokens];
    const int n = __popc(wide);
#pragma unroll
    for (int i = 0; i < kTokens; ++i) {                  // (the last one again where fewer are left)
      at[i] = wide != 0u ? (__ffs(wide) - 1) * E : at[i > 0 ? i - 1 : 0];
      wide &= wide - 1u;
    }
#pragma unroll 1
    for (int pass = 0; pass < 8; ++pass) {               // gate, quarter
      const int k0 = (pass & 3) * kQuarter;
      const float* w = (pass < 4 ? wx : wa) + (int64_t)k0 * kHW + lane * 8;
      float* z = (pass < 4 ? zx : za) + lane * 8;
      float2 sum[kTokens][4];
#pragma unroll
      for (int i = 0; i < kTokens; ++i)
#pragma unroll
        for (int q = 0; q < 4; ++q) sum[i][q] = make_float2(0.0f, 0.0f);
#pragma unroll 1
      for (int k = 0; k < kQuarter; k += 32) {
        float v[kTokens];
#pragma unroll
        for (int i = 0; i < kTokens; ++i) v[i] = x[at[i] + k0 + k + lane];
#pragma unroll 4
        for (int kk = 0; kk < 32; ++kk) {
          const float4 w0 = *reinterpret_cast<const float4*>(w + (k + kk) * kHW);
          const float4 w1 = *reinterpret_cast<const float4*>(w + (k + kk) * kHW + 4);
#pragma unroll
          for (int i = 0; i < kTokens; ++i) {
            const float xv = __shfl_sync(0xffffffffu, v[i], kk);
            const float2 x2 = make_float2(xv, xv);
            sum[i][0] = fma2(x2, make_float2(w0.x, w0.y), sum[i][0]);
            sum[i][1] = fma2(x2, make_float2(w0.z, w0.w), sum[i][1]);
            sum[i][2] = fma2(x2, make_float2(w1.x, w1.y), sum[i][2]);
            sum[i][3] = fma2(x2, make_float2(w1.z, w1.w), sum[i][3]);
          }
        }
      }
#pragma unroll
      for (int i = 0; i < kTokens; ++i) {
        if (i >= n || !mine) break;
        float4* p = reinterpret_cast<float4*>(z + at[i]);
#pragma unroll
        for (int q = 0; q < 2; ++q) {
          float4 v = make_float4(sum[i][2 * q].x, sum[i][2 * q].y, sum[i][2 * q + 1].x, sum[i][2 * q + 1].y);
          if ((pass & 3) != 0) {
            const float4 before = p[q];
            v = make_float4(before.x + v.x, before.y + v.y, before.z + v.z, before.w + v.w);
          }
          p[q] = v;
        }
      }
    }
  }
}

// v / (s0 s1), powers of two whose product or quotients may be out of range.
__device__ __forceinline__ uint32_t unscaled(float v, float s0, float s1) {
  return __float_as_uint(scalbnf(v, -(ilogbf(s0) + ilogbf(s1))));
}

// These arguments of a channel per lane (zx, za: at token 0) into the accumulators, under the scales (token_scale, and
// the channel's two rows) that the epilogue undoes.  (A call, so that nothing of it is in the way of the other tokens.)
__device__ __noinline__ void place_tokens(const float* zx, const float* za, int E, uint32_t wide,
                                          const float* token_scale, float scale_x, float scale_a, uint32_t taddr) {
#pragma unroll 1
  while (wide != 0u) {
    int at[4];                                           // (the last one again where fewer are left)
    float vx[4], va[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      at[i] = wide != 0u ? __ffs(wide) - 1 : at[i > 0 ? i - 1 : 0];
      wide &= wide - 1u;
      vx[i] = zx[(int64_t)at[i] * E];
      va[i] = za[(int64_t)at[i] * E];
    }
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const float s = token_scale[at[i]];
      tc_st_32x1(taddr + at[i], unscaled(vx[i], s, scale_x));
      tc_st_32x1(taddr + kUT + at[i], unscaled(va[i], s, scale_a));
    }
  }
  tc_wait_st();
}

// gelu_tanh(z) = z sigmoid(2 u), u = sqrt(2 / pi) (z + 0.044715 z^3), on the hardware exponential and reciprocal: no
// cancellation at negative z, where 1 + tanh(u) has some, so nearer to a 64-bit evaluation than the float32 tanh.
__device__ __forceinline__ float gelu_f32(float z) {
  constexpr float k0 = -2.0f * 0.7978845608028654f * 1.4426950408889634f;
  const float w = z * fmaf(z * z, k0 * 0.044715f, k0);
  return z * rcpf(1.0f + ex2f(w));
}

// The jobs of a CTA: whole heads (two units) round-robin, then a unit of the last round where that was cut.
struct Jobs {
  int n_full, cut;                         // whole jobs of this CTA, its unit of the cut round (or -1)
  int per_tt, heads, first_cut;
  __device__ __forceinline__ Jobs(int n_jobs, int per_tt_, int heads_) : per_tt(per_tt_), heads(heads_) {
    const int grid = (int)gridDim.x, id = (int)blockIdx.x;
    const int rounds = n_jobs / grid, rest = n_jobs - rounds * grid;
    const bool cuts = 2 * rest <= grid;
    n_full = rounds + (!cuts && id < rest ? 1 : 0);
    first_cut = rounds * grid;
    cut = cuts && id < 2 * rest ? id : -1;
  }
  __device__ __forceinline__ int count() const { return n_full + (cut >= 0 ? 1 : 0); }
  // (time tile, sequence, head) of job j; its units are `half` .. `half` + n - 1
  __device__ __forceinline__ void get(int j, int& tt, int& b, int& head, int& half, int& n) const {
    int i;
    if (j < n_full) {
      i = (int)blockIdx.x + j * (int)gridDim.x;
      half = 0;
      n = 2;
    } else {
      i = first_cut + (cut >> 1);
      half = cut & 1;
      n = 1;
    }
    place(i, tt, b, head);
  }
  __device__ __forceinline__ void place(int i, int& tt, int& b, int& head) const {
    tt = i / per_tt;
    const int r = i - tt * per_tt;
    b = r / heads;
    head = r - b * heads;
  }
};

// The same jobs by ticket: whole heads, then the units of a last round that is cut.
struct Tickets {
  int n, n_whole;
  __device__ __forceinline__ explicit Tickets(int n_jobs) {
    const int grid = (int)gridDim.x, rest = n_jobs % grid;
    const bool cuts = 2 * rest <= grid;
    n_whole = cuts ? n_jobs - rest : n_jobs;
    n = cuts ? n_jobs + rest : n_jobs;
  }
  __device__ __forceinline__ void get(const Jobs& jobs, int ticket, int& tt, int& b, int& head, int& half,
                                      int& units) const {
    const int c = ticket - n_whole;
    half = c >= 0 ? c & 1 : 0;
    units = c >= 0 ? 1 : 2;
    jobs.place(c >= 0 ? n_whole + (c >> 1) : ticket, tt, b, head);
  }
};

// What the CTAs of a call share, cleared in front of it.
struct Shared {
  int started, drawn;
  int pad[2];
};

// The state entering tile tt of a chain, one channel per lane: composes the published maps of earlier tiles,
// nearest first, until a tile with a known state or the start of the sequence is met.
__device__ __forceinline__ float look_back(const unsigned long long* agg, const unsigned long long* incl, float hs,
                                           int64_t word, int tt, int64_t tile_words, bool* timed_out_p,
                                           int64_t n_words, int* status) {
  float Pc = 1.0f, Hc = 0.0f;
  int pred = tt - 1;
  unsigned spins = 0;
  *timed_out_p = false;
  while (pred >= 0) {
    unsigned long long wi[kLookback], wp[kLookback], wh[kLookback];
#pragma unroll
    for (int i = 0; i < kLookback; ++i) {
      wi[i] = 0ull; wp[i] = 0ull; wh[i] = 0ull;
      const int64_t w = word - (int64_t)(tt - pred + i) * tile_words;
      if (pred - i >= 0 && RGK_IN_RANGE(w, n_words, status)) {
        wi[i] = ld_word(incl + w);
        wp[i] = ld_word(agg + 2 * w);
        wh[i] = ld_word(agg + 2 * w + 1);
      }
    }
    const int before = pred;
#pragma unroll
    for (int i = 0; i < kLookback; ++i) {
      // entry i belongs to `pred` only while every entry in front of it was absorbed
      if (pred >= 0 && pred == before - i) {
        if ((wi[i] >> 32) == 1ull) return fmaf(Pc, __uint_as_float((uint32_t)wi[i]), Hc);
        if ((wp[i] >> 32) == 1ull && (wh[i] >> 32) == 1ull) {
          Hc = fmaf(Pc, __uint_as_float((uint32_t)wh[i]), Hc);
          Pc *= __uint_as_float((uint32_t)wp[i]);
          --pred;
        }
      }
    }
    if (pred == before) {
      if (++spins > kLookbackSpins) {
        *timed_out_p = true;
        return 0.0f;
      }
      __nanosleep(32);
    }
  }
  return fmaf(Pc, hs, Hc);
}

// kJoin 0: out = y, 1: out = y * gelu_tanh(yb)
template <int kJoin, bool kDrawn>
__global__ void __launch_bounds__(kThreads, 1)
rglru_f32_kernel(const __grid_constant__ CUtensorMap map_wh, const __grid_constant__ CUtensorMap map_wl,
                 const float* w_scale, const WeightRange* ranges, const float* least,
                 const float* wx, const float* wa, float* zx_wide, float* za_wide, const float* c, const void* pos,
                 int pos64, const float* __restrict__ a_param, const float* __restrict__ bias_x,
                 const float* __restrict__ bias_a, const float* h0, const float* yb, int B, int T_, int E, int heads,
                 int n_jobs, float* out, float* h_last, WsHeader* hdr, Shared* shared, unsigned long long* agg,
                 unsigned long long* incl) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = smem_raw + ((1024u - (smem_u32(smem_raw) & 1023u)) & 1023u);
  const uint32_t s_base = smem_u32(smem);
  const uint32_t bar0 = s_base + kOffBar;
  auto bar_w_full = [&](int s) { return bar0 + 8u * s; };
  auto bar_w_empty = [&](int s) { return bar0 + 8u * (kRing + s); };
  auto bar_x_full = [&](int kb) { return bar0 + 8u * (2 * kRing + kb); };
  auto bar_x_empty = [&](int kb) { return bar0 + 8u * (2 * kRing + kKBlocks + kb); };
  auto bar_acc_full = [&](int s) { return bar0 + 8u * (2 * kRing + 2 * kKBlocks + s); };
  auto bar_acc_empty = [&](int s) { return bar0 + 8u * (2 * kRing + 2 * kKBlocks + 2 + s); };
  auto bar_draw_full = [&](int s) { return bar0 + 8u * (2 * kRing + 2 * kKBlocks + 4 + s); };
  auto bar_draw_empty = [&](int s) { return bar0 + 8u * (2 * kRing + 2 * kKBlocks + 4 + kDraws + s); };
  const uint32_t bar_draw_go = bar0 + 8u * (2 * kRing + 2 * kKBlocks + 4 + 2 * kDraws);
  int* s_draw = reinterpret_cast<int*>(smem + kOffDraw);
  float* s_scale = reinterpret_cast<float*>(smem + kOffScale);
  uint32_t* s_wide = reinterpret_cast<uint32_t*>(smem + kOffWide);
  volatile uint32_t* s_tmem = reinterpret_cast<volatile uint32_t*>(smem + kOffTmem);
  volatile int* s_abort = reinterpret_cast<volatile int*>(smem + kOffAbort);

  // (from a lane, so that the compiler knows it to be the same in the whole warp: barriers, addresses and what the
  // loops run over are then in uniform registers: with the weights' loop on its whole warp 5 to 7 % off the calls of up to
  // 5001 tokens, nothing beyond their spread off 8 x 4096)
  const int warp = __shfl_sync(0xffffffffu, (int)threadIdx.x >> 5, 0), lane = threadIdx.x & 31;
  const int tiles_t = (T_ + kUT - 1) / kUT;
  const Jobs jobs(n_jobs, B * heads, heads);
  const int n_my = jobs.count();
  // whether there is a job j for this CTA, and which (for a warp of the roles that work on it)
  int ticket = (int)blockIdx.x;
  auto next = [&](int j) -> bool {
    if constexpr (!kDrawn) {
      return j < n_my;
    } else {
      if (j > 0) {
        const int s = (j - 1) & (kDraws - 1);
        const bool got = __all_sync(0xffffffffu, mbar_wait(bar_draw_full(s), ((j - 1) / kDraws) & 1, s_abort + 1));
        ticket = __shfl_sync(0xffffffffu, got ? s_draw[s] : INT_MAX, 0);
        if (lane == 0) mbar_arrive(bar_draw_empty(s));
      }
      return ticket < Tickets(n_jobs).n;
    }
  };
  auto get = [&](int j, int& tt, int& b, int& head, int& half, int& n) {
    if constexpr (kDrawn) Tickets(n_jobs).get(jobs, ticket, tt, b, head, half, n);
    else jobs.get(j, tt, b, head, half, n);
  };

  if (threadIdx.x == 0) {
    s_abort[0] = s_abort[1] = 0;
    for (int s = 0; s < kRing; ++s) { mbar_init(bar_w_full(s), 1); mbar_init(bar_w_empty(s), 1); }
    for (int kb = 0; kb < kKBlocks; ++kb) { mbar_init(bar_x_full(kb), kSplit); mbar_init(bar_x_empty(kb), 1); }
    for (int s = 0; s < 2; ++s) { mbar_init(bar_acc_full(s), 1); mbar_init(bar_acc_empty(s), kGroup); }
    if constexpr (kDrawn) {
      for (int s = 0; s < kDraws; ++s) { mbar_init(bar_draw_full(s), 1); mbar_init(bar_draw_empty(s), kDrawReaders); }
      mbar_init(bar_draw_go, 1);
    }
    mbar_fence_init();
  }
  if (warp == kEpi + kSplit + 1) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;"
                 :: "r"(s_base + kOffTmem), "r"(512) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *s_tmem;
  grid_dependency_wait();

  if (warp < kEpi) {
    // ------------------------------ epilogue --------------------------------------------------------
    const int chq = warp & 3, th = (warp >> 2) & 1, group = warp >> 3;
    const int64_t n_state = (int64_t)B * E;
    const int64_t n_words = (int64_t)tiles_t * B * E, tile_words = (int64_t)B * E;
    (void)n_state; (void)n_words;
    constexpr float kNegLog2e = -1.4426950408889634f;
    bool ok = true;
    // ---- the first job's activations, a warp eight tokens, read once: 4 us less until the first MMA than by the
    // split warps, which read them twice ----
    if (next(0)) {
      int tt, b, head, half, n;
      get(0, tt, b, head, half, n);
      const int w0 = warp * (kUT / kEpi), tok0 = tt * kUT + w0;
      const float* x0 = c + ((int64_t)b * T_ + tok0) * E + head * kHW + lane * 4;
      const WeightRange* range = ranges + head * kRangesHead;
      const uint32_t limits = range[lane & (kRangesHead - 1)].limit;
      uint32_t tops = 0u;                                // bits of the largest magnitude of token `lane`
#pragma unroll 1
      for (int i0 = 0; i0 < kUT / kEpi; i0 += 4) {
        float4 v[4][2];
#pragma unroll
        for (int i = 0; i < 4; ++i)
#pragma unroll
          for (int q = 0; q < 2; ++q)
            v[i][q] = tok0 + i0 + i < T_ ? *reinterpret_cast<const float4*>(x0 + (int64_t)(i0 + i) * E + q * 128)
                                         : make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          const uint32_t top = largest(v[i][0], v[i][1]);
          const float s = scale_of(top);
          const int row = w0 + i0 + i;
          if (lane == i0 + i) tops = top;
#pragma unroll
          for (int q = 0; q < 2; ++q) {
            uint2 hi, lo;
            split_pair(v[i][q].x * s, v[i][q].y * s, hi.x, lo.x);
            split_pair(v[i][q].z * s, v[i][q].w * s, hi.y, lo.y);
            const int k = q * 128 + lane * 4;            // the lane's first channel of the head
            uint8_t* at = smem + kOffX + (k >> 6) * 2 * kXPart + row * 128 +
                          ((((k & 63) >> 3) ^ (row & 7)) << 4) + (k & 4) * 2;
            *reinterpret_cast<uint2*>(at) = hi;
            *reinterpret_cast<uint2*>(at + kXPart) = lo;
          }
        }
      }
      fence_proxy_async();
      if (lane < kUT / kEpi) s_scale[w0 + lane] = inverse_scale_of(tops);
      const uint32_t limit = __reduce_min_sync(0xffffffffu, limits);
      const uint32_t wide = __ballot_sync(0xffffffffu, tops > limit && tok0 + lane < T_ && lane < kUT / kEpi);
      if (lane == 0) reinterpret_cast<uint8_t*>(s_wide)[warp] = (uint8_t)wide;
    }
    named_bar_sync(kBarFirst, (kEpi + kSplit) * 32);
    int t = 0;
    for (int j = 0; next(j); ++j) {
      int tt, b, head, half, n;
      get(j, tt, b, head, half, n);
      const int u = (t ^ group) & 1;                     // the group's unit of this job, if it has one
      const int tu = t + u;
      t += n;
      if (u >= n) continue;
      const int as = group;
      const int tok0 = tt * kUT + th * kTokHalf;
      const int live = T_ - tok0;                        // tokens of the thread inside the sequence
      // tokens that start a document, and tokens past the end of the sequence (the identity map)
      uint32_t rs[2], inv[2];
#pragma unroll
      for (int q = 0; q < 2; ++q) {
        const int k = q * 32 + lane;
        rs[q] = __ballot_sync(0xffffffffu, k < live && pos_is_zero(pos, pos64, (int64_t)b * T_ + tok0 + k));
        inv[q] = __ballot_sync(0xffffffffu, k >= live);
      }
      const float* st_row = s_scale + (j & (kScaleBufs - 1)) * kUT + th * kTokHalf;
      const int grp = head * 2 + half + u;
      const int e = grp * kUC + chq * 32 + lane;
      const int64_t at0 = ((int64_t)b * T_ + tok0) * E + e;
      // z log2(e) with the sign turned: the sigmoid is 1 / (1 + 2^that)
      const int wrow = grp * 2 * kUC + chq * 32 + lane;
      const float kx = kNegLog2e * w_scale[wrow], ka = kNegLog2e * w_scale[wrow + kUC];
      const float bx = kNegLog2e * bias_x[e], ba = kNegLog2e * bias_a[e];
      const float m8sp = -8.0f * softplus_(a_param[e]);
      const uint32_t t_row = tmem_base + (static_cast<uint32_t>(chq * 32) << 16) + as * 2 * kUT + th * kTokHalf;
      auto load_rows = [&](const float* src, int k0, float (&v)[kBatch], bool whole) {
        const float* p = src + at0 + (int64_t)k0 * E;
        if (whole) {
#pragma unroll
          for (int k = 0; k < kBatch; ++k) v[k] = p[(int64_t)k * E];
        } else {
#pragma unroll
          for (int k = 0; k < kBatch; ++k) v[k] = k0 + k < live ? p[(int64_t)k * E] : 0.0f;
        }
      };
      const bool whole = live >= kTokHalf;
      if constexpr (kJoin != 0) {                        // the other branch into L2: pass two has little to hide it under
#pragma unroll
        for (int q = 0; q < 2; ++q) {
          const int k = q * 32 + lane;
          if (k < live) asm volatile("prefetch.global.L2 [%0];" :: "l"(yb + (at0 - lane) + (int64_t)k * E));
        }
      }
      const int end = min(kTokHalf, live);               // batches past the end of the sequence are left out
      float P = 1.0f, H = 0.0f;
      {
        float cn[kBatch];
        load_rows(c, 0, cn, whole);
        if (ok) ok = mbar_wait(bar_acc_full(as), (tu >> 1) & 1, s_abort);
        __syncwarp();
        tc_fence_after();
        const uint2 wide = *reinterpret_cast<const uint2*>(s_wide + (j & (kScaleBufs - 1)) * (kUT / 32) + th * 2);
        if (__builtin_expect((wide.x | wide.y) != 0u, 0)) {
#pragma unroll 1
          for (int q = 0; q < 2; ++q)
            place_tokens(zx_wide + at0 + (int64_t)q * 32 * E, za_wide + at0 + (int64_t)q * 32 * E, E,
                         q == 0 ? wide.x : wide.y, st_row + q * 32, w_scale[wrow], w_scale[wrow + kUC], t_row + q * 32);
        }
#pragma unroll 1
        for (int k0 = 0; k0 < end; k0 += kBatch) {
          uint32_t zx[kBatch], za[kBatch];
          tc_ld_32x8(t_row + k0, zx);
          tc_ld_32x8(t_row + kUT + k0, za);
          float cv[kBatch], st[kBatch];
#pragma unroll
          for (int k = 0; k < kBatch; ++k) cv[k] = cn[k];
#pragma unroll
          for (int k = 0; k < kBatch; k += 4) {
            const float4 s4 = *reinterpret_cast<const float4*>(st_row + k0 + k);
            st[k] = s4.x; st[k + 1] = s4.y; st[k + 2] = s4.z; st[k + 3] = s4.w;
          }
          if (k0 + kBatch < end) load_rows(c, k0 + kBatch, cn, whole);
          const uint32_t rs8 = ((k0 < 32 ? rs[0] : rs[1]) >> (k0 & 31)) & 0xffu;
          const uint32_t inv8 = ((k0 < 32 ? inv[0] : inv[1]) >> (k0 & 31)) & 0xffu;
          tc_wait_ld();
#pragma unroll
          for (int k = 0; k < kBatch; ++k) {
            const float ex = ex2f(fmaf(__uint_as_float(zx[k]) * st[k], kx, bx));
            const float ea = ex2f(fmaf(__uint_as_float(za[k]) * st[k], ka, ba));
            const float gate_x = rcpf(1.0f + ex), gate_a = rcpf(1.0f + ea);
            // exp(log_a) on the accurate function: a slow channel multiplies a into its state a thousand times
            const float a = expf(gate_a * m8sp);
            cv[k] *= gate_x;
            zx[k] = __float_as_uint(cv[k] * sqrtf_approx(fmaf(-a, a, 1.0f)));
            za[k] = __float_as_uint(a);
          }
          if ((rs8 | inv8) != 0u) {
            // a token that starts a document: a = 0, multiplier = 1; one past the end: a = 1, x = 0
#pragma unroll
            for (int k = 0; k < kBatch; ++k) {
              if ((rs8 >> k) & 1u) { zx[k] = __float_as_uint(cv[k]); za[k] = 0u; }
              if ((inv8 >> k) & 1u) { zx[k] = 0u; za[k] = 0x3f800000u; }
            }
          }
#pragma unroll
          for (int k = 0; k < kBatch; ++k) {
            P *= __uint_as_float(za[k]);
            H = fmaf(__uint_as_float(za[k]), H, __uint_as_float(zx[k]));
          }
          tc_st_32x8(t_row + k0, zx);
          tc_st_32x8(t_row + kUT + k0, za);
        }
        tc_wait_st();
      }

      // ---- the state that enters the thread's tokens -----------------------------------------------
      // (in front of the barrier, and so of all records of the tile: h_last may be h0)
      const float hs = (h0 != nullptr && RGK_IN_RANGE((int64_t)b * E + e, n_state, &hdr->status))
                           ? h0[(int64_t)b * E + e] : 0.0f;
      float2* s_map = reinterpret_cast<float2*>(smem + kOffMap) + group * kUC + chq * 32 + lane;
      if (th == 0) *s_map = make_float2(P, H);
      named_bar_sync(1 + group * 4 + chq, 64);
      const float2 first = *s_map;
      const int64_t word = (int64_t)tt * tile_words + (int64_t)b * E + e;
      const bool owner = th == 1;
      const float Pt = P * first.x, Ht = fmaf(P, first.y, H);     // of the whole tile, in the second half's threads
      if (owner && tt > 0 && tt < tiles_t - 1 && RGK_IN_RANGE(word, n_words, &hdr->status)) {
        st_word(agg + 2 * word, Pt);
        st_word(agg + 2 * word + 1, Ht);
      }
      float yn[kBatch];
      if constexpr (kJoin != 0) load_rows(yb, 0, yn, whole);      // in flight during the look-back
      bool timed_out = !ok;
      float hin = 0.0f;
      if (ok) hin = look_back(agg, incl, hs, word, tt, tile_words, &timed_out, n_words, &hdr->status);
      __syncwarp();
      if (__any_sync(0xffffffffu, timed_out)) {
        if (lane == 0) atomicExch(&hdr->status, kStatusTimeout);
        hin = 0.0f;
      }
      if (owner && tt < tiles_t - 1 && RGK_IN_RANGE(word, n_words, &hdr->status))
        st_word(incl + word, fmaf(Pt, hin, Ht));
      float h = owner ? fmaf(first.x, hin, first.y) : hin;

      auto release = [&] {                                 // the set has been read: it may be written again
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(bar_acc_empty(as));
      };
      if (end <= 0) release();

      // ---- the recurrence, join, stores ------------------------------------------------------------
#pragma unroll 1
      for (int k0 = 0; k0 < end; k0 += kBatch) {
        uint32_t xn[kBatch], av[kBatch];
        tc_ld_32x8(t_row + k0, xn);
        tc_ld_32x8(t_row + kUT + k0, av);
        float yv[kBatch];
        if constexpr (kJoin != 0) {
#pragma unroll
          for (int k = 0; k < kBatch; ++k) yv[k] = gelu_f32(yn[k]);
          if (k0 + kBatch < end) load_rows(yb, k0 + kBatch, yn, whole);
        }
        tc_wait_ld();
        if (k0 + kBatch >= end) release();
#pragma unroll
        for (int k = 0; k < kBatch; ++k) {
          h = fmaf(__uint_as_float(av[k]), h, __uint_as_float(xn[k]));
          xn[k] = __float_as_uint(kJoin != 0 ? h * yv[k] : h);
        }
        float* o = out + at0 + (int64_t)k0 * E;
        if (whole) {
#pragma unroll
          for (int k = 0; k < kBatch; ++k) o[(int64_t)k * E] = __uint_as_float(xn[k]);
        } else {
#pragma unroll
          for (int k = 0; k < kBatch; ++k)
            if (k0 + k < live) o[(int64_t)k * E] = __uint_as_float(xn[k]);
        }
      }
      if (owner && h_last != nullptr && tt == tiles_t - 1 &&
          RGK_IN_RANGE((int64_t)b * E + e, n_state, &hdr->status))
        h_last[(int64_t)b * E + e] = h;
    }
  } else if (warp >= kEpi + kSplit) {
    asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" :: "n"(kRegsOther) : "memory");
    if (warp == kEpi + kSplit) {
    // ------------------------------ weights ---------------------------------------------------------
    // (the whole warp runs the loop, one elected lane issues: as the MMA warp)
    bool ok = true;
    int s = 0;
    uint32_t phase = 1;
    for (int j = 0; (kDrawn || ok) && next(j); ++j) {
      int tt, b, head, half, n;
      get(j, tt, b, head, half, n);
      for (int u = 0; u < n && ok; ++u) {
        const int row = (head * 2 + half + u) * 2 * kUC;
        for (int i = 0; i < kKBlocks * 4; ++i) {       // slice, gate, half
          ok = __all_sync(0xffffffffu, mbar_wait(bar_w_empty(s), phase, s_abort));
          if (!ok) break;
          if (elect_one()) {
            mbar_expect_tx(bar_w_full(s), kWPart);
            tma_load_2d(s_base + kOffRing + s * kWPart, (i & 1) ? &map_wl : &map_wh, (i >> 2) * kKB,
                        row + ((i >> 1) & 1) * kUC, bar_w_full(s));
          }
          __syncwarp();
          if (++s == kRing) { s = 0; phase ^= 1; }
        }
      }
    }
  } else if (warp == kEpi + kSplit + 1) {
    // ------------------------------ MMA issue -------------------------------------------------------
    // (the whole warp runs the loop, one elected lane issues: see mma_ring)
    const uint64_t desc_x = smem_desc_sw128(s_base + kOffX), desc_w = smem_desc_sw128(s_base + kOffRing);
    bool ok = true;
    int s = 0, t = 0;
    uint32_t phase = 0;
    for (int j = 0; (kDrawn || ok) && next(j); ++j) {
      int tt, b, head, half, n;
      get(j, tt, b, head, half, n);
      for (int u = 0; u < n && ok; ++u, ++t) {
        const int as = t & 1;
        ok = __all_sync(0xffffffffu, mbar_wait(bar_acc_empty(as), ((t >> 1) & 1) ^ 1, s_abort));
        if (!ok) break;
        if (kDrawn && u == (kJoin == 0 ? 0 : n - 1) && lane == 0) mbar_arrive(bar_draw_go);
        tc_fence_after();
        for (int kb = 0; kb < kKBlocks && ok; ++kb) {
          if (u == 0) {
            ok = __all_sync(0xffffffffu, mbar_wait(bar_x_full(kb), j & 1, s_abort));
            if (!ok) break;
          }
          const uint64_t x1 = desc_x + (uint64_t)(kb * (2 * kXPart >> 4)), x2 = x1 + (kXPart >> 4);
          for (int g = 0; g < 2 && ok; ++g) {
            const uint32_t d = tmem_base + (as * 2 + g) * kUT;
#pragma unroll
            for (int part = 0; part < 2; ++part) {
              ok = __all_sync(0xffffffffu, mbar_wait(bar_w_full(s), phase, s_abort));
              if (!ok) break;
              tc_fence_after();
              if (elect_one()) {
                const uint64_t w = desc_w + (uint64_t)(s * (kWPart >> 4));
#pragma unroll
                for (int ks = 0; ks < kKB / 16; ++ks) {
                  tc_mma_bf16(d, w + 2 * ks, x1 + 2 * ks, kIdesc, (part | kb | ks) != 0 ? 1u : 0u);
                  if (part == 0) tc_mma_bf16(d, w + 2 * ks, x2 + 2 * ks, kIdesc, 1u);
                }
                tc_commit(bar_w_empty(s));
                if (part == 1 && g == 1) {
                  if (u == n - 1) tc_commit(bar_x_empty(kb));
                  if (kb == kKBlocks - 1) tc_commit(bar_acc_full(as));
                }
              }
              __syncwarp();
              if (++s == kRing) { s = 0; phase ^= 1; }
            }
          }
        }
      }
    }
  } else if (kDrawn && warp == kEpi + kSplit + 2) {
    // ------------------------------ tickets ---------------------------------------------------------
    // (with an expired wait somewhere jobs are drawn all the same: the other roles go on without work, and the
    // epilogue publishes the records that other CTAs wait for)
    if (lane == 0) atomicAdd(&shared->started, 1);
    const Tickets tickets(n_jobs);
    const volatile int* started = &shared->started;
    bool all = false;
    int i = ticket;
    for (int j = 0; i < tickets.n; ++j) {
      const int s = j & (kDraws - 1);
      mbar_wait(bar_draw_go, j & 1, s_abort);
      const bool free = j < kDraws || mbar_wait(bar_draw_empty(s), ((j / kDraws) & 1) ^ 1, s_abort + 1);
      if (!__all_sync(0xffffffffu, free)) break;
      if (lane == 0) {
        if (!all) {
          for (int k = 0; !(all = *started == (int)gridDim.x) && k < kStartPolls; ++k) __nanosleep(500);
        }
        i = all ? (int)gridDim.x + atomicAdd(&shared->drawn, 1) : tickets.n;
        s_draw[s] = i;
        mbar_arrive(bar_draw_full(s));
      }
      i = __shfl_sync(0xffffffffu, i, 0);
    }
    }
  } else {
    asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" :: "n"(kRegsSplit) : "memory");
    // ------------------------------ activations: scales and halves ----------------------------------
    const int w0 = (warp - kEpi) * 32;                   // first of the warp's 32 tokens
    bool ok = true;
    // (the first job's activations are the epilogue warps' work, who have nothing else to do yet)
    named_bar_sync(kBarFirst, (kEpi + kSplit) * 32);
    const bool any = next(0);
    const uint32_t first_wide = any ? s_wide[w0 >> 5] : 0u;
    if (lane == 0 && any)
      for (int kb = 0; kb < kKBlocks - (first_wide != 0u ? 1 : 0); ++kb) mbar_arrive(bar_x_full(kb));
    for (int j = first_wide != 0u ? 0 : 1; (kDrawn || ok) && next(j); ++j) {
      if (kDrawn && !ok) continue;
      int tt, b, head, half, n;
      get(j, tt, b, head, half, n);
      const int tok0 = tt * kUT + w0;
      const int live = T_ - tok0;                        // tokens of the warp inside the sequence (may be < 1)
      const float* x0 = c + ((int64_t)b * T_ + tok0) * E + head * kHW;
      const WeightRange* range = ranges + head * kRangesHead;
      uint32_t* wide_at = s_wide + (j & (kScaleBufs - 1)) * (kUT / 32) + (w0 >> 5);
      uint32_t wide = first_wide;                        // tokens whose gates may not be left to the halves
      if (j > 0) {
        const uint32_t limits = range[lane & (kRangesHead - 1)].limit;
        uint32_t top = 0u;                               // bits of the largest magnitude of token `lane`
#pragma unroll 1
        for (int i0 = 0; i0 < 32; i0 += 8) {
          float4 v[8][2];
#pragma unroll
          for (int i = 0; i < 8; ++i)
#pragma unroll
            for (int q = 0; q < 2; ++q) {
              v[i][q] = make_float4(0.f, 0.f, 0.f, 0.f);
              if (i0 + i < live)
                v[i][q] = *reinterpret_cast<const float4*>(x0 + (int64_t)(i0 + i) * E + q * 128 + lane * 4);
            }
#pragma unroll
          for (int i = 0; i < 8; ++i) {
            const uint32_t all = largest(v[i][0], v[i][1]);
            if (lane == i0 + i) top = all;
          }
        }
        wide = __ballot_sync(0xffffffffu, top > __reduce_min_sync(0xffffffffu, limits) && lane < live);
        // (four buffers: the job whose scales were here has passed the epilogue.  Its last unit's accumulators
        // were read before the set could be written for the unit two behind, of a job at most two behind, whose
        // slices were released before this job's scales are looked for.)
        s_scale[(j & (kScaleBufs - 1)) * kUT + w0 + lane] = inverse_scale_of(top);
        const float factor = scale_of(top);
        const int r = lane >> 3, p = lane & 7;
#pragma unroll 1
        for (int kb = 0; kb < kKBlocks; ++kb) {
          float4 v[8][2];
#pragma unroll
          for (int i = 0; i < 8; ++i)
#pragma unroll
            for (int q = 0; q < 2; ++q) {
              v[i][q] = make_float4(0.f, 0.f, 0.f, 0.f);
              if (4 * i + r < live)
                v[i][q] = *reinterpret_cast<const float4*>(x0 + (int64_t)(4 * i + r) * E + kb * kKB + p * 8 + q * 4);
            }
          ok = mbar_wait(bar_x_empty(kb), (j & 1) ^ 1, s_abort);
          ok = __all_sync(0xffffffffu, ok);
          if (!ok) break;
          uint8_t* hi_tile = smem + kOffX + kb * 2 * kXPart;
#pragma unroll
          for (int i = 0; i < 8; ++i) {
            const int row = w0 + 4 * i + r;
            const float s = __shfl_sync(0xffffffffu, factor, 4 * i + r);
            uint4 hi, lo;
            split_pair(v[i][0].x * s, v[i][0].y * s, hi.x, lo.x);
            split_pair(v[i][0].z * s, v[i][0].w * s, hi.y, lo.y);
            split_pair(v[i][1].x * s, v[i][1].y * s, hi.z, lo.z);
            split_pair(v[i][1].z * s, v[i][1].w * s, hi.w, lo.w);
            const int at = row * 128 + ((p ^ (row & 7)) << 4);
            *reinterpret_cast<uint4*>(hi_tile + at) = hi;
            *reinterpret_cast<uint4*>(hi_tile + kXPart + at) = lo;
          }
          fence_proxy_async();                           // the tensor core reads this through the async proxy
          __syncwarp();
          if (lane == 0 && kb < kKBlocks - 1) mbar_arrive(bar_x_full(kb));
        }
        if (!ok) continue;
      }
      if (__builtin_expect(wide != 0u, 0)) {             // in front of the last slice, and so of the epilogue
        const int64_t col = (int64_t)head * kHW * kHW, row0 = ((int64_t)b * T_ + tok0) * E + head * kHW;
        wide = wide_tokens(x0 + lane * 4, E, wide, range, least + head * kRangesHead * kHW + lane * 4, lane);
        exact_tokens(x0, E, wide, wx + col, wa + col, zx_wide + row0, za_wide + row0, n == 2 || (lane >> 4) == half,
                     lane);
        __threadfence_block();
        __syncwarp();
      }
      if (lane == 0) {
        *wide_at = wide;
        mbar_arrive(bar_x_full(kKBlocks - 1));
      }
    }
  }

  tc_fence_before();
  __syncthreads();
  if (threadIdx.x == 0 && (s_abort[0] | (kDrawn ? s_abort[1] : 0)) != 0) atomicExch(&hdr->status, kStatusTimeout);
  if (warp == kEpi + kSplit + 1) {
    tc_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" :: "r"(tmem_base), "r"(512)
                 : "memory");
  }
}

// Gate weights [H, 256 (k), 256 (n)] float32 -> [H, 2, 256 (n'), 256 (k)] float16, first and second halves of the
// scaled values (rows 0-127 of a group: the x-gate columns of its 128 channels, rows 128-255 the a-gate ones),
// 1 / scale of each row, and of each 32 rows the range, and the smallest weight by input channel.
__global__ void pack_gate_weights_f16_kernel(const float* __restrict__ wx, const float* __restrict__ wa,
                                             __half* __restrict__ hi, __half* __restrict__ lo,
                                             float* __restrict__ scale, WeightRange* __restrict__ ranges,
                                             float* __restrict__ least) {
  __shared__ float tile[kHW][33];                                  // [k][n']
  __shared__ WeightRange range;
  if (threadIdx.x == 0) range = WeightRange{__float_as_uint(kTopLimit), 0u, 0u, 0u};
  const int group = blockIdx.y, head = group >> 1, half = group & 1;
  const int n0 = blockIdx.x * 32;                                  // n' in [0, 256)
  const float* src = (n0 < kUC ? wx : wa) + (int64_t)head * kHW * kHW + half * kUC + (n0 % kUC);
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  for (int k = warp; k < kHW; k += 8) tile[k][lane] = src[(int64_t)k * kHW + lane];
  __syncthreads();
  for (int r = warp; r < 32; r += 8) {
    uint32_t m = 0u;
#pragma unroll
    for (int i = 0; i < 8; ++i) m = max(m, __float_as_uint(tile[lane * 8 + i][r]) & 0x7fffffffu);
    m = __reduce_max_sync(0xffffffffu, m);
    const float s = scale_of(m);
    const int64_t row = (int64_t)group * 2 * kUC + n0 + r;
    float sum = 0.0f, lost = 0.0f;
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      sum += fabsf(tile[lane * 8 + i][r]);
      lost += dropped(tile[lane * 8 + i][r] * s);
    }
#pragma unroll
    for (int i = 16; i > 0; i >>= 1) {
      sum += __shfl_xor_sync(0xffffffffu, sum, i);
      lost += __shfl_xor_sync(0xffffffffu, lost, i);
    }
    uint32_t h[4], l[4];
#pragma unroll
    for (int i = 0; i < 4; ++i)
      split_pair(tile[lane * 8 + 2 * i][r] * s, tile[lane * 8 + 2 * i + 1][r] * s, h[i], l[i]);
    *reinterpret_cast<uint4*>(hi + row * kHW + lane * 8) = make_uint4(h[0], h[1], h[2], h[3]);
    *reinterpret_cast<uint4*>(lo + row * kHW + lane * 8) = make_uint4(l[0], l[1], l[2], l[3]);
    if (lane == 0) {
      scale[row] = inverse_scale_of(m);
      // (sum and m may be no number or infinite: no token is trusted)
      lost *= inverse_scale_of(m);
      const float limit = kAllowed / fmaf(0x1p-39f, sum, lost);
      atomicMin(&range.limit, limit > 0.0f ? __float_as_uint(limit) : 0u);
      atomicMax(&range.lost, __float_as_uint(lost));
      atomicMax(&range.largest, m);
    }
  }
  __syncthreads();
  if (threadIdx.x == 0) ranges[group * (2 * kUC / 32) + blockIdx.x] = range;
  float smallest = fabsf(tile[threadIdx.x][0]);
  for (int r = 1; r < 32; ++r) smallest = fminf(smallest, fabsf(tile[threadIdx.x][r]));
  least[(int64_t)(group * (2 * kUC / 32) + blockIdx.x) * kHW + threadIdx.x] = smallest;
}

// (early launch of the kernel behind only where no CTA has a second unit: its CTAs, placed as this one's leave, would sit
// on the SMs in another order, neighbours of a chain farther apart: 8 x 4096 tokens 327 -> 340 us)
__global__ void rglru_f32_prepare_kernel(const ChanPrep p) {
  if (p.early) grid_launch_dependents();
  grid_dependency_wait();
  chan_prepare(p, (int64_t)blockIdx.x * blockDim.x + threadIdx.x, (int64_t)gridDim.x * blockDim.x);
}

struct Layout {
  int64_t n_words;
  size_t shared_off, incl_off, agg_off, total;
};
Layout layout(int64_t B, int64_t T, int64_t E) {
  Layout L;
  L.n_words = (T + kUT - 1) / kUT * B * E;
  L.shared_off = sizeof(WsHeader);
  L.incl_off = L.shared_off + 256;                       // (whole lines of records for a warp)
  L.agg_off = L.incl_off + (size_t)L.n_words * 8;
  L.total = (L.agg_off + (size_t)L.n_words * 16 + 255) & ~(size_t)255;
  return L;
}

template <int kJoin, bool kDrawn>
cudaError_t set_attributes() {
  cudaFuncAttributes a;
  if (const cudaError_t e = cudaFuncGetAttributes(&a, rglru_f32_kernel<kJoin, kDrawn>); e != cudaSuccess) return e;
  if (!registers_suffice(a.numRegs)) return cudaErrorLaunchOutOfResources;
  return cudaFuncSetAttribute(rglru_f32_kernel<kJoin, kDrawn>, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmem);
}

cudaError_t device_setup(int* num_sms) {
  static PerDeviceOnce once;
  return once.run([] {
    cudaError_t e = set_attributes<0, false>();
    if (e == cudaSuccess) e = set_attributes<1, false>();
    if (e == cudaSuccess) e = set_attributes<0, true>();
    if (e == cudaSuccess) e = set_attributes<1, true>();
    return e;
  }, num_sms);
}

constexpr int64_t packed_rows(int H) { return (int64_t)H * 2 * 2 * kUC; }

}  // namespace

// Every sequence begins a tile of its own, where the kernels of gates_tf32.cu and scan.cu cut the tokens of all
// sequences into tiles together.  Width 2560, us those / this: 6 x 50 tokens 20.3 / 17.0, 64 x 50 95 / 73, 20 x 43
// 27.8 / 28.8; few jobs run at once however empty their tiles: 8 x 1 token 19.7 / 16.5, 8 x 16 20.8 / 17.6.  Of 110 sizes
// of 1 to 16 heads and 1 to 16000 tokens in 1 to 128 sequences the worst is 16 x 50 of 10 heads, 28.0 / 28.7.
bool rglru_f32_supported(int dtype, int bw, int64_t B, int64_t T, int H) {
  if (dtype != 0 || bw != kHW || B < 1 || T < 1) return false;
  const int64_t tiles = (T + kUT - 1) / kUT * B;
  return tiles < ((int64_t)1 << 17) && (5 * tiles * kUT <= 13 * B * T || tiles * H <= 128);
}

size_t rglru_f32_workspace_bytes(int64_t B, int64_t T, int64_t E) { return T < 1 ? 0 : layout(B, T, E).total; }

size_t rglru_f32_packed_bytes(int H) {
  return (size_t)packed_rows(H) * (kHW * 2 * 2 + 4) + (size_t)H * kRangesHead * (sizeof(WeightRange) + kHW * 4);
}

namespace {
struct Packed {
  __half *hi, *lo;
  float* scale;
  WeightRange* ranges;
  float* least;
  Packed(void* p, int H) {
    hi = static_cast<__half*>(p);
    lo = hi + packed_rows(H) * kHW;
    scale = reinterpret_cast<float*>(lo + packed_rows(H) * kHW);
    ranges = reinterpret_cast<WeightRange*>(scale + packed_rows(H));
    least = reinterpret_cast<float*>(ranges + H * kRangesHead);
  }
};
}  // namespace

cudaError_t launch_pack_gate_weights_f16(const void* wx, const void* wa, int H, void* packed_w, cudaStream_t s) {
  const Packed p(packed_w, H);
  pack_gate_weights_f16_kernel<<<dim3(2 * kUC / 32, 2 * H), 256, 0, s>>>(
      (const float*)wx, (const float*)wa, p.hi, p.lo, p.scale, p.ranges, p.least);
  return cudaGetLastError();
}

ChanPrep rglru_f32_prep(void* ws, int64_t B, int64_t T, int H) {
  const Layout L = layout(B, T, (int64_t)H * kHW);
  ChanPrep p;
  int num_sms = 0;
  if (device_setup(&num_sms) != cudaSuccess) return p;
  p.zero = reinterpret_cast<uint4*>(static_cast<char*>(ws) + L.shared_off);
  p.n_zero = (256 + L.n_words * 24) / 16;
  p.early = 2 * ((T + kUT - 1) / kUT * B * H) <= num_sms;
  return p;
}

cudaError_t launch_rglru_f32(const void* c, const void* pos, int pos64, const void* a_param, const void* wx,
                             const void* bx, const void* wa, const void* ba, const void* packed_w, const float* h0,
                             const void* yb, int64_t B, int64_t T, int H, float* zx, float* za, void* out,
                             float* h_last, void* ws, cudaStream_t s, bool prepared) {
  const int E = H * kHW;
  const Layout L = layout(B, T, E);
  int num_sms = 0;
  cudaError_t err = device_setup(&num_sms);
  if (err != cudaSuccess) return err;
  const int64_t n_jobs = (T + kUT - 1) / kUT * B * H;     // below 2^29
  if (!prepared) {
    const ChanPrep prep = rglru_f32_prep(ws, B, T, H);
    const int64_t blocks = (prep.n_zero + 1023) / 1024;
    err = launch_dependent(rglru_f32_prepare_kernel, dim3((unsigned)(blocks < 8 * num_sms ? blocks : 8 * num_sms)),
                           dim3(256), 0, s, prep);
    if (err != cudaSuccess) return err;
  }
  const Packed w(const_cast<void*>(packed_w), H);
  CUtensorMap map_wh, map_wl;
  if (!tensor_map_2d(&map_wh, w.hi, (uint64_t)packed_rows(H), kHW, kUC, kKB, true) ||
      !tensor_map_2d(&map_wl, w.lo, (uint64_t)packed_rows(H), kHW, kUC, kKB, true))
    return cudaErrorInvalidValue;
  // as many CTAs as SMs, or as there are units
  const int grid = 2 * n_jobs < num_sms ? (int)(2 * n_jobs) : num_sms;
  auto run = [&](auto kernel) {
    return launch_dependent(kernel, dim3(grid), dim3(kThreads), (size_t)kSmem, s, map_wh, map_wl, w.scale,
                            w.ranges, w.least, (const float*)wx, (const float*)wa, zx, za, (const float*)c, pos,
                            pos64, (const float*)a_param, (const float*)bx, (const float*)ba, h0,
                            (const float*)yb, (int)B, (int)T, E, H, (int)n_jobs, (float*)out, h_last,
                            reinterpret_cast<WsHeader*>(ws),
                            reinterpret_cast<Shared*>(static_cast<char*>(ws) + L.shared_off),
                            reinterpret_cast<unsigned long long*>(static_cast<char*>(ws) + L.agg_off),
                            reinterpret_cast<unsigned long long*>(static_cast<char*>(ws) + L.incl_off));
  };
  if (n_jobs > grid && T > kUT) return yb == nullptr ? run(rglru_f32_kernel<0, true>) : run(rglru_f32_kernel<1, true>);
  return yb == nullptr ? run(rglru_f32_kernel<0, false>) : run(rglru_f32_kernel<1, false>);
}

}  // namespace rgk
