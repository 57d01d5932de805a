// Local (sliding-window) multi-query attention of the attention residual blocks, prefill form
// (recurrentgemma torch/modules.py:399-493 with the helpers at 58-140), bfloat16, head dimension
// 256, one key/value head:
//   attn_prepare_kernel everything between the projections and the attention in one launch: rotary
//                       embedding of queries and keys in place (torch/modules.py:58-86), the ring
//                       cache a prompt leaves behind (torch/modules.py:238-258), per token the first
//                       visible key max(start of its document, t - window) (the mask of
//                       torch/modules.py:89-140 is "lo(t) <= s <= t": documents are contiguous, so
//                       "same segment" is "not before the start of mine"), and the values as
//                       [B,256,Tp], key index contiguous, zero padded: the second contraction then
//                       has a K-major B operand like the first;
//   attn_prefill_kernel the attention itself on tcgen05.
//
// The logits are rounded to bfloat16 as the reference rounds them; the softmax runs in float32 in one
// pass over the key tiles with a running reference m per row: P = 2^(s - m) rounded to bfloat16, O and
// the row sum l in float32, O / l at the end.  m follows the row's maximum only when a tile exceeds it
// by more than 2^8 (p and the sums stay far inside their ranges, and relative roundings do not depend
// on the reference), so that O is hardly ever rescaled.  An earlier version computed Q K^T twice to
// round the normalised probabilities: half again as many tensor instructions and twice the softmax
// work, 451 us for 4 x 4096 tokens, 10 heads, window 2048.
//
// A unit of work is (sequence, query head, 128 queries); units are dealt out round-robin to
// persistent CTAs, longest first.  Roles in a CTA (20 warps):
//   warps 0-15 softmax: group g = (warp / 4) % 2 takes the key tiles of parity g (its own S
//              accumulator); a thread owns a query row (TMEM lane quarter warp % 4) and the 64 keys
//              of column half warp / 8 of every tile of its group.  The reference of a row passes
//              from tile to tile through shared memory (bar_m), early in each tile's turn.  The
//              rounded probabilities go back into tensor memory over the logits (two bfloat16 per
//              32-bit column, the layout of an operand A held in tensor memory);
//   warp 16    TMA producer: the query tile once per unit (four slices of 64 of the head dimension)
//              and the key tiles as slices of 64 into a 5-slot ring;
//   warp 19    TMA producer of the transposed values (two 64-key slices per key tile);
//   warp 17    TMEM allocation and issue of S = Q K^T (M 128, N 128, 16 K-steps) into S[parity];
//   warp 18    issue of O += P V (M 128, N 256, 8 K-steps, A = P from tensor memory) once the
//              group has written P.  Two issuing warps, so that a P V never queues behind the
//              sixteen instructions of the next Q K^T; the Q K^T warp waits for the P V that read
//              P from S[parity] before it overwrites S[parity].
// TMEM: S[0], S[1] (128 columns each), O (256 columns).  All waits are bounded; on expiry the
// status word is raised and the CTA runs to its end.
#include <cuda.h>
#include <math.h>

#include "rgk_common.cuh"
#include "rgk_internal.h"
#include "tc_common.cuh"

namespace rgk {
namespace {

// ------------------------------------------------------------------------------------------------
// Rotary embedding: x [rows, heads, hd] in place, positions [rows].  The first half of a head is
// rotated in pairs (i, i + hd/4), the second half is left alone.
// ------------------------------------------------------------------------------------------------
template <typename T>
__global__ void rope_kernel(T* __restrict__ x, const void* __restrict__ pos, int pos64, int64_t rows,
                            int heads, int hd) {
  constexpr bool kBf16 = Traits<T>::kBf16;
  const int quarter = hd / 4;
  const int64_t idx = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  const int64_t total = rows * heads * quarter;
  if (idx >= total) return;
  const int i = (int)(idx % quarter);
  const int64_t rh = idx / quarter;            // row * heads + head
  const int64_t row = rh / heads;
  const float p = pos64 ? (float)reinterpret_cast<const long long*>(pos)[row]
                        : (float)reinterpret_cast<const int*>(pos)[row];
  const float exponent = 2.0f * (float)i / (float)(hd / 2);
  const float inv = 1.0f / powf(10000.0f, exponent);
  const float ang = p * inv;
  const float sn = rnd<kBf16>(sinf(ang)), cs = rnd<kBf16>(cosf(ang));
  T* h = x + rh * hd;
  const float a = (float)h[i], b = (float)h[i + quarter];
  const float o0 = rnd<kBf16>(rnd<kBf16>(a * cs) - rnd<kBf16>(b * sn));
  const float o1 = rnd<kBf16>(rnd<kBf16>(b * cs) + rnd<kBf16>(a * sn));
  h[i] = (T)o0;
  h[i + quarter] = (T)o1;
}

// Blocks by role: [0, B) the visible ranges (and token counts) of one sequence each; then blocks of 32
// tokens: rotary embedding, cache rows, transposed values.  A thread of the latter owns 8 of the 64
// rotated pairs of a row and walks the heads, so that sine and cosine are computed once per row and
// position and not once per head (a kernel with a thread per pair and head took 95 us for 16384 rows
// of 10 heads; the memory it touches, 20).
constexpr int kPrepRows = 32;
struct PrepArgs {
  __nv_bfloat16 *q, *k;
  const __nv_bfloat16* v;
  const void* pos;
  int pos64, B, T, Tp, N, window;
  int rotate;                            // 0: q and k are rotated already
  int* lo;
  __nv_bfloat16* vt;
  __nv_bfloat16 *cache_k, *cache_v;      // [B, window, 256], or NULL
  int* num_tokens;
};

__device__ __forceinline__ int pos_at(const PrepArgs& a, int64_t i) {
  return a.pos64 ? (int)reinterpret_cast<const long long*>(a.pos)[i] : reinterpret_cast<const int*>(a.pos)[i];
}

// bfloat16 pairs (a, b) of one register each, rotated with the reference's roundings
__device__ __forceinline__ void rotate2(uint32_t& a2, uint32_t& b2, uint32_t cs2, uint32_t sn2) {
  const uint32_t a = a2, b = b2;
  a2 = bsub2(bmul2(a, cs2), bmul2(b, sn2));
  b2 = badd2(bmul2(b, cs2), bmul2(a, sn2));
}

__global__ void __launch_bounds__(256) attn_prepare_kernel(const PrepArgs a) {
  __shared__ __align__(16) uint4 s_tile[kPrepRows * 33];      // a value row per 33 packs; also the scan's scratch
  const int tid = threadIdx.x;
  const int T_ = a.T;
  grid_dependency_wait();
  grid_launch_dependents();
  if ((int)blockIdx.x < a.B) {
    // ---- visible ranges: a thread scans a chunk for document starts, then a maximum over the chunks
    // in front (the first token starts a document whatever its position)
    int* s_last = reinterpret_cast<int*>(s_tile);
    const int b = blockIdx.x;
    const int64_t base = (int64_t)b * T_;
    const int chunk = (T_ + 255) / 256, t0 = tid * chunk, t1 = min(t0 + chunk, T_);
    int last = 0;
    for (int t = t0; t < t1; ++t)
      if (pos_is_zero(a.pos, a.pos64, base + t)) last = t;
    int incl = last;
    const int lane = tid & 31, warp = tid >> 5;
#pragma unroll
    for (int d = 1; d < 32; d *= 2) {
      const int o = __shfl_up_sync(0xffffffffu, incl, d);
      if (lane >= d) incl = max(incl, o);
    }
    if (lane == 31) s_last[warp] = incl;
    __syncthreads();
    int start = __shfl_up_sync(0xffffffffu, incl, 1);
    if (lane == 0) start = 0;
    for (int w = 0; w < warp; ++w) start = max(start, s_last[w]);
    for (int t = t0; t < t1; ++t) {
      if (pos_is_zero(a.pos, a.pos64, base + t)) start = t;
      a.lo[base + t] = max(start, t - a.window);
    }
    if (tid == 0 && a.num_tokens != nullptr) a.num_tokens[b] = pos_at(a, base + T_ - 1) + 1;
    return;
  }
  // a sequence's rows, and behind them the ring slots a short prompt leaves empty
  const int slots = min(a.window, T_);
  const int rows = a.cache_k != nullptr ? T_ + (a.window - slots) : T_;
  const int per_seq = (max(rows, a.Tp) - 1) / kPrepRows + 1;      // (a window of 2^31 - 1 does not overflow)
  const int blk = (int)blockIdx.x - a.B;
  const int b = blk / per_seq, t_base = (blk - b * per_seq) * kPrepRows;
  const int r = tid >> 3, part = tid & 7;
  const int t = t_base + r;
  const int64_t row = (int64_t)b * T_ + t;
  uint4 vv[4];
#pragma unroll
  for (int j = 0; j < 4; ++j) vv[j] = make_uint4(0u, 0u, 0u, 0u);
  if (t < T_) {
    uint4* kr = reinterpret_cast<uint4*>(a.k + row * 256);
    uint4 k0 = kr[part], k1 = kr[part + 8];
    const uint4* vr = reinterpret_cast<const uint4*>(a.v + row * 256);
#pragma unroll
    for (int j = 0; j < 4; ++j) vv[j] = vr[part + 8 * j];
    if (a.rotate) {
      const float p = a.pos64 ? (float)reinterpret_cast<const long long*>(a.pos)[row]
                              : (float)reinterpret_cast<const int*>(a.pos)[row];
      // five heads of the row at a time, the first ones on their way while sine and cosine are computed
      constexpr int kHeads = 5;
      uint4* qr = reinterpret_cast<uint4*>(a.q + row * a.N * 256);
      uint4 qa[kHeads], qb[kHeads];
      auto load_heads = [&](int h0) {
#pragma unroll
        for (int h = 0; h < kHeads; ++h) {
          if (h0 + h < a.N) {
            qa[h] = qr[(h0 + h) * 32 + part];
            qb[h] = qr[(h0 + h) * 32 + 8 + part];
          }
        }
      };
      load_heads(0);
      uint32_t cs[4], sn[4];
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        float c[2], s[2];
#pragma unroll
        for (int e = 0; e < 2; ++e) {
          const float exponent = 2.0f * (float)(part * 8 + j * 2 + e) / 128.0f;
          const float ang = p * (1.0f / powf(10000.0f, exponent));
          s[e] = sinf(ang);
          c[e] = cosf(ang);
        }
        cs[j] = pack_bf16x2(c[0], c[1]);
        sn[j] = pack_bf16x2(s[0], s[1]);
      }
      auto rotate = [&](uint4& x, uint4& y) {
        rotate2(x.x, y.x, cs[0], sn[0]);
        rotate2(x.y, y.y, cs[1], sn[1]);
        rotate2(x.z, y.z, cs[2], sn[2]);
        rotate2(x.w, y.w, cs[3], sn[3]);
      };
      for (int h0 = 0; h0 < a.N; h0 += kHeads) {
        if (h0 > 0) load_heads(h0);
#pragma unroll
        for (int h = 0; h < kHeads; ++h) {
          if (h0 + h < a.N) {
            rotate(qa[h], qb[h]);
            qr[(h0 + h) * 32 + part] = qa[h];
            qr[(h0 + h) * 32 + 8 + part] = qb[h];
          }
        }
      }
      rotate(k0, k1);
      kr[part] = k0;
      kr[part + 8] = k1;
    }
    const int u = t - (T_ - slots);              // place among the tokens the ring keeps
    if (a.cache_k != nullptr && u >= 0) {
      // the ring's slot: position modulo the window (rolled by the number of tokens)
      const int seen = pos_at(a, (int64_t)b * T_ + T_ - 1) + 1;
      int shift = seen % a.window;
      if (shift < 0) shift += a.window;
      const int slot = (int)(((int64_t)u + shift) % slots);
      uint4* ck = reinterpret_cast<uint4*>(a.cache_k + ((int64_t)b * a.window + slot) * 256);
      uint4* cv = reinterpret_cast<uint4*>(a.cache_v + ((int64_t)b * a.window + slot) * 256);
      ck[part] = k0;
      ck[part + 8] = k1;
      ck[part + 16] = kr[part + 16];
      ck[part + 24] = kr[part + 24];
#pragma unroll
      for (int j = 0; j < 4; ++j) cv[part + 8 * j] = vv[j];
    }
  } else if (t < rows) {
    const int64_t at = ((int64_t)b * a.window + slots + (t - T_)) * 256;
    uint4 *ck = reinterpret_cast<uint4*>(a.cache_k + at), *cv = reinterpret_cast<uint4*>(a.cache_v + at);
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      ck[part + 8 * j] = make_uint4(0u, 0u, 0u, 0u);
      cv[part + 8 * j] = make_uint4(0u, 0u, 0u, 0u);
    }
  }
  if (t_base >= a.Tp) return;
  // transposed values: a thread gathers one of the 256 dimensions over the block's 32 tokens
#pragma unroll
  for (int j = 0; j < 4; ++j) s_tile[r * 33 + part + 8 * j] = vv[j];
  __syncthreads();
  const uint16_t* col = reinterpret_cast<const uint16_t*>(s_tile) + tid;
  __nv_bfloat16* dst = a.vt + ((int64_t)b * 256 + tid) * a.Tp + t_base;
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    uint32_t w[4];
#pragma unroll
    for (int e = 0; e < 4; ++e)
      w[e] = col[(j * 8 + 2 * e) * 264] | ((uint32_t)col[(j * 8 + 2 * e + 1) * 264] << 16);
    if (t_base + j * 8 < a.Tp) *reinterpret_cast<uint4*>(dst + j * 8) = make_uint4(w[0], w[1], w[2], w[3]);
  }
}

// ------------------------------------------------------------------------------------------------
// The attention kernel.
// ------------------------------------------------------------------------------------------------
constexpr int kHd = 256;                  // head dimension = K of Q K^T, N of P V
constexpr int kTq = 128, kTk = 128;       // queries / keys per tile
constexpr int kSl = 64;                   // slice width (one 128-byte swizzle row of bfloat16)
constexpr int kSlice = kTq * kSl * 2;                // a [128 x 64] bfloat16 slice: 16 KiB
constexpr int kRingK = 5;                            // key slices in flight
constexpr int kVStage = kHd * kSl * 2;               // a 64-key slice of V^T: 32 KiB
constexpr int kOffQ = 0;                             // the query tile, four slices
constexpr int kOffK = (kHd / kSl) * kSlice;          //  65536
constexpr int kOffV = kOffK + kRingK * kSlice;       // 147456
// A row's maximum over the 64 keys of each thread [group][half][row]; its reference after the last tile
// of each parity [group][row]; its partial sums [unit parity][group, half][row].
constexpr int kOffMx = kOffV + 2 * kVStage;          // 212992
constexpr int kOffRef = kOffMx + 4 * kTq * 4;
constexpr int kOffSum = kOffRef + 2 * kTq * 4;
constexpr int kOffBarA = kOffSum + 8 * kTq * 4;
constexpr int kNumBarA = 2 + 2 * kRingK + 4 + 10 + 2; // q, key ring, v, s_full/s_empty/p_full/pv_done/m [2], o
constexpr int kOffTmemA = kOffBarA + kNumBarA * 8;
constexpr int kOffAbortA = kOffTmemA + 4;
constexpr int kSmemA = kOffAbortA + 4 + 1024;
static_assert(kSmemA <= 232448, "exceeds the 227 KiB of shared memory a CTA may use");
constexpr int kSoftWarps = 16;
constexpr int kThreadsA = (kSoftWarps + 4) * 32;
constexpr uint32_t kIdescS = tc_idesc_bf16(kTq, kTk);
constexpr uint32_t kIdescO = tc_idesc_bf16(kTq, kHd);
constexpr float kNegBig = -3.0e38f;
constexpr float kLogitScale = 0.0625f * 1.4426950408889634f;  // hd^-1/2 log2(e): exponent per logit unit
constexpr float kSlack = 8.0f / kLogitScale;         // logits a row may exceed its reference by: p <= 2^8

__global__ void __launch_bounds__(kThreadsA, 1)
attn_prefill_kernel(const __grid_constant__ CUtensorMap map_q, const __grid_constant__ CUtensorMap map_k,
                    const __grid_constant__ CUtensorMap map_vt, const int* lo_all, int B,
                    int T_, int N, int window, int n_units, __nv_bfloat16* __restrict__ out,
                    int* status) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = smem_raw + ((1024u - (smem_u32(smem_raw) & 1023u)) & 1023u);
  const uint32_t s_base = smem_u32(smem);
  const uint32_t bar0 = s_base + kOffBarA;
  const uint32_t bar_q_full = bar0, bar_q_empty = bar0 + 8u;
  auto bar_full = [&](int s) { return bar0 + 8u * (2 + s); };
  auto bar_empty = [&](int s) { return bar0 + 8u * (2 + kRingK + s); };
  auto bar_v_full = [&](int s) { return bar0 + 8u * (2 + 2 * kRingK + s); };
  auto bar_v_empty = [&](int s) { return bar0 + 8u * (2 + 2 * kRingK + 2 + s); };
  auto bar_s_full = [&](int g) { return bar0 + 8u * (2 + 2 * kRingK + 4 + g); };
  auto bar_s_empty = [&](int g) { return bar0 + 8u * (2 + 2 * kRingK + 6 + g); };
  auto bar_p_full = [&](int g) { return bar0 + 8u * (2 + 2 * kRingK + 8 + g); };
  auto bar_pv_done = [&](int g) { return bar0 + 8u * (2 + 2 * kRingK + 10 + g); };
  auto bar_m = [&](int g) { return bar0 + 8u * (2 + 2 * kRingK + 12 + g); };
  const uint32_t bar_o_full = bar0 + 8u * (2 + 2 * kRingK + 14);
  const uint32_t bar_o_empty = bar0 + 8u * (2 + 2 * kRingK + 15);
  volatile uint32_t* s_tmem = reinterpret_cast<volatile uint32_t*>(smem + kOffTmemA);
  volatile int* s_abort = reinterpret_cast<volatile int*>(smem + kOffAbortA);
  float* s_mx = reinterpret_cast<float*>(smem + kOffMx);
  float* s_ref = reinterpret_cast<float*>(smem + kOffRef);
  float* s_sum = reinterpret_cast<float*>(smem + kOffSum);

  // (from a lane, so that the compiler knows it to be the same in the whole warp and keeps barriers, addresses and loop
  // bounds in uniform registers: 698 -> 688 us a forward pass of the layer at 4 x 4096 tokens)
  const int warp = __shfl_sync(0xffffffffu, (int)threadIdx.x >> 5, 0), lane = threadIdx.x & 31;
  const int q_tiles = (T_ + kTq - 1) / kTq;
  // whole rounds, and whether this CTA has a unit in the last one
  const int rounds = n_units / (int)gridDim.x, rest = n_units - rounds * (int)gridDim.x;
  const int last = (rounds & 1) ? (int)gridDim.x - 1 - (int)blockIdx.x : (int)blockIdx.x;
  const int n_my = rounds + (last < rest ? 1 : 0);

  if (threadIdx.x == 0) {
    *s_abort = 0;
    mbar_init(bar_q_full, 1);
    mbar_init(bar_q_empty, 1);
    for (int s = 0; s < kRingK; ++s) { mbar_init(bar_full(s), 1); mbar_init(bar_empty(s), 1); }
    for (int s = 0; s < 2; ++s) {
      mbar_init(bar_v_full(s), 1); mbar_init(bar_v_empty(s), 1);
      mbar_init(bar_s_full(s), 1); mbar_init(bar_s_empty(s), 8);
      mbar_init(bar_p_full(s), 8);
      mbar_init(bar_pv_done(s), 1);
      mbar_init(bar_m(s), 8);
    }
    mbar_init(bar_o_full, 1);
    mbar_init(bar_o_empty, kSoftWarps);
    mbar_fence_init();
  }
  if (warp == kSoftWarps + 1) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;"
                 :: "r"(s_base + kOffTmemA), "r"(512) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *s_tmem;
  grid_dependency_wait();
  grid_launch_dependents();

  // unit -> (sequence, head, query tile); the key tiles it needs
  auto unit_of = [&](int i, int& b, int& n, int& t0, int& j_lo, int& j_hi) {
    // (back and forth over the CTAs, so that whoever took the longest of a round takes the shortest of
    // the next)
    const int u = i * gridDim.x + ((i & 1) ? gridDim.x - 1 - blockIdx.x : blockIdx.x);
    const int qt = q_tiles - 1 - u / (B * N), bn = u % (B * N);   // longest first
    n = bn % N;
    b = bn / N;
    t0 = qt * kTq;
    j_lo = max(0, t0 - window) / kTk;
    j_hi = min(t0 + kTq - 1, T_ - 1) / kTk;       // inclusive
  };

  if (warp == kSoftWarps) {
    // ------------------------------ TMA producer --------------------------------------------------
    // The whole warp runs the loop and waits; one elected lane issues.
    {
      int slot = 0;
      unsigned slot_phase = 1;
      bool ok = true;
      for (int i = 0; i < n_my && ok; ++i) {
        int b, n, t0, j_lo, j_hi;
        unit_of(i, b, n, t0, j_lo, j_hi);
        // the query tile, once the previous unit's last Q K^T has read the old one
        ok = mbar_wait(bar_q_empty, (i & 1) ^ 1, s_abort);
        if (!ok) break;
        if (elect_one()) {
          mbar_expect_tx(bar_q_full, (kHd / kSl) * kSlice);
#pragma unroll
          for (int ks = 0; ks < kHd / kSl; ++ks)
            tma_load_3d(s_base + kOffQ + ks * kSlice, &map_q, n * kHd + ks * kSl, t0, b, bar_q_full);
        }
        __syncwarp();
        for (int j = j_lo; j <= j_hi && ok; ++j) {
#pragma unroll
          for (int ks = 0; ks < kHd / kSl; ++ks) {
            if (ok) ok = mbar_wait(bar_empty(slot), slot_phase, s_abort);
            if (!ok) break;
            if (elect_one()) {
              mbar_expect_tx(bar_full(slot), kSlice);
              tma_load_3d(s_base + kOffK + slot * kSlice, &map_k, ks * kSl, j * kTk, b,
                          bar_full(slot));
            }
            __syncwarp();
            if (++slot == kRingK) { slot = 0; slot_phase ^= 1; }
          }
        }
      }
    }
  } else if (warp == kSoftWarps + 3) {
    // ------------------------------ TMA producer of V^T -------------------------------------------
    {
      unsigned iv = 0;
      bool ok = true;
      for (int i = 0; i < n_my && ok; ++i) {
        int b, n, t0, j_lo, j_hi;
        unit_of(i, b, n, t0, j_lo, j_hi);
        for (int j = j_lo; j <= j_hi && ok; ++j) {
#pragma unroll
          for (int c = 0; c < kTk / kSl; ++c, ++iv) {
            const int s = iv & 1;
            if (ok) ok = mbar_wait(bar_v_empty(s), ((iv >> 1) & 1) ^ 1, s_abort);
            if (!ok) break;
            if (elect_one()) {
              mbar_expect_tx(bar_v_full(s), kVStage);
              tma_load_3d(s_base + kOffV + s * kVStage, &map_vt, j * kTk + c * kSl, 0, b,
                          bar_v_full(s));
            }
            __syncwarp();
          }
        }
      }
    }
  } else if (warp == kSoftWarps + 1) {
    // ------------------------------ Q K^T issue ---------------------------------------------------
    // The whole warp runs the loop and waits; one elected lane issues.
    {
      int slot = 0;
      unsigned slot_phase = 0;
      unsigned s_use[2] = {0, 0};
      unsigned pv_issued[2] = {0, 0}, pv_seen[2] = {0, 0};   // P V on S[g]: scheduled / waited for
      bool ok = true;
      bool k_ready = false;      // the next key slice was already there when last asked
      auto issue_qk = [&](int g) {
        // S[g] = Q K^T for the next key tile in the ring, once the softmax warps have read the old
        // logits and every P V that takes its probabilities from S[g] has completed
        if (ok) ok = mbar_wait(bar_s_empty(g), (s_use[g] & 1) ^ 1, s_abort);
        ++s_use[g];
        while (ok && pv_seen[g] != pv_issued[g]) {
          ok = mbar_wait(bar_pv_done(g), pv_seen[g] & 1, s_abort);
          ++pv_seen[g];
        }
        tc_fence_after();
#pragma unroll
        for (int ks = 0; ks < kHd / kSl; ++ks) {
          // (every lane sees the same barrier state and abort flag, so `ok` stays warp-uniform)
          if (ok && !k_ready) ok = mbar_wait(bar_full(slot), slot_phase, s_abort);
          if (!ok) break;
          tc_fence_after();
          // a K step of 16 bfloat16 is 32 bytes = 2 units of the descriptor's start address
          const uint64_t dq = smem_desc_sw128(s_base + kOffQ + ks * kSlice);
          const uint64_t dk = smem_desc_sw128(s_base + kOffK + slot * kSlice);
          // ask about the slice after this one now; the answer is looked at after the issue
          const int slot_n = slot + 1 == kRingK ? 0 : slot + 1;
          k_ready = mbar_test(bar_full(slot_n), slot_n == 0 ? slot_phase ^ 1 : slot_phase);
          if (elect_one()) {
#pragma unroll
            for (int kk = 0; kk < kSl / 16; ++kk)
              tc_mma_bf16(tmem_base + g * kTk, dq + 2 * kk, dk + 2 * kk, kIdescS,
                          (ks | kk) != 0 ? 1u : 0u);
            tc_commit(bar_empty(slot));
          }
          __syncwarp();
          if (++slot == kRingK) { slot = 0; slot_phase ^= 1; }
        }
        if (ok && elect_one()) tc_commit(bar_s_full(g));
        __syncwarp();
      };
      for (int i = 0; i < n_my; ++i) {
        ok = __all_sync(0xffffffffu, ok);
        if (!ok) break;
        int b, n, t0, j_lo, j_hi;
        unit_of(i, b, n, t0, j_lo, j_hi);
        const int nt = j_hi - j_lo + 1;
        ok = mbar_wait(bar_q_full, i & 1, s_abort);
        // the other warp issues P V for tile j once its P is written
        for (int j = 0; j < nt && ok; ++j) {
          issue_qk(j & 1);
          ++pv_issued[j & 1];
        }
        if (ok && elect_one()) tc_commit(bar_q_empty);       // the unit's last Q K^T is in the pipe
        __syncwarp();
      }
    }
  } else if (warp == kSoftWarps + 2) {
    // ------------------------------ P V issue -----------------------------------------------------
    {
      unsigned iv = 0;
      unsigned p_use[2] = {0, 0};
      bool ok = true;
      for (int i = 0; i < n_my; ++i) {
        ok = __all_sync(0xffffffffu, ok);
        if (!ok) break;
        int b, n, t0, j_lo, j_hi;
        unit_of(i, b, n, t0, j_lo, j_hi);
        const int nt = j_hi - j_lo + 1;
        // the epilogue has read the previous unit's accumulator
        ok = mbar_wait(bar_o_empty, (i & 1) ^ 1, s_abort);
        tc_fence_after();
        for (int j = 0; j < nt && ok; ++j) {
          // O += P V for the key tile whose probabilities group g has just written over S[g]: the
          // keys of half c are the 32 columns from S[g] + 64 c, 8 columns per K step of 16
          const int g = j & 1;
          ok = mbar_wait(bar_p_full(g), p_use[g] & 1, s_abort);
          ++p_use[g];
          tc_fence_after();
#pragma unroll
          for (int c = 0; c < kTk / kSl; ++c, ++iv) {
            const int s = iv & 1;
            if (ok) ok = mbar_wait(bar_v_full(s), (iv >> 1) & 1, s_abort);
            if (!ok) break;
            tc_fence_after();
            const uint32_t p0 = tmem_base + g * kTk + c * 64;
            const uint64_t dv = smem_desc_sw128(s_base + kOffV + s * kVStage);
            if (elect_one()) {
#pragma unroll
              for (int kk = 0; kk < kSl / 16; ++kk)
                tc_mma_bf16_ts(tmem_base + 2 * kTk, p0 + kk * 8, dv + 2 * kk, kIdescO,
                               (j == 0 && c == 0 && kk == 0) ? 0u : 1u);
              tc_commit(bar_v_empty(s));
            }
            __syncwarp();
          }
          if (ok && elect_one()) tc_commit(bar_pv_done(g));
          __syncwarp();
        }
        if (ok && elect_one()) tc_commit(bar_o_full);
        __syncwarp();
      }
    }
  } else {
    // ------------------------------ softmax and epilogue ------------------------------------------
    const int g = (warp >> 2) & 1, quarter = warp & 3, chalf = warp >> 3;
    const int row = quarter * 32 + lane;                     // query row inside the tile = TMEM lane
    const uint32_t t_s = tmem_base + (static_cast<uint32_t>(quarter * 32) << 16) + g * kTk + chalf * 64;
    const uint32_t t_orow = tmem_base + (static_cast<uint32_t>(quarter * 32) << 16) + 2 * kTk;
    unsigned mine = 0, theirs = 0;             // tiles of this and of the other group in earlier units
    bool ok = true;
    for (int i = 0; i < n_my; ++i) {
      int b, n, t0, j_lo, j_hi;
      unit_of(i, b, n, t0, j_lo, j_hi);
      const int nt = j_hi - j_lo + 1;
      const int t = t0 + row;
      const bool row_ok = t < T_;
      // visible keys of this row: lo .. t (a row past the end sees key 0 only; it is never stored)
      const int lo = row_ok ? lo_all[(int64_t)b * T_ + t] : 0;
      const int hi = row_ok ? t : 0;
      float m = kNegBig, l = 0.0f;             // the reference l is relative to, this thread's part of l
      for (int j = g; j < nt; j += 2) {
        const unsigned k = mine + (j >> 1);    // which of this group's tiles
        if (ok) ok = mbar_wait(bar_s_full(g), k & 1, s_abort);
        __syncwarp();
        tc_fence_after();
        const int s0 = (j_lo + j) * kTk + chalf * 64;
        uint32_t v[32];                        // the 64 logits, rounded, in pairs
        uint32_t mx2 = 0xff80ff80u;
#pragma unroll
        for (int cc = 0; cc < 2; ++cc) {
          uint32_t acc[32];
          if (ok) {
            tc_ld_32x32(t_s + cc * 32, acc);
            tc_wait_ld();
          } else {
#pragma unroll
            for (int c = 0; c < 32; ++c) acc[c] = 0u;
          }
          const int sc = s0 + cc * 32;
#pragma unroll
          for (int c = 0; c < 16; ++c)
            v[cc * 16 + c] = pack_bf16x2(__uint_as_float(acc[2 * c]), __uint_as_float(acc[2 * c + 1]));
          if (!(sc >= lo && sc + 31 <= hi)) {  // some key is not visible: its logit is -inf
#pragma unroll
            for (int c = 0; c < 16; ++c) {
              const int key = sc + 2 * c;
              uint32_t& x = v[cc * 16 + c];
              if (!(key >= lo && key <= hi)) x = (x & 0xffff0000u) | 0xff80u;
              if (!(key + 1 >= lo && key + 1 <= hi)) x = (x & 0xffffu) | 0xff800000u;
            }
          }
#pragma unroll
          for (int c = 0; c < 16; ++c) mx2 = bmax2(mx2, v[cc * 16 + c]);
        }
        // the row's maximum over the tile, and its reference after the tile in front
        float tmax = fmaxf(bf16_lo(mx2), bf16_hi(mx2));
        s_mx[(g * 2 + chalf) * kTq + row] = tmax;
        named_bar_sync(2 + g, 256);
        tmax = fmaxf(tmax, s_mx[(g * 2 + (chalf ^ 1)) * kTq + row]);
        float before = kNegBig;
        if (j > 0) {
          if (ok) ok = mbar_wait(bar_m(g ^ 1), (theirs + ((j - 1) >> 1)) & 1, s_abort);
          __syncwarp();
          before = s_ref[(g ^ 1) * kTq + row];
        }
        // (a row without a visible key so far has no reference: -inf is below kNegBig)
        const float ref = tmax > before + (before > kNegBig ? kSlack : 0.0f) ? tmax : before;
        if (chalf == 0) s_ref[g * kTq + row] = ref;
        __syncwarp();
        if (lane == 0) mbar_arrive(bar_m(g));
        if (__any_sync(0xffffffffu, ref > before && before > kNegBig)) {
          // rare: O follows, once the tile in front has been added
          if (ok) ok = mbar_wait(bar_pv_done(g ^ 1), (theirs + ((j - 1) >> 1)) & 1, s_abort);
          __syncwarp();
          tc_fence_after();
          const float f = before > kNegBig ? ex2f(fmaxf((before - ref) * kLogitScale, -200.0f)) : 1.0f;
          if (ok) {
#pragma unroll 1
            for (int cc = 0; cc < 8; ++cc) {
              uint32_t acc[16];
              tc_ld_32x16(t_orow + chalf * 128 + cc * 16, acc);
              tc_wait_ld();
#pragma unroll
              for (int c = 0; c < 16; ++c) acc[c] = __float_as_uint(__uint_as_float(acc[c]) * f);
              tc_st_32x16(t_orow + chalf * 128 + cc * 16, acc);
            }
            tc_wait_st();
          }
        }
        if (ref != m) {
          l *= ex2f(fmaxf((m - ref) * kLogitScale, -200.0f));
          m = ref;
        }
        const float off = -ref * kLogitScale;
        float add[4] = {0.0f, 0.0f, 0.0f, 0.0f};
#pragma unroll
        for (int cc = 0; cc < 2; ++cc) {
          uint32_t pk[16];
#pragma unroll
          for (int c = 0; c < 16; ++c) {
            const uint32_t x = v[cc * 16 + c];
            const float p0 = ex2f(fmaf(bf16_lo(x), kLogitScale, off)), p1 = ex2f(fmaf(bf16_hi(x), kLogitScale, off));
            add[(2 * c) & 3] += p0;
            add[(2 * c + 1) & 3] += p1;
            pk[c] = pack_bf16x2(p0, p1);
          }
          // 32 keys = 16 columns, over logits this thread has already read
          if (ok) tc_st_32x16(t_s + cc * 16, pk);
        }
        l += (add[0] + add[1]) + (add[2] + add[3]);
        tc_wait_st();
        tc_fence_before();
        __syncwarp();
        if (lane == 0 && ok) {
          mbar_arrive(bar_s_empty(g));
          mbar_arrive(bar_p_full(g));
        }
      }
      mine += (unsigned)((nt + 1 - g) >> 1);
      theirs += (unsigned)((nt + g) >> 1);

      // ---- the four partial sums of a row, and O / l -> bfloat16 -> encoded [B, T, N * 256]: a thread
      // takes 64 columns.  The sums alternate between two places, so one barrier a unit is enough.
      float* sums = s_sum + (i & 1) * 4 * kTq;
      float last = m;
      if (g != ((nt - 1) & 1)) {
        // the other group took the last tile: its reference is the final one
        if (ok) ok = mbar_wait(bar_m(g ^ 1), (theirs - 1) & 1, s_abort);
        __syncwarp();
        last = s_ref[(g ^ 1) * kTq + row];
      }
      sums[(g * 2 + chalf) * kTq + row] = l * ex2f(fmaxf((m - last) * kLogitScale, -200.0f));
      named_bar_sync(1, kSoftWarps * 32);
      const float sum = (sums[row] + sums[kTq + row]) + (sums[2 * kTq + row] + sums[3 * kTq + row]);
      const float inv = 1.0f / sum;
      if (ok) ok = mbar_wait(bar_o_full, i & 1, s_abort);
      __syncwarp();
      tc_fence_after();
      const int c0 = (g * 2 + chalf) * 64;
      __nv_bfloat16* orow = out + ((int64_t)b * T_ + t) * ((int64_t)N * kHd) + (int64_t)n * kHd + c0;
#pragma unroll
      for (int cc = 0; cc < 2; ++cc) {
        uint32_t acc[32];
        if (ok) {
          tc_ld_32x32(t_orow + c0 + cc * 32, acc);
          tc_wait_ld();
        } else {
#pragma unroll
          for (int c = 0; c < 32; ++c) acc[c] = 0u;
        }
        if (cc == 1) {
          tc_fence_before();
          __syncwarp();
          if (lane == 0 && ok) mbar_arrive(bar_o_empty);
        }
        if (row_ok) {
#pragma unroll
          for (int u4 = 0; u4 < 4; ++u4) {
            uint32_t o[4];
#pragma unroll
            for (int e = 0; e < 4; ++e)
              o[e] = pack_bf16x2(__uint_as_float(acc[8 * u4 + 2 * e]) * inv,
                                 __uint_as_float(acc[8 * u4 + 2 * e + 1]) * inv);
            *reinterpret_cast<uint4*>(orow + cc * 32 + u4 * 8) = make_uint4(o[0], o[1], o[2], o[3]);
          }
        }
      }
    }
  }

  tc_fence_before();
  __syncthreads();
  if (threadIdx.x == 0 && *s_abort && status != nullptr) atomicExch(status, kStatusTimeout);
  if (warp == kSoftWarps + 1) {
    tc_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" :: "r"(tmem_base), "r"(512)
                 : "memory");
  }
}

}  // namespace

cudaError_t launch_rope(void* x, const void* pos, int pos64, int64_t rows, int heads, int hd,
                        int dtype, cudaStream_t s) {
  const int64_t total = rows * heads * (hd / 4);
  if (total == 0) return cudaSuccess;
  const unsigned grid = (unsigned)((total + 255) / 256);
  if (dtype)
    rope_kernel<__nv_bfloat16><<<grid, 256, 0, s>>>((__nv_bfloat16*)x, pos, pos64, rows, heads, hd);
  else
    rope_kernel<float><<<grid, 256, 0, s>>>((float*)x, pos, pos64, rows, heads, hd);
  return cudaGetLastError();
}

size_t attention_workspace_bytes(int64_t B, int64_t T) {
  auto up = [](size_t v) { return (v + 255) & ~(size_t)255; };
  const int64_t Tp = (T + 7) / 8 * 8;
  return 256 + up((size_t)B * T * sizeof(int)) + up((size_t)B * kHd * Tp * 2);
}

bool attention_supported(int dtype, int hd, int64_t B, int64_t T, int N) {
  return dtype == 1 && hd == kHd && B >= 1 && T >= 1 && N >= 1 && T < ((int64_t)1 << 30) &&
         B * N * ((T + kTq - 1) / kTq) < ((int64_t)1 << 31);
}

// q [B,T,N,256] and k [B,T,256], rotated in place first if `rotate`, v [B,T,256]; out [B,T,N*256] may be q (a unit reads
// the queries it will overwrite before it writes).  cache_k, cache_v, num_tokens: the ring cache of
// the prompt, or NULL.
cudaError_t launch_attention_prefill(void* q, void* k, const void* v, const void* pos, int pos64, int64_t B,
                                     int64_t T, int N, int window, bool rotate, void* cache_k,
                                     void* cache_v, int* num_tokens, void* out, void* ws, cudaStream_t s) {
  using T_ = __nv_bfloat16;
  auto up = [](size_t x) { return (x + 255) & ~(size_t)255; };
  const int64_t Tp = (T + 7) / 8 * 8;
  char* base = static_cast<char*>(ws);
  int* status = reinterpret_cast<int*>(base);
  int* lo = reinterpret_cast<int*>(base + 256);
  T_* vt = reinterpret_cast<T_*>(base + 256 + up((size_t)B * T * sizeof(int)));
  PrepArgs a = {};
  a.q = static_cast<T_*>(q);
  a.k = static_cast<T_*>(k);
  a.v = static_cast<const T_*>(v);
  a.pos = pos;
  a.pos64 = pos64;
  a.B = (int)B;
  a.T = (int)T;
  a.Tp = (int)Tp;
  a.N = N;
  a.window = window;
  a.rotate = rotate ? 1 : 0;
  a.lo = lo;
  a.vt = vt;
  a.cache_k = static_cast<T_*>(cache_k);
  a.cache_v = static_cast<T_*>(cache_v);
  a.num_tokens = num_tokens;
  int64_t rows = Tp;
  if (cache_k != nullptr && T < window) rows = rows > window ? rows : window;
  const int64_t blocks = B + B * ((rows + kPrepRows - 1) / kPrepRows);
  if (blocks > 0x7fffffff) return cudaErrorInvalidValue;
  cudaError_t err = launch_dependent(attn_prepare_kernel, dim3((unsigned)blocks), dim3(256), 0, s, a);
  if (err != cudaSuccess) return err;
  CUtensorMap map_q, map_k, map_vt;
  if (!tensor_map_bte(&map_q, q, (uint64_t)B, (uint64_t)T, (uint64_t)N * kHd, kTq, kSl, true) ||
      !tensor_map_bte(&map_k, k, (uint64_t)B, (uint64_t)T, kHd, kTk, kSl, true) ||
      !tensor_map_bte(&map_vt, vt, (uint64_t)B, kHd, (uint64_t)Tp, kHd, kSl, true))
    return cudaErrorInvalidValue;
  static PerDeviceOnce once;
  int num_sms = 0;
  cudaError_t e0 = once.run([] {
    return cudaFuncSetAttribute(attn_prefill_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmemA);
  }, &num_sms);
  if (e0 != cudaSuccess) return e0;
  const int q_tiles = (int)((T + kTq - 1) / kTq);
  const int n_units = (int)(B * N * q_tiles);
  const int grid = n_units < num_sms ? n_units : num_sms;
  return launch_dependent(attn_prefill_kernel, dim3(grid), dim3(kThreadsA), kSmemA, s, map_q, map_k, map_vt, lo,
                          (int)B, (int)T, N, window, n_units, (T_*)out, status);
}

}  // namespace rgk
