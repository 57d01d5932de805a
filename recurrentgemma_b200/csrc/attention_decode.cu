// Local attention for one new token per sequence against the ring-buffer cache
// (recurrentgemma torch/modules.py:437-476 with the cache branch, the mask of
// torch/modules.py:155-184 and the ring update of torch/modules.py:187-286), head dimension 256,
// one key/value head:
// bfloat16: one kernel for the whole step (attn_decode_ring_kernel below).
// float32, on the CUDA cores, bandwidth work on the ring with 16 CTAs per sequence and the loads of a
// whole batch of rows in flight per warp (~200 instructions per row are what bounds it):
//   attn_decode_logits_kernel    logits of the N query heads against the W ring entries and the
//                                new key, scaled by head_dim^-1/2; per CTA the softmax statistics;
//   attn_decode_values_kernel    probabilities times the ring's values and the new value, a partial
//                                sum per CTA;
//   attn_decode_finish_kernel    sum of the partials; then the new key and value take their ring
//                                slot and num_tokens grows.
#include <math.h>

#include "rgk_common.cuh"
#include "rgk_internal.h"
#include "tc_common.cuh"

namespace rgk {
namespace {

constexpr int kHdD = 256;
constexpr int kPerLane = kHdD / 32;        // 8 elements of a row per lane
constexpr float kMasked = -3.0e38f;        // "no logit yet" in the running maxima
constexpr int kSplits = 16;                // CTAs per sequence in the logits and values kernels
constexpr int kHeadPad = 16;               // heads of a logits row, padded
constexpr int kWarps = 8;                  // warps per CTA

// The 16-byte packs of this lane's 8 elements of a row.
struct RowPack { uint4 v[2]; };

__device__ __forceinline__ RowPack load_pack(const float* row, int lane) {
  return {{ld_stream(row + lane * kPerLane), ld_stream(row + lane * kPerLane + 4)}};
}
__device__ __forceinline__ void unpack_row(const RowPack& r, float (&f)[kPerLane]) {
  unpack<float>(r.v[0], f);
  unpack<float>(r.v[1], f + 4);
}

// Ring slot j holds the latest position congruent to j (mod W) that is below nt, the number of
// tokens seen; the query, at position nt, sees positions nt - W .. nt (torch/modules.py:155-184).
// Once the ring is full every slot holds such a position; before that only slots below nt are
// filled.  So the visible slots are exactly j < nt.
__device__ __forceinline__ int visible_slots(int nt, int W) { return nt < W ? nt : W; }

// The visible entries of a sequence are numbered 0 .. n_vis: ring slots 0 .. n_vis - 1, then the
// new token.  CTA c of kSplits takes entries [c * chunk, (c + 1) * chunk), its warp w every 8th of
// them starting at w.
__device__ __forceinline__ int chunk_of(int total) { return (total + kSplits - 1) / kSplits; }

// grid (B, kSplits).  logits: float [B, W + 1, 16] (head-minor; row e = visible entry e);
// stats: float2 [B, kSplits, kN] = the maximum of the CTA's logits of a head and the sum of
// exp(logit - maximum) over them.
template <int kN>
__global__ void __launch_bounds__(kWarps * 32)
attn_decode_logits_kernel(const float* __restrict__ q, const float* __restrict__ k_new,
                          const float* __restrict__ keys, const int* __restrict__ num_tokens, int W,
                          float* __restrict__ logits, float2* __restrict__ stats) {
  constexpr int kBatch = 4;   // rows whose loads are in flight together
  __shared__ float2 s_part[kWarps][kN];
  const int b = blockIdx.x, warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int nt = num_tokens[b];
  const int n_vis = visible_slots(nt, W);
  const int total = n_vis + 1;
  const int chunk = chunk_of(total);
  const int e_begin = blockIdx.y * chunk, e_end = min(e_begin + chunk, total);
  const float scale = 0.0625f;                     // 256^-1/2
  float qf[kN][kPerLane];
#pragma unroll
  for (int n = 0; n < kN; ++n) {
    const RowPack r = load_pack(q + ((int64_t)b * kN + n) * kHdD, lane);
    unpack_row(r, qf[n]);
  }
  float* lg = logits + (int64_t)b * (W + 1) * kHeadPad;
  float m_run = kMasked, l_run = 0.0f;             // lanes < kN: this warp's statistics of head `lane`
  for (int e0 = e_begin + warp; e0 < e_end; e0 += kWarps * kBatch) {
    RowPack raw[kBatch];
#pragma unroll
    for (int u = 0; u < kBatch; ++u) {
      const int e = e0 + u * kWarps;
      if (e < e_end)
        raw[u] = load_pack(e == n_vis ? k_new + (int64_t)b * kHdD
                                      : keys + ((int64_t)b * W + e) * kHdD, lane);
    }
#pragma unroll
    for (int u = 0; u < kBatch; ++u) {
      const int e = e0 + u * kWarps;
      if (e < e_end) {                             // (the same for every lane of the warp)
        float kf[kPerLane];
        unpack_row(raw[u], kf);
        float part[kN];
#pragma unroll
        for (int n = 0; n < kN; ++n) {
          float a = 0.0f;
#pragma unroll
          for (int i = 0; i < kPerLane; ++i) a = fmaf(qf[n][i], kf[i], a);
          part[n] = a;
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
#pragma unroll
          for (int n = 0; n < kN; ++n) part[n] += __shfl_xor_sync(0xffffffffu, part[n], o);
        }
        float mine = 0.0f;
#pragma unroll
        for (int n = 0; n < kN; ++n)
          if (lane == n) mine = part[n] * scale;
        if (lane < kN) {
          lg[(int64_t)e * kHeadPad + lane] = mine;
          const float m_new = fmaxf(m_run, mine);
          l_run = l_run * __expf(m_run - m_new) + __expf(mine - m_new);
          m_run = m_new;
        }
      }
    }
  }
  if (lane < kN) s_part[warp][lane] = make_float2(m_run, l_run);
  __syncthreads();
  if (threadIdx.x < kN) {
    float m = kMasked, l = 0.0f;
    for (int w = 0; w < kWarps; ++w) m = fmaxf(m, s_part[w][threadIdx.x].x);
    for (int w = 0; w < kWarps; ++w) {
      const float2 p = s_part[w][threadIdx.x];
      if (p.x > kMasked) l += p.y * __expf(p.x - m);
    }
    stats[((int64_t)b * kSplits + blockIdx.y) * kN + threadIdx.x] = make_float2(m, l);
  }
}

// grid (B, kSplits): CTA (b, c) multiplies the probabilities of its entries with their value rows,
// all 256 columns (a lane holds 8 of them), for the kN heads.  partial: float [B, kSplits, kN, 256].
template <int kN>
__global__ void __launch_bounds__(kWarps * 32)
attn_decode_values_kernel(const float* __restrict__ logits, const float2* __restrict__ stats,
                          const float* __restrict__ v_new, const float* __restrict__ values,
                          const int* __restrict__ num_tokens, int W, float* __restrict__ partial) {
  constexpr int kBatch = 4;
  static_assert(kN <= kHeadPad, "a logits row holds 16 heads");
  __shared__ float s_acc[kWarps / 2][kN][kHdD];    // 40 KiB at 10 heads
  __shared__ float s_stat[2][kHeadPad];            // maximum and 1 / sum of every head
  const int b = blockIdx.x, warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int nt = num_tokens[b];
  const int n_vis = visible_slots(nt, W);
  const int total = n_vis + 1;
  const int chunk = chunk_of(total);
  const int e_begin = blockIdx.y * chunk, e_end = min(e_begin + chunk, total);
  const float* lg = logits + (int64_t)b * (W + 1) * kHeadPad;
  if (threadIdx.x < kHeadPad) {
    float m = kMasked, l = 0.0f;
    if (threadIdx.x < kN) {
      const float2* st = stats + (int64_t)b * kSplits * kN + threadIdx.x;
      for (int c = 0; c < kSplits; ++c) m = fmaxf(m, st[c * kN].x);
      for (int c = 0; c < kSplits; ++c) {
        const float2 p = st[c * kN];
        if (p.x > kMasked) l += p.y * __expf(p.x - m);
      }
    }
    s_stat[0][threadIdx.x] = m;
    s_stat[1][threadIdx.x] = l > 0.0f ? 1.0f / l : 0.0f;
  }
  __syncthreads();
  const float my_m = s_stat[0][lane & (kHeadPad - 1)], my_inv = s_stat[1][lane & (kHeadPad - 1)];
  float acc[kN][kPerLane];
#pragma unroll
  for (int n = 0; n < kN; ++n)
#pragma unroll
    for (int i = 0; i < kPerLane; ++i) acc[n][i] = 0.0f;
  for (int e0 = e_begin + warp; e0 < e_end; e0 += kWarps * kBatch) {
    RowPack raw[kBatch];
    float lgv[kBatch];
#pragma unroll
    for (int u = 0; u < kBatch; ++u) {
      const int e = e0 + u * kWarps;
      lgv[u] = kMasked;
      if (e < e_end) {
        raw[u] = load_pack(e == n_vis ? v_new + (int64_t)b * kHdD
                                      : values + ((int64_t)b * W + e) * kHdD, lane);
        if (lane < kN) lgv[u] = lg[(int64_t)e * kHeadPad + lane];
      }
    }
#pragma unroll
    for (int u = 0; u < kBatch; ++u) {
      const int e = e0 + u * kWarps;
      if (e < e_end) {                             // (the same for every lane of the warp)
        float vf[kPerLane];
        unpack_row(raw[u], vf);
        // lane n < kN: the normalised probability of head n
        const float p_mine = lgv[u] > kMasked ? __expf(lgv[u] - my_m) * my_inv : 0.0f;
#pragma unroll
        for (int n = 0; n < kN; ++n) {
          const float p = __shfl_sync(0xffffffffu, p_mine, n);
#pragma unroll
          for (int i = 0; i < kPerLane; ++i) acc[n][i] = fmaf(p, vf[i], acc[n][i]);
        }
      }
    }
  }
  // the 8 warps: the upper half hands its sums to the lower half, three times over
#pragma unroll
  for (int half = kWarps / 2; half >= 1; half >>= 1) {
    if (warp >= half && warp < 2 * half) {
#pragma unroll
      for (int n = 0; n < kN; ++n)
#pragma unroll
        for (int i = 0; i < kPerLane; ++i) s_acc[warp - half][n][lane * kPerLane + i] = acc[n][i];
    }
    __syncthreads();
    if (warp < half) {
#pragma unroll
      for (int n = 0; n < kN; ++n)
#pragma unroll
        for (int i = 0; i < kPerLane; ++i) acc[n][i] += s_acc[warp][n][lane * kPerLane + i];
    }
    __syncthreads();
  }
  if (warp == 0) {
    float* dst = partial + (((int64_t)b * kSplits + blockIdx.y) * kN) * kHdD + lane * kPerLane;
#pragma unroll
    for (int n = 0; n < kN; ++n) {
      *reinterpret_cast<float4*>(dst + n * kHdD) = make_float4(acc[n][0], acc[n][1], acc[n][2], acc[n][3]);
      *reinterpret_cast<float4*>(dst + n * kHdD + 4) = make_float4(acc[n][4], acc[n][5], acc[n][6], acc[n][7]);
    }
  }
}

// ------------------------------------------------------------------------------------------------
// bfloat16: the whole step in one kernel.
//
// Bound: reading the ring (2 W 512 bytes a sequence), and writing it where the caller wants a new ring
// instead of an updated one.  A cluster of S CTAs serves a sequence, each a share of the slots: stages
// of 32 keys and 32 values come in by TMA (128-byte swizzle, 3 stages, two CTAs an SM), and for a new
// ring go out again by TMA from the same shared memory, so that the copy costs no pass of its own.
// Per stage: logits on the warp-level tensor-core instruction (m16n8k16: 16 keys x 8 heads; a tile of
// 128 rows as tcgen05 wants it would be mostly padding), four combinations of 16 keys and 8 heads times two
// halves of the 256 elements for the 8 warps; a running softmax per head (16 threads each); then P V,
// 32 columns a warp.  The new token is where the last CTA's running softmax starts.  At the end the CTAs
// exchange (maximum, sum, O) through distributed shared memory and finish 256 / S columns each.
// 64 sequences with full rings of 2048 and a new ring took 111 us as three kernels behind three copies.
//
// The logits are rounded to bfloat16 twice as the reference does; weights 2^(s - m) are rounded to
// bfloat16 before the division by their sum instead of behind it.
// ------------------------------------------------------------------------------------------------
__device__ __forceinline__ void ldsm_x4(uint32_t addr, uint32_t (&r)[4]) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0, %1, %2, %3}, [%4];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr) : "memory");
}
__device__ __forceinline__ void ldsm_x4_trans(uint32_t addr, uint32_t (&r)[4]) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0, %1, %2, %3}, [%4];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr) : "memory");
}
__device__ __forceinline__ float ld_peer_f32(uint32_t addr) {
  float v;
  asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(v) : "r"(addr) : "memory");
  return v;
}

constexpr int kRows = 32;                          // ring slots of a stage
constexpr int kSliceR = kRows * 128;               // 64 columns of them: 4 KiB
constexpr int kStageR = 8 * kSliceR;               // four slices of keys, four of values
constexpr int kStagesR = 3;
constexpr int kMaxClusterR = 16;                   // more than 8 has to be allowed per kernel
constexpr int kQPitch = 528;                       // bytes of a query row, padded
constexpr int kLogPitch = 17;                      // floats of a logits row
constexpr int kPPitch = 80;                        // bytes of a head's 32 weights, padded
constexpr int kOffQR = kStagesR * kStageR;
constexpr int kOffLogR = kOffQR + 16 * kQPitch;    // [half of the contraction][row][head]
constexpr int kOffPR = kOffLogR + 2 * kRows * kLogPitch * 4;
constexpr int kOffStatR = kOffPR + 16 * kPPitch;   // maximum, sum, rescaling factor of the heads
constexpr int kOffRot = kOffStatR + 3 * 16 * 4;    // cosine, sine of the 64 rotated pairs
constexpr int kOffNew = kOffRot + 2 * 64 * 4;      // the new key (rotated) and value
constexpr int kOffBarR = kOffNew + 2 * 512;
constexpr int kOffAbortR = kOffBarR + kStagesR * 8;
constexpr int kSmemR = kOffAbortR + 8 + 1024;
static_assert(kOffLogR % 16 == 0 && kOffPR % 16 == 0 && kOffNew % 16 == 0 && kOffBarR % 8 == 0, "alignment");
static_assert(2 * (kSmemR + 1024) <= 233472, "two CTAs an SM");
static_assert(16 * kHdD * 4 + 16 * kMaxClusterR * 4 <= kOffQR, "the exchanged sums lie over the stages");

struct RingArgs {
  const __nv_bfloat16 *q, *k_new, *v_new;          // [B, kN, 256], [B, 256], [B, 256]
  const void* pos;                                 // [B]: rotates q and k_new; NULL: they are rotated
  int pos64;
  const int* seen_in;
  int* seen_out;
  __nv_bfloat16 *keys, *values;                    // where the new token goes (update)
  int W, copy, update, S;                          // S: CTAs of a sequence
  __nv_bfloat16* out;
  int* status;
};

// The last step of a CTA: its 256 / S columns of every head from the S CTAs' (maximum, sum, O), S up to kMax
// (the loads of all are in flight together: with sixteen places for eight CTAs the step took 1 us longer).
template <int kN, int kMax>
__device__ __forceinline__ void combine_ctas(uint32_t s_base, float* s_w, int S, int split, int b,
                                             __nv_bfloat16* __restrict__ out) {
  const int tid = threadIdx.x;
  if (tid < 16) {
    float m = kMasked, sum = 0.0f;
    float ms[kMax], ls[kMax];
#pragma unroll
    for (int c = 0; c < kMax; ++c) {
      ms[c] = kMasked;
      ls[c] = 0.0f;
      if (c < S) {
        const uint32_t peer = peer_smem(s_base + kOffStatR, c);
        ms[c] = ld_peer_f32(peer + tid * 4);
        ls[c] = ld_peer_f32(peer + 64 + tid * 4);
      }
      m = fmaxf(m, ms[c]);
    }
#pragma unroll
    for (int c = 0; c < kMax; ++c) {
      ms[c] = __expf(ms[c] - m);
      sum = fmaf(ls[c], ms[c], sum);
    }
#pragma unroll
    for (int c = 0; c < kMax; ++c) s_w[c * 16 + tid] = ms[c] / sum;
  }
  __syncthreads();
  const int cols = kHdD / S, pairs = cols / 2;
  for (int i = tid; i < kN * pairs; i += 256) {
    const int h = i / pairs, col = split * cols + (i - h * pairs) * 2;
    float o0 = 0.0f, o1 = 0.0f;
#pragma unroll
    for (int c = 0; c < kMax; ++c) {
      if (c < S) {
        const uint32_t src = peer_smem(s_base + (uint32_t)(h * kHdD + col) * 4, c);
        const float w = s_w[c * 16 + h];
        o0 = fmaf(ld_peer_f32(src), w, o0);
        o1 = fmaf(ld_peer_f32(src + 4), w, o1);
      }
    }
    *reinterpret_cast<uint32_t*>(out + ((int64_t)b * kN + h) * kHdD + col) = pack_bf16x2(o0, o1);
  }
}

template <int kN>
__global__ void __launch_bounds__(256, 2)
attn_decode_ring_kernel(const __grid_constant__ CUtensorMap map_k, const __grid_constant__ CUtensorMap map_v,
                        const __grid_constant__ CUtensorMap map_k_out,
                        const __grid_constant__ CUtensorMap map_v_out, const __grid_constant__ RingArgs a) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = smem_raw + ((1024u - (smem_u32(smem_raw) & 1023u)) & 1023u);
  const uint32_t s_base = smem_u32(smem);
  float* s_log = reinterpret_cast<float*>(smem + kOffLogR);
  float* s_m = reinterpret_cast<float*>(smem + kOffStatR);
  float* s_l = s_m + 16;
  float* s_alpha = s_m + 32;
  float* s_cos = reinterpret_cast<float*>(smem + kOffRot);
  float* s_sin = s_cos + 64;
  __nv_bfloat16* s_new = reinterpret_cast<__nv_bfloat16*>(smem + kOffNew);
  volatile int* s_abort = reinterpret_cast<volatile int*>(smem + kOffAbortR);
  auto bar = [&](int s) { return s_base + kOffBarR + 8u * s; };

  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, g = lane >> 2, t = lane & 3;
  const int S = a.S, b = blockIdx.x / S, split = blockIdx.x - b * S;
  if (tid == 0) {
    *s_abort = 0;
    for (int s = 0; s < kStagesR; ++s) mbar_init(bar(s), 1);
    mbar_fence_init();
  }
  grid_dependency_wait();
  grid_launch_dependents();
  const int nt = a.seen_in[b];
  const int n_vis = visible_slots(nt, a.W);
  // this CTA's slots: a share of the whole ring where all of it is copied, else of the visible part
  const int of = a.copy ? a.W : n_vis;
  const int chunk = ((of + S - 1) / S + kRows - 1) / kRows * kRows;
  const int begin = split * chunk, end = min(begin + chunk, of);
  const int n_st = end > begin ? (end - begin + kRows - 1) / kRows : 0;
  __syncthreads();
  auto load = [&](int i) {
    const int s = i % kStagesR;
    const uint32_t st = s_base + s * kStageR;
    mbar_expect_tx(bar(s), kStageR);
#pragma unroll
    for (int c = 0; c < 4; ++c) {
      tma_load_3d(st + c * kSliceR, &map_k, c * 64, begin + i * kRows, b, bar(s));
      tma_load_3d(st + (4 + c) * kSliceR, &map_v, c * 64, begin + i * kRows, b, bar(s));
    }
  };
  if (tid == 0) {
    for (int i = 0; i < n_st && i < kStagesR; ++i) load(i);
  }

  // ---- the rotated queries and the new key
  if (a.pos != nullptr && tid < 64) {
    const float p = a.pos64 ? (float)reinterpret_cast<const long long*>(a.pos)[b]
                            : (float)reinterpret_cast<const int*>(a.pos)[b];
    const float ang = p * (1.0f / powf(10000.0f, 2.0f * (float)tid / 128.0f));
    s_cos[tid] = round_bf16(cosf(ang));
    s_sin[tid] = round_bf16(sinf(ang));
  }
  __syncthreads();
  for (int i = tid; i < 18 * 32; i += 256) {       // rows: 16 heads, the new key, the new value
    const int row = i >> 5, j = i & 31;            // a pack of 8 columns
    const __nv_bfloat16* src = row < 16 ? a.q + ((int64_t)b * kN + row) * kHdD
                                        : (row == 16 ? a.k_new : a.v_new) + (int64_t)b * kHdD;
    uint4 v = make_uint4(0u, 0u, 0u, 0u);
    if (row >= 16 || row < kN) {
      v = *reinterpret_cast<const uint4*>(src + j * 8);
      if (a.pos != nullptr && row != 17 && j < 16) {
        // columns 0-63 pair with 64-127
        const uint4 o = *reinterpret_cast<const uint4*>(src + (j ^ 8) * 8);
        const uint32_t mine[4] = {v.x, v.y, v.z, v.w}, other[4] = {o.x, o.y, o.z, o.w};
        uint32_t r[4];
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          const int f = (j & 7) * 8 + 2 * e;
          const uint32_t cs = pack_bf16x2(s_cos[f], s_cos[f + 1]), sn = pack_bf16x2(s_sin[f], s_sin[f + 1]);
          r[e] = j < 8 ? bsub2(bmul2(mine[e], cs), bmul2(other[e], sn))
                       : badd2(bmul2(mine[e], cs), bmul2(other[e], sn));
        }
        v = make_uint4(r[0], r[1], r[2], r[3]);
      }
    }
    uint8_t* dst = row < 16 ? smem + kOffQR + row * kQPitch : smem + kOffNew + (row - 16) * 512;
    *reinterpret_cast<uint4*>(dst + j * 16) = v;
  }
  __syncthreads();

  // ---- the new token: the last CTA's softmax starts with it
  float acc[4][4];                                 // heads g and g + 8, columns 32 warp + 8 n + 2 t, + 1
#pragma unroll
  for (int n = 0; n < 4; ++n) acc[n][0] = acc[n][1] = acc[n][2] = acc[n][3] = 0.0f;
  const bool with_new = split == S - 1;
  for (int h = warp; h < 16; h += 8) {
    float dot = 0.0f;
    if (with_new) {
      const uint4 x = *reinterpret_cast<const uint4*>(smem + kOffQR + h * kQPitch + lane * 16);
      const uint4 y = *reinterpret_cast<const uint4*>(smem + kOffNew + lane * 16);
      const uint32_t xs[4] = {x.x, x.y, x.z, x.w}, ys[4] = {y.x, y.y, y.z, y.w};
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        dot = fmaf(bf16_lo(xs[e]), bf16_lo(ys[e]), dot);
        dot = fmaf(bf16_hi(xs[e]), bf16_hi(ys[e]), dot);
      }
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) dot += __shfl_xor_sync(0xffffffffu, dot, o);
    }
    if (lane == 0) {
      // (the maximum stays a number, and above -inf; a logit that is neither leaves its mark in the sum)
      const float x = round_bf16(round_bf16(dot) * 0.0625f), m = with_new ? fmaxf(x, kMasked) : kMasked;
      s_m[h] = m;
      s_l[h] = with_new ? __expf(x - m) : 0.0f;
    }
  }
  if (with_new) {
#pragma unroll
    for (int n = 0; n < 4; ++n) {
      const uint32_t v = *reinterpret_cast<const uint32_t*>(s_new + kHdD + warp * 32 + n * 8 + 2 * t);
      acc[n][0] = acc[n][2] = bf16_lo(v);
      acc[n][1] = acc[n][3] = bf16_hi(v);
    }
  }
  // this warp's part of a stage's logits: 16 keys, 8 heads, half of the contraction
  const int row_tile = warp & 1, head_tile = (warp >> 1) & 1, khalf = warp >> 2;
  uint32_t qf[8][2];
#pragma unroll
  for (int ks = 0; ks < 8; ++ks) {
    const uint8_t* src = smem + kOffQR + (head_tile * 8 + g) * kQPitch + khalf * 256 + ks * 32 + t * 4;
    qf[ks][0] = *reinterpret_cast<const uint32_t*>(src);
    qf[ks][1] = *reinterpret_cast<const uint32_t*>(src + 16);
  }
  const int m_row = (lane & 7) + ((lane >> 3) & 1) * 8;      // row of an 8 x 8 matrix pair this lane names
  const int m_piece = lane >> 4;
  __syncthreads();
  if (with_new) {                                  // (times one, unless the new logit is infinite or no number)
    const float f0 = s_l[g], f1 = s_l[g + 8];
#pragma unroll
    for (int n = 0; n < 4; ++n) {
      acc[n][0] *= f0; acc[n][1] *= f0;
      acc[n][2] *= f1; acc[n][3] *= f1;
    }
  }

  bool ok = true;
  for (int i = 0; i < n_st; ++i) {
    const int s = i % kStagesR;
    const uint32_t st = s_base + s * kStageR;
    const int e0 = begin + i * kRows;
    if (ok) ok = mbar_wait(bar(s), (i / kStagesR) & 1, s_abort);
    if (a.copy && tid == 0) {
#pragma unroll
      for (int c = 0; c < 4; ++c) {
        tma_store_3d(&map_k_out, c * 64, e0, b, st + c * kSliceR);
        tma_store_3d(&map_v_out, c * 64, e0, b, st + (4 + c) * kSliceR);
      }
      bulk_commit();
    }
    const int lim = min(end, n_vis) - e0;          // rows of the stage that count
    if (lim > 0) {
      __syncwarp();
      float c4[4] = {0.0f, 0.0f, 0.0f, 0.0f};
      {
        const int r = row_tile * 16 + m_row;
#pragma unroll
        for (int ks = 0; ks < 8; ++ks) {
          const int j = khalf * 16 + ks * 2 + m_piece;       // 16-byte piece of the key's row
          uint32_t f[4];
          ldsm_x4(st + (j >> 3) * kSliceR + r * 128 + (((j & 7) ^ (r & 7)) << 4), f);
          mma_16816(c4, f[0], f[1], f[2], f[3], qf[ks][0], qf[ks][1]);
        }
        float* dst = s_log + (khalf * kRows + row_tile * 16 + g) * kLogPitch + head_tile * 8 + 2 * t;
        dst[0] = c4[0];
        dst[1] = c4[1];
        dst[8 * kLogPitch] = c4[2];
        dst[8 * kLogPitch + 1] = c4[3];
      }
      __syncthreads();
      {
        // thread (head, pair of keys); the 16 threads of a head are half a warp
        const int h = tid >> 4, e = (tid & 15) * 2;
        const float* l0 = s_log + e * kLogPitch + h;
        const float* l1 = l0 + kRows * kLogPitch;
        // two tensor operations in the reference: the contraction, then the scaling by 256^-1/2
        float x = round_bf16(round_bf16(l0[0] + l1[0]) * 0.0625f);
        float y = round_bf16(round_bf16(l0[kLogPitch] + l1[kLogPitch]) * 0.0625f);
        if (e >= lim) x = -INFINITY;
        if (e + 1 >= lim) y = -INFINITY;
        float mx = fmaxf(x, y);
#pragma unroll
        for (int o = 1; o < 16; o <<= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, o));
        const float m_old = s_m[h], l_old = s_l[h];
        const float m = fmaxf(mx, m_old);
        // (0 where nothing is visible: m is at least kMasked; what is no number stays none)
        const float p0 = __expf(x - m), p1 = __expf(y - m);
        float sum = p0 + p1;
#pragma unroll
        for (int o = 1; o < 16; o <<= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
        *reinterpret_cast<uint32_t*>(smem + kOffPR + h * kPPitch + e * 2) = pack_bf16x2(p0, p1);
        if ((tid & 15) == 0) {
          const float alpha = __expf(m_old - m);   // 0 from "no logit yet"
          s_alpha[h] = alpha;
          s_m[h] = m;
          s_l[h] = fmaf(l_old, alpha, sum);
        }
      }
      __syncthreads();
      {
        const float f0 = s_alpha[g], f1 = s_alpha[g + 8];
#pragma unroll
        for (int n = 0; n < 4; ++n) {
          acc[n][0] *= f0; acc[n][1] *= f0;
          acc[n][2] *= f1; acc[n][3] *= f1;
        }
#pragma unroll
        for (int ks = 0; ks < 2; ++ks) {
          uint32_t p[4];
          ldsm_x4(s_base + kOffPR + m_row * kPPitch + (ks * 2 + m_piece) * 16, p);
          // whatever lies in slots that do not count is not multiplied by their zero weights
          const int k0 = ks * 16 + 2 * t;
          const uint32_t keep0 = (k0 < lim ? 0xffffu : 0u) | (k0 + 1 < lim ? 0xffff0000u : 0u);
          const uint32_t keep1 = (k0 + 8 < lim ? 0xffffu : 0u) | (k0 + 9 < lim ? 0xffff0000u : 0u);
          const int r = ks * 16 + m_row;
#pragma unroll
          for (int n2 = 0; n2 < 2; ++n2) {
            const int j = warp * 4 + n2 * 2 + m_piece;
            uint32_t f[4];
            ldsm_x4_trans(st + (4 + (j >> 3)) * kSliceR + r * 128 + (((j & 7) ^ (r & 7)) << 4), f);
            mma_16816(acc[2 * n2], p[0], p[1], p[2], p[3], f[0] & keep0, f[1] & keep1);
            mma_16816(acc[2 * n2 + 1], p[0], p[1], p[2], p[3], f[2] & keep0, f[3] & keep1);
          }
        }
      }
    }
    __syncthreads();                               // the stage has been read
    if (tid == 0 && i + kStagesR < n_st && ok) {
      if (a.copy) bulk_wait_read();                // by the store as well
      load(i + kStagesR);
    }
  }

  // ---- the CTAs of the sequence: (maximum, sum, O) of all through distributed shared memory
  if (a.copy && tid == 0) bulk_wait_all();
  __syncthreads();
  float* s_o = reinterpret_cast<float*>(smem);     // [16][256]
  float* s_w = s_o + 16 * kHdD;                    // [CTA][16]: what its O counts
#pragma unroll
  for (int n = 0; n < 4; ++n) {
    const int col = warp * 32 + n * 8 + 2 * t;
    *reinterpret_cast<float2*>(s_o + g * kHdD + col) = make_float2(acc[n][0], acc[n][1]);
    *reinterpret_cast<float2*>(s_o + (g + 8) * kHdD + col) = make_float2(acc[n][2], acc[n][3]);
  }
  __syncwarp();
  cluster_arrive();
  cluster_wait();
  if (S <= 8) combine_ctas<kN, 8>(s_base, s_w, S, split, b, a.out);
  else combine_ctas<kN, kMaxClusterR>(s_base, s_w, S, split, b, a.out);
  if (a.update && split == 0) {
    // every CTA of the sequence has read its slots (and written its copies)
    if (tid < 64) {
      const int64_t at = ((int64_t)b * a.W + nt % a.W) * kHdD + (tid & 31) * 8;
      *reinterpret_cast<uint4*>((tid < 32 ? a.keys : a.values) + at) =
          *reinterpret_cast<const uint4*>(s_new + tid * 8);
    }
    if (tid == 0) a.seen_out[b] = nt + 1;
  }
  if (tid == 0 && *s_abort && a.status != nullptr) atomicExch(a.status, kStatusTimeout);
  __syncwarp();
  cluster_arrive();
  cluster_wait();                                  // nobody reads this CTA's memory any more
}

template <int kN>
cudaError_t launch_ring(RingArgs a, const void* keys_in, const void* values_in, int64_t B, cudaStream_t s) {
  CUtensorMap mk, mv, mk_out, mv_out;
  if (!tensor_map_bte(&mk, keys_in, (uint64_t)B, (uint64_t)a.W, kHdD, kRows, 64, true) ||
      !tensor_map_bte(&mv, values_in, (uint64_t)B, (uint64_t)a.W, kHdD, kRows, 64, true))
    return cudaErrorInvalidValue;
  mk_out = mk;
  mv_out = mv;
  if (a.copy && (!tensor_map_bte(&mk_out, a.keys, (uint64_t)B, (uint64_t)a.W, kHdD, kRows, 64, true) ||
                 !tensor_map_bte(&mv_out, a.values, (uint64_t)B, (uint64_t)a.W, kHdD, kRows, 64, true)))
    return cudaErrorInvalidValue;
  static PerDeviceOnce once;
  int num_sms = 0;
  cudaError_t e = once.run([] {
    const cudaError_t r =
        cudaFuncSetAttribute(attn_decode_ring_kernel<kN>, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmemR);
    return r != cudaSuccess ? r : cudaFuncSetAttribute(attn_decode_ring_kernel<kN>,
                                                       cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
  }, &num_sms);
  if (e != cudaSuccess) return e;
  // as many CTAs as run at once, two an SM; sixteen only for a few sequences whose whole rings are gone
  // through (one of 2048 slots 48.0 -> 43.5 us a block, but 65 -> 71 at 16 sequences: clusters that large
  // do not all find a place at once; and a ring that is updated in place may hold a few slots only)
  int S = 1;
  while (S < kMaxClusterR && 2 * S * B <= (S < 8 ? 2 : a.copy) * num_sms) S *= 2;
  if (S * B > 0x7fffffff) return cudaErrorInvalidValue;
  a.S = S;
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = (unsigned)S;
  attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
  attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[1].val.programmaticStreamSerializationAllowed = 1;
  cudaLaunchConfig_t cfg = {};
  cfg.blockDim = dim3(256);
  cfg.dynamicSmemBytes = kSmemR;
  cfg.stream = s;
  cfg.attrs = attr;
  cfg.numAttrs = 2;
  cfg.gridDim = dim3((unsigned)(S * B));
  e = cudaLaunchKernelEx(&cfg, attn_decode_ring_kernel<kN>, mk, mv, mk_out, mv_out, a);
  return e != cudaSuccess ? e : cudaGetLastError();
}

// grid (B, kN), 256 threads = the 256 columns: out [B, kN, 256] = the rounded sum of the partials;
// then (update != 0; the CTAs of head 0) the new key and value take ring slot num_tokens % W and
// num_tokens grows by one.
template <int kN>
__global__ void __launch_bounds__(kHdD)
attn_decode_finish_kernel(const float* __restrict__ partial, const float* __restrict__ k_new,
                          const float* __restrict__ v_new, float* __restrict__ keys, float* __restrict__ values,
                          int* __restrict__ num_tokens, int W, int update, float* __restrict__ out) {
  const int b = blockIdx.x, n = blockIdx.y, c = threadIdx.x;
  float a = 0.0f;
#pragma unroll
  for (int s = 0; s < kSplits; ++s) a += partial[(((int64_t)b * kSplits + s) * kN + n) * kHdD + c];
  out[((int64_t)b * kN + n) * kHdD + c] = a;
  if (update && n == 0) {
    const int nt = num_tokens[b];
    const int slot = nt % W;
    keys[((int64_t)b * W + slot) * kHdD + c] = k_new[(int64_t)b * kHdD + c];
    values[((int64_t)b * W + slot) * kHdD + c] = v_new[(int64_t)b * kHdD + c];
    __syncthreads();                                // every thread has read nt
    if (c == 0) num_tokens[b] = nt + 1;
  }
}

// the logits [B, W + 1, 16], the per-CTA softmax statistics [B, kSplits, N], the partial sums
// [B, kSplits, N, 256]
size_t logits_bytes(int64_t B, int W) {
  return (((size_t)B * (W + 1) * kHeadPad * sizeof(float)) + 255) & ~(size_t)255;
}
size_t stats_bytes(int64_t B, int N) {
  return (((size_t)B * kSplits * N * sizeof(float2)) + 255) & ~(size_t)255;
}
size_t partial_bytes(int64_t B, int N) {
  return (((size_t)B * kSplits * N * kHdD * sizeof(float)) + 255) & ~(size_t)255;
}

template <int kN>
cudaError_t launch_decode_f32(const void* q, const void* k_new, const void* v_new, void* keys,
                            void* values, int* num_tokens, int64_t B, int W, int update, void* out,
                            void* ws, cudaStream_t s) {
  uint8_t* base = reinterpret_cast<uint8_t*>(ws) + 256;      // behind the status word
  float* lg = reinterpret_cast<float*>(base);
  float2* st = reinterpret_cast<float2*>(base + logits_bytes(B, W));
  float* part = reinterpret_cast<float*>(base + logits_bytes(B, W) + stats_bytes(B, kN));
  const dim3 grid((unsigned)B, kSplits);
  attn_decode_logits_kernel<kN><<<grid, kWarps * 32, 0, s>>>(
      (const float*)q, (const float*)k_new, (const float*)keys, num_tokens, W, lg, st);
  attn_decode_values_kernel<kN><<<grid, kWarps * 32, 0, s>>>(
      lg, st, (const float*)v_new, (const float*)values, num_tokens, W, part);
  attn_decode_finish_kernel<kN><<<dim3((unsigned)B, kN), kHdD, 0, s>>>(
      part, (const float*)k_new, (const float*)v_new, (float*)keys, (float*)values, num_tokens, W, update, (float*)out);
  return cudaGetLastError();
}

}  // namespace

bool attention_decode_supported(int hd, int N, int W) {
  const bool heads = N == 1 || N == 2 || N == 4 || N == 8 || N == 10;
  return hd == kHdD && heads && W >= 1;
}

size_t attention_decode_workspace_bytes(int64_t B, int N, int W) {
  return 256 + logits_bytes(B, W) + stats_bytes(B, N) + partial_bytes(B, N);
}

cudaError_t launch_attention_decode(const void* q, const void* k_new, const void* v_new, void* keys,
                                    void* values, int* num_tokens, int64_t B, int N, int W,
                                    int update, void* out, void* ws, cudaStream_t s) {
  if (B == 0) return cudaSuccess;
#define RGK_DEC(NN)                                                                               \
  case NN:                                                                                        \
    return launch_decode_f32<NN>(q, k_new, v_new, keys, values, num_tokens, B, W, update, out, ws, s)
  switch (N) {
    RGK_DEC(1); RGK_DEC(2); RGK_DEC(4); RGK_DEC(8); RGK_DEC(10);
    default: return cudaErrorInvalidValue;
  }
#undef RGK_DEC
}

cudaError_t launch_attention_decode_ring(const void* q, const void* k_new, const void* v_new, const void* pos,
                                         int pos64, const void* keys_in, const void* values_in,
                                         const int* seen_in, void* keys, void* values, int* seen, int64_t B,
                                         int N, int W, int update, void* out, int* status, cudaStream_t s) {
  if (B == 0) return cudaSuccess;
  using T_ = __nv_bfloat16;
  RingArgs a = {};
  a.q = static_cast<const T_*>(q);
  a.k_new = static_cast<const T_*>(k_new);
  a.v_new = static_cast<const T_*>(v_new);
  a.pos = pos;
  a.pos64 = pos64;
  a.seen_in = seen_in;
  a.seen_out = seen;
  a.keys = static_cast<T_*>(keys);
  a.values = static_cast<T_*>(values);
  a.W = W;
  a.copy = update && keys_in != keys ? 1 : 0;
  a.update = update;
  a.out = static_cast<T_*>(out);
  a.status = status;
  switch (N) {
    case 1: return launch_ring<1>(a, keys_in, values_in, B, s);
    case 2: return launch_ring<2>(a, keys_in, values_in, B, s);
    case 4: return launch_ring<4>(a, keys_in, values_in, B, s);
    case 8: return launch_ring<8>(a, keys_in, values_in, B, s);
    case 10: return launch_ring<10>(a, keys_in, values_in, B, s);
    default: return cudaErrorInvalidValue;
  }
}

}  // namespace rgk
