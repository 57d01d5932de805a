// Dense projections of FEW rows (up to some hundreds: the batch of a decode step, or a short prompt)
// on the 5th-generation tensor cores: torch.nn.Linear, the MLP's up-projection with its GeGLU, and
// the logits with their soft cap (recurrentgemma torch/modules.py:437-452, 531-548, 626-647,
// 749-752, 1001-1003; torch/griffin.py:183-185).
//
// Bound: streaming the weights (N x K bfloat16, 13 MB at 2560 x 2560) exactly once; the 128 x 256
// output tiles of the prefill GEMM would leave most SMs without a tile.  Here the WEIGHTS are the
// tall operand: a CTA owns F output features (a multiple of 8 up to 128) x a slice of K for up to
// 256 rows of x and computes the TRANSPOSED tile  D[feature, row] = W_tile x^T  with tcgen05.mma
// (M 128 = features, N = the rows of x, K 16).  F and the number of K slices are chosen per call so
// that the CTAs fill all SMs evenly: at 15360 features 148 CTAs own 104 each, where 128 would occupy
// 120 SMs (instruction rows beyond F multiply whatever lies behind the weights and are not read).
//
// The K slices of one feature tile are the CTAs of one thread-block cluster, and their partial sums
// meet in distributed shared memory: CTA r finishes the r-th share of the rows; every CTA lays its
// partial sums out in its idle ring, one block per destination, and sends each block with one bulk
// copy that signals the destination's mbarrier (stores from the registers of each thread into peers'
// memory, as an earlier version had them, moved 12-25 GB/s per SM and cost 4.5 us at 64 rows); CTA r
// adds the slices in rank order - a fixed order, so the result is the same bits on every run -
// applies the bias in float32, rounds once, applies gelu / residual / GeGLU with their own
// roundings, and writes its rows.  With a single K slice the epilogue writes the output from tensor
// memory directly.  Neighbouring lanes are neighbouring features, so pairs of lanes trade values of
// two rows and store 4 bytes each.
//
// Launched as a programmatic dependent: set-up and (where allowed, see `early`) the first weight
// tiles overlap the tail of the kernel in front.  Every mbarrier wait is bounded; on expiry the
// status word (if given) is raised and the CTA goes on to the cluster barriers (so its peers are
// not left waiting) and leaves.
#include <cuda.h>

#include <mutex>

#include "rgk_common.cuh"
#include "rgk_internal.h"
#include "tc_common.cuh"

namespace rgk {
namespace {

constexpr int SK = 64;                            // K per stage
constexpr int kFMax = 128;                        // features per CTA at most
constexpr int kRMax = 256;                        // rows of x per CTA at most
constexpr int kDataS = 220 * 1024;                // ring + exchange buffers, one CTA per SM
constexpr int kDataHalfS = 109 * 1024;            // the same when two CTAs are to share an SM
constexpr int kMaxStagesS = 12;
constexpr int kMaxClusterS = 8;
constexpr int kEpiS = 8;                          // 4 TMEM lane quarters x 2 column halves
constexpr int kThreadsS = (kEpiS + 2) * 32;
// behind the data: full[] empty[] acc recv barriers, the TMEM address, the abort flag, the biases of
// the CTA's features in float32; 1 KiB to align
constexpr int kOffTmemS = (2 * kMaxStagesS + 2) * 8;
constexpr int kOffAbortS = kOffTmemS + 4;
constexpr int kOffBiasS = 256;
constexpr int kTailS = 256 + 512 + 1024;
static_assert(kOffAbortS + 4 <= kOffBiasS, "tail too small");
static_assert(kDataS + kTailS <= 232448, "exceeds the 227 KiB of shared memory a CTA may use");
// Two kinds of shared-memory footprint, for kernels that alternate on the stream.  A kernel launched
// as a programmatic dependent is placed while its predecessor still holds most SMs, and SMs that the
// predecessor does not use would take two of its CTAs (the up-projection at 64 rows took 24 us instead
// of 15 that way).  A `wide` CTA fills more than half of an SM: two never share one, while a narrow CTA
// of the kernel in front or behind still fits beside it.
constexpr int kWideS = 114 * 1024;
static_assert(2 * (kWideS + 1024) > 233472, "two wide CTAs would fit an SM");
static_assert(kWideS + kDataHalfS + kTailS + 2 * 1024 <= 233472, "wide and narrow do not fit an SM");

__device__ __forceinline__ void tensor_prefetch_l2(const CUtensorMap* map, int x, int y) {
  asm volatile("cp.async.bulk.prefetch.tensor.2d.L2.global [%0, {%1, %2}];"
               :: "l"(map), "r"(x), "r"(y) : "memory");
}
__device__ __forceinline__ float bf16_value(__nv_bfloat16 v) {
  return __uint_as_float(static_cast<uint32_t>(__bfloat16_as_ushort(v)) << 16);
}

enum { kActNone = 0, kActGelu = 1, kActGeglu = 2, kActCap = 3 };

// One output value from its float32 sum: + bias, one rounding to bfloat16, then gelu (of the first matrix
// only) or the soft cap with their own roundings - the tensor operations of the reference, in its order.
template <int kAct>
__device__ __forceinline__ float finish1(float sum, float bias, float cap, bool first) {
  float y = round_bf16(sum + bias);
  if constexpr (kAct == kActGelu) y = first ? gelu_tanh_<true>(y) : y;
  if constexpr (kAct == kActCap) y = round_bf16(tanhf(round_bf16(__fdiv_rn(y, cap)))) * cap;
  return y;                                       // the caller's packing is the last rounding
}
// GeGLU: gate and value = round(round(sum) + bias) - the contraction and the bias add are two tensor
// operations in the reference (torch/layers.py:700-703, torch/modules.py:749-751).
__device__ __forceinline__ float geglu(float gate_sum, float value_sum, float gate_bias, float value_bias) {
  const float gate = round_bf16(round_bf16(gate_sum) + gate_bias);
  const float value = round_bf16(round_bf16(value_sum) + value_bias);
  return round_bf16(gelu_tanh_<true>(gate)) * value;
}

struct SmallMat {
  const __nv_bfloat16* bias;
  __nv_bfloat16* out;
  int n;                             // features
};
struct SmallArgs {
  SmallMat mat[3];
  const __nv_bfloat16* residual;
  int tile1, tile2;                  // the first feature tiles of the second and third matrix
  int M, R, F;                       // rows of x, rows and features per CTA
  int k_blocks, kb_per_split, splits;
  int n_stages, tmem_cols;
  int rows_per_rank, row_stride;     // rows a CTA of the cluster finishes; their pitch in the buffers
  int recv_off, bar_off;             // receive buffer and barriers behind the ring
  int early;                         // the kernel in front does not write weights
  float cap;
};

template <int kAct>
__global__ void __launch_bounds__(kThreadsS, 2)
gemm_small_kernel(const __grid_constant__ CUtensorMap map_x, const __grid_constant__ CUtensorMap map_w0,
                  const __grid_constant__ CUtensorMap map_w1, const __grid_constant__ CUtensorMap map_w2,
                  const __grid_constant__ SmallArgs a, int* status) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = smem_raw + ((1024u - (smem_u32(smem_raw) & 1023u)) & 1023u);
  const uint32_t s_base = smem_u32(smem);
  const uint32_t bar0 = s_base + a.bar_off;
  auto bar_full = [&](int s) { return bar0 + 8u * s; };
  auto bar_empty = [&](int s) { return bar0 + 8u * (kMaxStagesS + s); };
  const uint32_t bar_acc = bar0 + 8u * (2 * kMaxStagesS), bar_recv = bar_acc + 8u;
  volatile uint32_t* s_tmem = reinterpret_cast<volatile uint32_t*>(smem + a.bar_off + kOffTmemS);
  volatile int* s_abort = reinterpret_cast<volatile int*>(smem + a.bar_off + kOffAbortS);

  // (from a lane, so that the compiler knows it to be the same in the whole warp; with it the first copies, too, are
  // issued under elect_one: a block's decode step of 64 rows 106.1 -> 105.1 us)
  const int warp = __shfl_sync(0xffffffffu, (int)threadIdx.x >> 5, 0), lane = threadIdx.x & 31;
  const int F = a.F, R = a.R, splits = a.splits, n_stages = a.n_stages;
  const int split = splits > 1 ? (int)cluster_rank() : 0;   // cluster = (1, splits, 1)
  // the matrix this feature tile belongs to, its first feature there, the rows of x of this CTA
  const int mi = ((int)blockIdx.x >= a.tile1) + ((int)blockIdx.x >= a.tile2);
  const int f0 = ((int)blockIdx.x - (mi == 0 ? 0 : (mi == 1 ? a.tile1 : a.tile2))) * F;
  const CUtensorMap* map_w = mi == 0 ? &map_w0 : (mi == 1 ? &map_w1 : &map_w2);
  const __nv_bfloat16* bias = mi == 0 ? a.mat[0].bias : (mi == 1 ? a.mat[1].bias : a.mat[2].bias);
  __nv_bfloat16* out = mi == 0 ? a.mat[0].out : (mi == 1 ? a.mat[1].out : a.mat[2].out);
  const int n = mi == 0 ? a.mat[0].n : (mi == 1 ? a.mat[1].n : a.mat[2].n);
  const int row0 = blockIdx.z * R;
  const int M = min(a.M - row0, R);                // rows of x of this CTA that exist
  const int kb0 = split * a.kb_per_split;
  const int n_kb = min(kb0 + a.kb_per_split, a.k_blocks) - kb0;
  const uint32_t w_bytes = (uint32_t)F * 128, stage_bytes = w_bytes + (uint32_t)R * 128;
  const int pre = min(n_kb, n_stages);
  const int rpr = a.rows_per_rank, stride = a.row_stride;
  const uint32_t block_bytes = (uint32_t)(F * stride) * 4;   // partial sums of one rank's rows

  if (warp == kEpiS && elect_one()) {
    *s_abort = 0;
    for (int s = 0; s < n_stages; ++s) { mbar_init(bar_full(s), 1); mbar_init(bar_empty(s), 1); }
    mbar_init(bar_acc, 1);
    mbar_init(bar_recv, 1);
    mbar_fence_init();
    // the first weight tiles are on their way before anything else happens - into shared memory, or
    // only into L2 (the point of coherence) while the kernel in front may still be writing them
    for (int i = 0; i < pre; ++i) {
      if (a.early) {
        mbar_expect_tx(bar_full(i), stage_bytes);
        tma_load_2d(s_base + i * stage_bytes, map_w, (kb0 + i) * SK, f0, bar_full(i));
      } else {
        tensor_prefetch_l2(map_w, (kb0 + i) * SK, f0);
      }
    }
  }
  if (warp == kEpiS + 1) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;"
                 :: "r"(bar0 + kOffTmemS), "r"(a.tmem_cols) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *s_tmem;
  if (splits > 1) cluster_arrive();                // "this CTA runs and its barriers are set up"
  if (a.early) {
    grid_launch_dependents();
    grid_dependency_wait();
  } else {
    // the kernel behind may fetch weights as soon as it starts: not before the one in front, which
    // may have written them, has completed
    grid_dependency_wait();
    grid_launch_dependents();
  }

  float* s_bias = reinterpret_cast<float*>(smem + a.bar_off + kOffBiasS);
  if (threadIdx.x < kFMax) {                       // read behind a barrier of the epilogue warps
    const int f = threadIdx.x;
    s_bias[f] = bias != nullptr && f < F && f0 + f < n ? bf16_value(bias[f0 + f]) : 0.0f;
  }
  if (warp == kEpiS) {
    // ------------------------------ TMA producer --------------------------------------------------
    if (elect_one()) {
      for (int i = 0; i < pre; ++i) {
        if (!a.early) {
          mbar_expect_tx(bar_full(i), stage_bytes);
          tma_load_2d(s_base + i * stage_bytes, map_w, (kb0 + i) * SK, f0, bar_full(i));
        }
        tma_load_2d(s_base + i * stage_bytes + w_bytes, &map_x, (kb0 + i) * SK, row0, bar_full(i));
      }
    }
    __syncwarp();
    // the whole warp runs the loop and one elected lane issues (see mma_ring)
    bool ok = true;
    int s = 0;
    uint32_t phase = 0;                            // of the stage's previous contents
    for (int i = pre; i < n_kb; ++i) {
      ok = __all_sync(0xffffffffu, mbar_wait(bar_empty(s), phase, s_abort));
      if (!ok) break;
      if (elect_one()) {
        const uint32_t st = s_base + s * stage_bytes;
        mbar_expect_tx(bar_full(s), stage_bytes);
        tma_load_2d(st, map_w, (kb0 + i) * SK, f0, bar_full(s));
        tma_load_2d(st + w_bytes, &map_x, (kb0 + i) * SK, row0, bar_full(s));
      }
      __syncwarp();
      if (++s == n_stages) { s = 0; phase ^= 1; }
    }
    __syncwarp();
  } else if (warp == kEpiS + 1) {
    // ------------------------------ MMA issue -----------------------------------------------------
    RingPos at;
    if (mma_ring<SK / 16>(tmem_base, smem_desc_sw128(s_base), smem_desc_sw128(s_base + w_bytes),
                          stage_bytes >> 4, tc_idesc_bf16(128, R), n_kb, n_stages, bar_full(0),
                          bar_empty(0), at, s_abort) && elect_one())
      tc_commit(bar_acc);
    __syncwarp();
  }
  if (splits > 1) cluster_wait();                  // every CTA of the cluster runs

  // ------------------------------ epilogue (warps 0-7) ---------------------------------------------
  // a lane is a feature, an accumulator column a row of x; from 64 columns on, warps 4-7 take the
  // upper half of the columns
  const bool epi = warp < kEpiS;
  const int quarter = warp & 3, half = warp >> 2;
  const int f = quarter * 32 + lane;               // feature within the tile
  const bool two_halves = R >= 64;
  const int cols = two_halves ? R / 2 : R;
  const int col0 = two_halves ? half * cols : 0;
  const bool warp_active = epi && (two_halves || half == 0) && col0 < M && quarter * 32 < F;
  bool ok = true;
  if (epi) {
    named_bar_sync(1, kEpiS * 32);                 // the biases are in place
    ok = mbar_wait(bar_acc, 0, s_abort);
    __syncwarp();
    tc_fence_after();
  }
  const uint32_t t_row = tmem_base + (static_cast<uint32_t>(quarter * 32) << 16);

  if (splits > 1) {
    if (epi) {
      // blocks [destination rank][feature][row_stride] over the ring, which is idle: every load
      // has landed and every MMA has read it
      if (warp_active) {
        float* mine = reinterpret_cast<float*>(smem) + f * stride;
        int d = col0 / rpr, lm = col0 - d * rpr;   // the rank that finishes row m, its number there
        auto send4 = [&](int m, uint32_t v0, uint32_t v1, uint32_t v2, uint32_t v3) {
          // m is a multiple of 4, and so is rows_per_rank
          if (m < M && f < F)
            *reinterpret_cast<uint4*>(mine + d * F * stride + lm) = make_uint4(v0, v1, v2, v3);
          lm += 4;
          if (lm == rpr) { lm = 0; ++d; }
        };
        int c = col0;
        for (; c + 32 <= col0 + cols && c < M; c += 32) {
          uint32_t acc[32];
          tc_ld_32x32(t_row + c, acc);
          tc_wait_ld();
#pragma unroll
          for (int j = 0; j < 32; j += 4) send4(c + j, acc[j], acc[j + 1], acc[j + 2], acc[j + 3]);
        }
        if (c < col0 + cols && c < M) {
          uint32_t acc[16];
          tc_ld_32x16(t_row + c, acc);
          tc_wait_ld();
#pragma unroll
          for (int j = 0; j < 16; j += 4) send4(c + j, acc[j], acc[j + 1], acc[j + 2], acc[j + 3]);
        }
      }
      fence_proxy_async();
      named_bar_sync(1, kEpiS * 32);
      const bool have_rows = split * rpr < M;
      if (threadIdx.x == 0 && have_rows) mbar_expect_tx(bar_recv, (uint32_t)(splits - 1) * block_bytes);
      if ((int)threadIdx.x < splits - 1) {         // one lane per destination
        int d = split + 1 + (int)threadIdx.x;      // each rank starts with another one
        if (d >= splits) d -= splits;
        if (d * rpr < M) {
          const int slot = split < d ? split : split - 1;
          bulk_to_peer(peer_smem(s_base + a.recv_off + slot * block_bytes, d), s_base + d * block_bytes,
                       block_bytes, peer_smem(bar_recv, d));
        }
      }
      const int m_base = split * rpr;
      const int f_out = kAct == kActGeglu ? F / 2 : F;
      const int pairs = f_out / 2, n_out = kAct == kActGeglu ? n / 2 : n;
      const int o_base = kAct == kActGeglu ? f0 / 2 : f0;
      // the residual of this thread's first item, in flight while the partial sums travel
      auto load_residual = [&](int i, uint32_t (&res)[4]) {
        const int p = i % pairs, lm = (i / pairs) * 4, o = o_base + 2 * p;
#pragma unroll
        for (int j = 0; j < 4; ++j)
          if (lm < rpr && o < n_out && m_base + lm + j < M)
            res[j] = *reinterpret_cast<const uint32_t*>(a.residual + (int64_t)(row0 + m_base + lm + j) * n_out + o);
      };
      uint32_t res[4] = {};
      if (a.residual != nullptr) load_residual(threadIdx.x, res);
      if (have_rows && ok) ok = mbar_wait(bar_recv, 0, s_abort);
      __syncwarp();
      cluster_arrive();                            // everything sent to me has arrived
      if (have_rows && ok) {
        // the slices of my rows, added in rank order
        const float* own = reinterpret_cast<const float*>(smem) + split * F * stride;
        const float* recv = reinterpret_cast<const float*>(smem + a.recv_off);
        auto sum4 = [&](int feature, int lm) {
          float4 p[kMaxClusterS];                  // all loads before the first addition
#pragma unroll
          for (int s = 0; s < kMaxClusterS; ++s) {
            p[s] = make_float4(0.f, 0.f, 0.f, 0.f);
            if (s < splits) {
              const float* src = s == split ? own : recv + (s < split ? s : s - 1) * F * stride;
              p[s] = *reinterpret_cast<const float4*>(src + feature * stride + lm);
            }
          }
          float4 sum = p[0];
#pragma unroll
          for (int s = 1; s < kMaxClusterS; ++s) {
            if (s < splits) { sum.x += p[s].x; sum.y += p[s].y; sum.z += p[s].z; sum.w += p[s].w; }
          }
          return sum;
        };
        for (int i = threadIdx.x; i < pairs * (rpr / 4); i += kEpiS * 32) {
          const int p = i % pairs, lm = (i / pairs) * 4;
          const int o = o_base + 2 * p;            // first of two output features
          if (o >= n_out || m_base + lm >= M) continue;
          float v0[4], v1[4];
          if (a.residual != nullptr && i != (int)threadIdx.x) load_residual(i, res);
          if constexpr (kAct == kActGeglu) {
            const int fg = (p >> 1) * 8 + (p & 1) * 2;
            const float4 g0 = sum4(fg, lm), g1 = sum4(fg + 1, lm), u0 = sum4(fg + 4, lm), u1 = sum4(fg + 5, lm);
            const float bg0 = s_bias[fg], bg1 = s_bias[fg + 1], bu0 = s_bias[fg + 4], bu1 = s_bias[fg + 5];
            v0[0] = geglu(g0.x, u0.x, bg0, bu0); v1[0] = geglu(g1.x, u1.x, bg1, bu1);
            v0[1] = geglu(g0.y, u0.y, bg0, bu0); v1[1] = geglu(g1.y, u1.y, bg1, bu1);
            v0[2] = geglu(g0.z, u0.z, bg0, bu0); v1[2] = geglu(g1.z, u1.z, bg1, bu1);
            v0[3] = geglu(g0.w, u0.w, bg0, bu0); v1[3] = geglu(g1.w, u1.w, bg1, bu1);
          } else {
            const float4 s0 = sum4(2 * p, lm), s1 = sum4(2 * p + 1, lm);
            const float b0 = s_bias[2 * p], b1 = s_bias[2 * p + 1];
            v0[0] = finish1<kAct>(s0.x, b0, a.cap, mi == 0); v1[0] = finish1<kAct>(s1.x, b1, a.cap, mi == 0);
            v0[1] = finish1<kAct>(s0.y, b0, a.cap, mi == 0); v1[1] = finish1<kAct>(s1.y, b1, a.cap, mi == 0);
            v0[2] = finish1<kAct>(s0.z, b0, a.cap, mi == 0); v1[2] = finish1<kAct>(s1.z, b1, a.cap, mi == 0);
            v0[3] = finish1<kAct>(s0.w, b0, a.cap, mi == 0); v1[3] = finish1<kAct>(s1.w, b1, a.cap, mi == 0);
          }
#pragma unroll
          for (int j = 0; j < 4; ++j) {
            const int m = m_base + lm + j;
            if (m < M) {
              uint32_t y = pack_bf16x2(v0[j], v1[j]);
              if (a.residual != nullptr) y = badd2(y, res[j]);
              *reinterpret_cast<uint32_t*>(out + (int64_t)(row0 + m) * n_out + o) = y;
            }
          }
        }
      }
    } else {
      cluster_arrive();
    }
    cluster_wait();                                // and so has everything I sent
  } else if (warp_active) {
    // a single K slice: the output straight from tensor memory
    const bool f_ok = f < F && f0 + f < n;
    const bool upper = (lane & 1) != 0;
    if constexpr (kAct == kActGeglu) {
      // lanes 0-3 of 8 hold gates, 4-7 the values of the same features: they trade so that the first
      // finish even rows and the second odd ones, then neighbours trade to store two features
      const bool val = (lane & 4) != 0;
      const float b_own = f_ok ? s_bias[f] : 0.0f;
      const float b_other = __shfl_xor_sync(0xffffffffu, b_own, 4);
      const float bg = val ? b_other : b_own, bu = val ? b_own : b_other;
      const int n_out = n / 2;
      const int o = (f0 + f) / 8 * 4 + (lane & 2);
#pragma unroll 1
      for (int c = col0; c < col0 + cols && c < M; c += 16) {
        uint32_t acc[16];
        tc_ld_32x16(t_row + c, acc);
        tc_wait_ld();
#pragma unroll
        for (int j = 0; j < 16; j += 4) {
          float y[2];
#pragma unroll
          for (int k = 0; k < 2; ++k) {
            const float e0 = __uint_as_float(acc[j + 2 * k]), e1 = __uint_as_float(acc[j + 2 * k + 1]);
            const float got = __shfl_xor_sync(0xffffffffu, val ? e0 : e1, 4);
            y[k] = geglu(val ? got : e0, val ? e1 : got, bg, bu);
          }
          const float got = __shfl_xor_sync(0xffffffffu, upper ? y[0] : y[1], 1);
          const int m = c + j + (upper ? 2 : 0) + (val ? 1 : 0);
          if (f_ok && ok && m < M)
            *reinterpret_cast<uint32_t*>(out + (int64_t)(row0 + m) * n_out + o) =
                upper ? pack_bf16x2(got, y[1]) : pack_bf16x2(y[0], got);
        }
      }
    } else {
      const float b = f_ok ? s_bias[f] : 0.0f;
      const int o = f0 + (f & ~1);
#pragma unroll 1
      for (int c = col0; c < col0 + cols && c < M; c += 16) {
        uint32_t acc[16];
        tc_ld_32x16(t_row + c, acc);
        uint32_t res[8] = {};
        if (a.residual != nullptr) {
#pragma unroll
          for (int j = 0; j < 8; ++j) {
            const int m = c + 2 * j + (upper ? 1 : 0);
            if (f_ok && m < M) res[j] = *reinterpret_cast<const uint32_t*>(a.residual + (int64_t)(row0 + m) * n + o);
          }
        }
        tc_wait_ld();
#pragma unroll
        for (int j = 0; j < 8; ++j) {
          const float y0 = finish1<kAct>(__uint_as_float(acc[2 * j]), b, a.cap, mi == 0);
          const float y1 = finish1<kAct>(__uint_as_float(acc[2 * j + 1]), b, a.cap, mi == 0);
          const float got = __shfl_xor_sync(0xffffffffu, upper ? y0 : y1, 1);
          uint32_t y = upper ? pack_bf16x2(got, y1) : pack_bf16x2(y0, got);
          if (a.residual != nullptr) y = badd2(y, res[j]);
          const int m = c + 2 * j + (upper ? 1 : 0);
          if (f_ok && ok && m < M) *reinterpret_cast<uint32_t*>(out + (int64_t)(row0 + m) * n + o) = y;
        }
      }
    }
  }

  tc_fence_before();
  __syncthreads();
  if (threadIdx.x == 0 && *s_abort && status != nullptr) atomicExch(status, kStatusTimeout);
  if (warp == kEpiS + 1) {
    tc_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" :: "r"(tmem_base), "r"(a.tmem_cols)
                 : "memory");
  }
}

template <int kAct>
cudaError_t launch_small(const cudaLaunchConfig_t& cfg, const CUtensorMap& mx, const CUtensorMap (&mw)[3],
                         const SmallArgs& a, int* status) {
  return cudaLaunchKernelEx(&cfg, gemm_small_kernel<kAct>, mx, mw[0], mw[1], mw[2], a, status);
}

// How many clusters of c CTAs, one CTA per SM, the current device runs at once (clusters do not span
// GPCs, so this is less than SMs / c); looked up once per device.
const int* cluster_capacity() {
  static std::mutex mu;
  static int cache[64][kMaxClusterS + 1] = {};
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return nullptr;
  std::lock_guard<std::mutex> lock(mu);
  if (cache[dev][0] == 0) {
    for (int c = 2; c <= kMaxClusterS; ++c) {
      cudaLaunchAttribute attr[1];
      attr[0].id = cudaLaunchAttributeClusterDimension;
      attr[0].val.clusterDim.x = 1;
      attr[0].val.clusterDim.y = (unsigned)c;
      attr[0].val.clusterDim.z = 1;
      cudaLaunchConfig_t cfg = {};
      cfg.gridDim = dim3(1, (unsigned)c);
      cfg.blockDim = dim3(kThreadsS);
      cfg.dynamicSmemBytes = kDataS + kTailS;
      cfg.attrs = attr;
      cfg.numAttrs = 1;
      int n = 0;
      if (cudaOccupancyMaxActiveClusters(&n, gemm_small_kernel<0>, &cfg) != cudaSuccess) {
        cudaGetLastError();
        n = 0;
      }
      cache[dev][c] = n;
    }
    cache[dev][0] = 1;
  }
  return cache[dev];
}

// Ring and buffers for one choice of tile; false if they do not fit `budget`.
bool plan_smem(SmallArgs* a, int budget) {
  const int stage = (a->F + a->R) * 128;
  const int block = a->splits > 1 ? a->F * a->row_stride * 4 : 0;
  const int recv = (a->splits - 1) * block;
  int ns = (budget - recv) / stage;
  if (ns > kMaxStagesS) ns = kMaxStagesS;
  if (ns > a->kb_per_split) ns = a->kb_per_split;
  if (ns < 1 || (ns < 3 && ns < a->kb_per_split)) return false;
  // the partial sums lie over the ring; the instruction reads 128 rows of weights whatever F is
  int ring = ns * stage;
  if (ring < a->splits * block) ring = a->splits * block;
  const int reach = (ns - 1) * stage + 128 * 128;
  a->n_stages = ns;
  a->recv_off = ring;
  a->bar_off = ring + recv > reach ? ring + recv : reach;
  a->bar_off = (a->bar_off + 15) & ~15;
  return a->bar_off <= budget;
}

// Rows, F and K slices with the least expected time, in microseconds (constants from device-timer
// traces of the kernel): per K block a CTA takes what its loads need at 100 GB/s or what four
// instructions need (0.19 us up to 128 rows, 0.27 us at 256), 1 us goes by before the first block and
// behind the last one; all CTAs together need at least the weights' time at the HBM rate; the
// exchange costs 1.4 us and 0.2 ns per accumulator, the direct epilogue a third of that.
bool plan_tiles(SmallArgs* a, int n_mats, int* row_tiles, int num_sms) {
  const int* cap = cluster_capacity();
  if (cap == nullptr) return false;
  double best = 1e30, hbm = 0.0;
  for (int i = 0; i < n_mats; ++i) hbm += (double)a->mat[i].n * a->k_blocks * (SK * 2) / 6.4e6;
  SmallArgs pick = *a;
  int last = 0;
  for (int most = kRMax; most >= 64; most /= 2) {
    // the narrow operand's rows: a multiple of 16, of 32 from 64 on (the epilogue halves them)
    const int rows = (a->M + most - 1) / most, each = (a->M + rows - 1) / rows;
    if (rows == last) continue;
    last = rows;
    a->R = each <= 48 ? (each + 15) / 16 * 16 : (each + 31) / 32 * 32;
    for (int f = kFMax; f >= 32; f -= 8) {
      int tiles = 0, t1 = 0, t2 = 0;
      for (int i = 0; i < n_mats; ++i) {
        if (i == 1) t1 = tiles;
        if (i == 2) t2 = tiles;
        tiles += (a->mat[i].n + f - 1) / f;
      }
      for (int c = 1; c <= kMaxClusterS && c <= a->k_blocks; ++c) {
        SmallArgs p = *a;
        p.F = f;
        p.tile1 = n_mats > 1 ? t1 : tiles;
        p.tile2 = n_mats > 2 ? t2 : tiles;
        p.kb_per_split = (a->k_blocks + c - 1) / c;
        p.splits = (a->k_blocks + p.kb_per_split - 1) / p.kb_per_split;
        if (p.splits != c) continue;
        const int m_here = a->M < a->R ? a->M : a->R;
        p.rows_per_rank = ((m_here + c - 1) / c + 3) & ~3;
        p.row_stride = (p.rows_per_rank / 4) % 2 == 1 ? p.rows_per_rank : p.rows_per_rank + 4;
        const int slots = c == 1 ? num_sms : cap[c];
        if (slots < 1) continue;
        const int waves = (tiles * rows + slots - 1) / slots;
        const double loads = (f + a->R) / 800.0, mma = a->R <= 128 ? 0.19 : 0.19 + 0.08 * (a->R - 128) / 128;
        double cost = waves * (p.kb_per_split * (loads > mma ? loads : mma) + 1.0);
        if (cost < hbm) cost = hbm;
        cost += c > 1 ? 1.4 + 0.0002 * f * a->R : 0.5 + 0.00006 * f * a->R;
        if (cost >= best) continue;
        if (!plan_smem(&p, kDataHalfS) && !plan_smem(&p, kDataS)) continue;
        best = cost;
        pick = p;
        *row_tiles = rows;
      }
    }
  }
  *a = pick;
  return best < 1e30;
}

// The plan for a shape, remembered per thread (making one costs several microseconds of host time).
bool plan_for(SmallArgs* a, int n_mats, int* row_tiles, int num_sms) {
  struct Entry {
    int key[7];
    int rows;
    bool ok;
    SmallArgs plan;
  };
  constexpr int kEntries = 64;
  static thread_local Entry table[kEntries];      // key[6] = n_mats: 0 = empty
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess) return false;
  const int key[7] = {dev, a->M, a->k_blocks, a->mat[0].n, n_mats > 1 ? a->mat[1].n : 0,
                      n_mats > 2 ? a->mat[2].n : 0, n_mats};
  unsigned h = 0;
  for (int v : key) h = h * 1000003u + (unsigned)v;
  Entry& e = table[(h >> 8) % kEntries];
  bool same = true;
  for (int i = 0; i < 7; ++i) same = same && e.key[i] == key[i];
  if (!same) {
    e.plan = *a;
    e.ok = plan_tiles(&e.plan, n_mats, &e.rows, num_sms);
    for (int i = 0; i < 7; ++i) e.key[i] = key[i];
  }
  SmallArgs p = e.plan;                           // everything but the call's own pointers and options
  for (int i = 0; i < 3; ++i) p.mat[i] = a->mat[i];
  p.residual = a->residual;
  p.early = a->early;
  p.cap = a->cap;
  *a = p;
  *row_tiles = e.rows;
  return e.ok;
}

}  // namespace

bool dense_small_supported(int dtype, int64_t M, int64_t K, int64_t N) {
  return dtype == 1 && M >= 1 && M < (1 << 20) && K >= 8 && N >= 8 && K % 8 == 0 && N % 8 == 0 &&
         K < (1 << 28) && N < (1 << 28);
}

cudaError_t launch_dense_small(const void* x, const RowsMatrix* mats, int n_mats, const void* residual,
                               int64_t M, int K, int act, float cap, int* status, bool early, bool wide,
                               cudaStream_t s) {
  if (n_mats < 1 || n_mats > 3 || (n_mats > 1 && residual != nullptr)) return cudaErrorInvalidValue;
  if (act == 2 && (n_mats != 1 || residual != nullptr || mats[0].n % 128 != 0 || mats[0].bias == nullptr))
    return cudaErrorInvalidValue;
  if (cap != 0.0f && (n_mats != 1 || residual != nullptr || mats[0].bias != nullptr || act != 0))
    return cudaErrorInvalidValue;
  static PerDeviceOnce once;
  int num_sms = 0;
  cudaError_t e = once.run([] {
    cudaError_t r = cudaSuccess;
    auto set = [&](auto* kernel) {
      if (r == cudaSuccess)
        r = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kDataS + kTailS);
    };
    set(gemm_small_kernel<kActNone>);
    set(gemm_small_kernel<kActGelu>);
    set(gemm_small_kernel<kActGeglu>);
    set(gemm_small_kernel<kActCap>);
    return r;
  }, &num_sms);
  if (e != cudaSuccess) return e;

  SmallArgs a = {};
  for (int i = 0; i < 3; ++i) {
    const RowsMatrix& m = mats[i < n_mats ? i : 0];
    a.mat[i] = {static_cast<const __nv_bfloat16*>(m.bias), static_cast<__nv_bfloat16*>(m.out), m.n};
  }
  a.residual = static_cast<const __nv_bfloat16*>(residual);
  a.M = (int)M;
  a.k_blocks = (K + SK - 1) / SK;
  a.early = early ? 1 : 0;
  a.cap = cap;
  int rows = 1;
  if (!plan_for(&a, n_mats, &rows, num_sms)) return cudaErrorInvalidValue;
  a.tmem_cols = 32;
  while (a.tmem_cols < a.R) a.tmem_cols *= 2;

  CUtensorMap map_x, map_w[3];
  if (!tensor_map_2d(&map_x, x, (uint64_t)M, (uint64_t)K, (uint32_t)a.R, SK, true)) return cudaErrorInvalidValue;
  int tiles = 0;
  for (int i = 0; i < 3; ++i) {
    if (i >= n_mats) {
      map_w[i] = map_w[0];
      continue;
    }
    tiles += (mats[i].n + a.F - 1) / a.F;
    if (!tensor_map_2d(&map_w[i], mats[i].w, (uint64_t)mats[i].n, (uint64_t)K, (uint32_t)a.F, SK, true))
      return cudaErrorInvalidValue;
  }
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  attr[1].id = cudaLaunchAttributeClusterDimension;       // the K slices of a feature tile
  attr[1].val.clusterDim.x = 1;
  attr[1].val.clusterDim.y = (unsigned)a.splits;
  attr[1].val.clusterDim.z = 1;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)tiles, (unsigned)a.splits, (unsigned)rows);
  cfg.blockDim = dim3(kThreadsS);
  cfg.dynamicSmemBytes = (size_t)(a.bar_off + kTailS);
  if (wide && cfg.dynamicSmemBytes < kWideS) cfg.dynamicSmemBytes = kWideS;
  cfg.stream = s;
  cfg.attrs = attr;
  cfg.numAttrs = a.splits > 1 ? 2 : 1;
  if (cap != 0.0f) e = launch_small<kActCap>(cfg, map_x, map_w, a, status);
  else if (act == 2) e = launch_small<kActGeglu>(cfg, map_x, map_w, a, status);
  else if (act == 1) e = launch_small<kActGelu>(cfg, map_x, map_w, a, status);
  else e = launch_small<kActNone>(cfg, map_x, map_w, a, status);
  return e != cudaSuccess ? e : cudaGetLastError();
}

}  // namespace rgk
