// Dense projection out = x W^T + b (torch.nn.Linear as RecurrentBlock uses it, recurrentgemma
// torch/modules.py:531-548, 627-631, 647) on the 5th-generation tensor cores, bfloat16 in and out,
// float32 accumulation, optional gelu_tanh epilogue (the y branch, torch/modules.py:628).
//
// x [M, K] and W [N, K] are both K-contiguous, i.e. K-major operands as they are.  (Up to 128 rows of the
// logits go to single CTAs, see launch_dense_tc.)  Two CTAs of a
// cluster share one tile of 256 rows x BN columns (tcgen05.mma.cta_group::2, M 256): each brings its
// 128 rows of x and its HALF of the tile's columns of W (128 x 64 and BN/2 x 64 boxes, 128-byte
// swizzle) into a ring of its own and keeps the accumulator of its rows, so an SM reads 32 KB per K
// block of a 256-wide tile where a CTA by itself reads 48 KB.  At 32768 rows both kinds of tile are
// bound by what the SMs can fetch from L2 and by the power limit: 2560 x 2560 345 -> 284 us,
// 7680 -> 2560 924 -> 813 us, 2560 -> 15360 2407 -> 1934 us; at 3002 rows 38.0 -> 30.1 us,
// 95.7 -> 85.7 us, 228 -> 172 us.  One thread of the even CTA issues into one of two accumulators in
// the TMEM of both, and 16 epilogue warps per CTA drain the other: tcgen05.ld, + bias in float32, one
// rounding to bfloat16 (then gelu and a second rounding if asked, as torch does for a separate gelu
// op), a 32 x 32 transposition through shared memory and 64-byte-contiguous stores.  Persistent pairs
// walk the output tiles in groups of rows (kGroupRows); BN is chosen per call (tile_columns).
//
// Every mbarrier wait is bounded; on expiry WsHeader::status (if given) is raised and the CTA leaves.
#include <cuda.h>

#include "rgk_common.cuh"
#include "rgk_internal.h"
#include "tc_common.cuh"

namespace rgk {
namespace {

constexpr int BM = 128, BK = 64;                 // rows of a CTA (a pair: 256), K per stage
constexpr int kBnMax = 256;                      // columns of a tile at most
constexpr int kABytes = BM * BK * 2;             // 16 KiB
constexpr int kRingBytes = 192 * 1024;           // 6 stages of a 256-wide tile, 9 of a 64-wide one
constexpr int kMaxStages = 9;
constexpr int kEpi = 16;
constexpr int kThreadsG = (kEpi + 3) * 32;     // epilogue, two TMA producers around the MMA warp
constexpr int kOffRing = 0;
constexpr int kOffStageOut = kRingBytes;                         // per-warp 2 KiB staging
constexpr int kOffBarG = kOffStageOut + kEpi * 2048;             // full[] empty[] acc_full[2] acc_empty[2]
constexpr int kOffTmemG = kOffBarG + (2 * kMaxStages + 4) * 8;
constexpr int kOffAbortG = kOffTmemG + 4;
constexpr int kSmemG = kOffAbortG + 4 + 1024;
static_assert(kSmemG <= 232448, "exceeds the 227 KiB of shared memory a CTA may use");

// kMode 0: bias only; 1: gelu_tanh of the rounded result of the first matrix; 2: + residual (rounded again);
// 3: GeGLU - W holds, per group of 8 rows, 4 gate rows then the 4 value rows of the same features
//    (see pack_mlp_up_kernel: groups this small leave every kernel free to cut tiles at multiples of
//    8 rows); out [M, N/2] = gelu_tanh(gate) * value, where gate and
//    value are round(round(acc) + bias): the contraction and the bias add are two tensor operations
//    in the reference (torch/layers.py:700-703, torch/modules.py:749-751);
// 4: logits soft cap - round(tanh(round(round(acc) / cap)) * cap), the three tensor operations of
//    torch/griffin.py:183-185 after the contraction of torch/modules.py:1003.
// Where tile number `tile` lies: groups of `group` rows of tiles, m-fastest within a group and n-fastest
// across it.
__device__ __forceinline__ void tile_at(int tile, int m_tiles, int n_tiles, int group, int* m, int* n) {
  const int g = tile / (group * n_tiles), in = tile - g * group * n_tiles;
  const int rows = min(group, m_tiles - g * group);
  *n = in / rows;
  *m = g * group + in - *n * rows;
}

struct DenseMat {
  const __nv_bfloat16* bias;
  __nv_bfloat16* out;
  int n, tile0;                        // columns, number of the first tile
};
struct DenseArgs {
  DenseMat mat[3];                     // absent ones start behind the last tile
  const __nv_bfloat16* residual;
  int64_t M;
  int k_blocks, m_tiles, n_tiles, group, bn;
  int load_bytes;                      // what a CTA's loads of a stage bring
  float cap;
};

// kCtas = 1: a CTA by itself, tiles of 128 rows.
template <int kMode, int kCtas>
__global__ void __launch_bounds__(kThreadsG, 1)
gemm_tc_kernel(const __grid_constant__ CUtensorMap map_x, const __grid_constant__ CUtensorMap map_w0,
               const __grid_constant__ CUtensorMap map_w1, const __grid_constant__ CUtensorMap map_w2,
               const __grid_constant__ DenseArgs a, int* status) {
  extern __shared__ uint8_t smem_raw[];
  // aligned by an offset into the shared array, so that the address space stays known to the
  // compiler (shared-memory load/store instructions instead of generic ones)
  uint8_t* smem = smem_raw + ((1024u - (smem_u32(smem_raw) & 1023u)) & 1023u);
  const uint32_t s_base = smem_u32(smem);
  const uint32_t bar0 = s_base + kOffBarG;
  auto bar_full = [&](int s) { return bar0 + 8u * s; };
  auto bar_empty = [&](int s) { return bar0 + 8u * (kMaxStages + s); };
  auto bar_acc_full = [&](int s) { return bar0 + 8u * (2 * kMaxStages + s); };
  auto bar_acc_empty = [&](int s) { return bar0 + 8u * (2 * kMaxStages + 2 + s); };
  volatile uint32_t* s_tmem = reinterpret_cast<volatile uint32_t*>(smem + kOffTmemG);
  volatile int* s_abort = reinterpret_cast<volatile int*>(smem + kOffAbortG);

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int rank = kCtas == 2 ? (int)cluster_rank() : 0;   // cluster = (2, 1, 1)
  const int pair = blockIdx.x / kCtas, pairs = gridDim.x / kCtas;
  const int k_blocks = a.k_blocks, m_tiles = a.m_tiles, n_tiles = a.n_tiles, group = a.group, bn = a.bn;
  const int64_t M = a.M;
  const int n_my = (m_tiles * n_tiles - pair + pairs - 1) / pairs;
  const uint32_t stage_bytes = kABytes + (uint32_t)bn * (BK * 2 / kCtas);
  const int n_stages = min(kMaxStages, kRingBytes / (int)stage_bytes);

  if (threadIdx.x == 0) {
    *s_abort = 0;
    for (int s = 0; s < n_stages; ++s) { mbar_init(bar_full(s), 1); mbar_init(bar_empty(s), 1); }
    for (int s = 0; s < 2; ++s) { mbar_init(bar_acc_full(s), 1); mbar_init(bar_acc_empty(s), kCtas * kEpi); }
    mbar_fence_init();
  }
  if (warp == kEpi + 1) {
    if constexpr (kCtas == 2) {
      asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;"
                   :: "r"(s_base + kOffTmemG), "r"(512) : "memory");
      asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
    } else {
      asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;"
                   :: "r"(s_base + kOffTmemG), "r"(512) : "memory");
      asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
  }
  tc_fence_before();
  __syncthreads();
  if constexpr (kCtas == 2) {
    cluster_arrive();
    cluster_wait();                                // the peer's barriers are set up, its TMEM is there
  }
  tc_fence_after();
  const uint32_t tmem_base = *s_tmem;
  // everything up to here overlaps the kernel in front
  grid_dependency_wait();
  grid_launch_dependents();

  if (warp == kEpi || warp == kEpi + 2) {
    // ------------------------------ TMA producers -------------------------------------------------
    // Two, for even and odd K blocks: a turn of this loop takes one 340 cycles, as long as the MMAs of a
    // narrow tile's K blocks.  The whole warp runs it and one elected lane issues (see mma_ring).
    const uint32_t full0 = kCtas == 2 ? peer_smem(bar_full(0), 0) : bar_full(0);   // the loads of both report to the even one
    int kb = warp == kEpi ? 0 : 1, s = kb;
    uint32_t phase = 1;
    bool ok = true, ready = false;       // ready: the stage was already free when last asked
    for (int t = 0; t < n_my && ok; ++t) {
      int m0, n0;
      tile_at(pair + t * pairs, m_tiles, n_tiles, group, &m0, &n0);
      const int mi = (n0 >= a.mat[1].tile0) + (n0 >= a.mat[2].tile0);
      const CUtensorMap* map_w = mi == 0 ? &map_w0 : (mi == 1 ? &map_w1 : &map_w2);
      m0 = m0 * (kCtas * BM) + rank * BM;
      n0 = (n0 - (mi == 0 ? 0 : (mi == 1 ? a.mat[1].tile0 : a.mat[2].tile0))) * bn + rank * (bn / kCtas);
      for (; kb < k_blocks; kb += 2) {
        if (!ready) {
          ok = __all_sync(0xffffffffu, mbar_wait(bar_empty(s), phase, s_abort));
          if (!ok) break;
        }
        int next = s + 2;
        uint32_t next_phase = phase;
        if (next >= n_stages) { next -= n_stages; next_phase ^= 1; }
        const bool free_next = mbar_test(bar_empty(next), next_phase);   // looked at behind the loads
        if (elect_one()) {
          if (rank == 0) mbar_expect_tx(bar_full(s), kCtas * a.load_bytes);
          const uint32_t st = s_base + kOffRing + s * stage_bytes;
          if constexpr (kCtas == 2) {
            tma_load_2d_pair(st, &map_x, kb * BK, m0, full0 + 8u * s);
            tma_load_2d_pair(st + kABytes, map_w, kb * BK, n0, full0 + 8u * s);
          } else {
            tma_load_2d(st, &map_x, kb * BK, m0, full0 + 8u * s);
            tma_load_2d(st + kABytes, map_w, kb * BK, n0, full0 + 8u * s);
          }
        }
        __syncwarp();
        ready = __all_sync(0xffffffffu, free_next);
        s = next;
        phase = next_phase;
      }
      kb -= k_blocks;
    }
  } else if (warp == kEpi + 1) {
    // ------------------------------ MMA issue: the even CTA for both -------------------------------
    if (rank == 0) {
      RingPos at;
      bool ok = true;
      for (int t = 0; t < n_my; ++t) {
        const int as = t & 1;
        const uint32_t parity = ((t >> 1) & 1) ^ 1;
        ok = __all_sync(0xffffffffu, kCtas == 2 ? mbar_wait_cluster(bar_acc_empty(as), parity, s_abort)
                                                : mbar_wait(bar_acc_empty(as), parity, s_abort));
        if (!ok) break;
        tc_fence_after();
        ok = mma_ring<BK / 16, kCtas>(tmem_base + as * kBnMax, smem_desc_sw128(s_base + kOffRing),
                                  smem_desc_sw128(s_base + kOffRing + kABytes), stage_bytes >> 4,
                                  tc_idesc_bf16(kCtas * BM, bn), k_blocks, n_stages, bar_full(0), bar_empty(0),
                                  at, s_abort);
        if (!ok) break;
        if (elect_one()) {
          if constexpr (kCtas == 2) tc_commit_pair(bar_acc_full(as));
          else tc_commit(bar_acc_full(as));
        }
        __syncwarp();
      }
    }
  } else {
    // ------------------------------ epilogue ------------------------------------------------------
    // all warps on every tile: what a pair does behind its last MMA is as short as it can be
    const int lane_base = (warp & 3) * 32;   // TMEM lanes this warp may read
    const int col_group = warp >> 2;         // takes every fourth group of columns
    uint8_t* stage = smem + kOffStageOut + warp * 2048;
    bool ok = true;
    for (int t = 0; t < n_my && ok; ++t) {
      const int as = t & 1;                  // accumulator
      int mt, n0;
      tile_at(pair + t * pairs, m_tiles, n_tiles, group, &mt, &n0);
      const int64_t m0 = (int64_t)mt * (kCtas * BM) + rank * BM;
      // (copies, so that nothing indexes the parameters dynamically)
      const int mi = (n0 >= a.mat[1].tile0) + (n0 >= a.mat[2].tile0);
      const __nv_bfloat16* bias = mi == 0 ? a.mat[0].bias : (mi == 1 ? a.mat[1].bias : a.mat[2].bias);
      __nv_bfloat16* out = mi == 0 ? a.mat[0].out : (mi == 1 ? a.mat[1].out : a.mat[2].out);
      const int N = mi == 0 ? a.mat[0].n : (mi == 1 ? a.mat[1].n : a.mat[2].n);
      n0 = (n0 - (mi == 0 ? 0 : (mi == 1 ? a.mat[1].tile0 : a.mat[2].tile0))) * bn;
      // bias and residual of a chunk of 32 columns, the latter as the pieces this thread will add
      // after the transposition; the first chunk's are loaded ahead of the wait for the accumulator
      [[maybe_unused]] uint32_t bv[16];
      [[maybe_unused]] uint4 rv[4];
      auto load_chunk = [&](int cc) {
        const int nc = n0 + cc * 32;
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          uint4 b4 = make_uint4(0u, 0u, 0u, 0u);
          if (bias != nullptr && nc + 8 * j < N) b4 = *reinterpret_cast<const uint4*>(bias + nc + 8 * j);
          bv[4 * j] = b4.x; bv[4 * j + 1] = b4.y; bv[4 * j + 2] = b4.z; bv[4 * j + 3] = b4.w;
        }
        if constexpr (kMode == 2) {
#pragma unroll
          for (int k = 0; k < 4; ++k) {
            const int64_t grow = m0 + lane_base + (lane >> 2) + 8 * k;
            const int gcol = nc + (lane & 3) * 8;
            rv[k] = (grow < M && gcol < N) ? ld_stream(a.residual + grow * N + gcol)
                                           : make_uint4(0u, 0u, 0u, 0u);
          }
        }
      };
      if constexpr (kMode != 3) {
        if (col_group < bn / 32) load_chunk(col_group);
      }
      ok = mbar_wait(bar_acc_full(as), (t >> 1) & 1, s_abort);
      if (!ok) break;
      tc_fence_after();
      const uint32_t t_row = tmem_base + (static_cast<uint32_t>(lane_base) << 16) + as * kBnMax;
      if constexpr (kMode == 3) {
        const int n_out = N / 2;
        const int oc0 = n0 / 2;                // first output feature of the tile
#pragma unroll 1
        for (int cc = col_group; cc < bn / 64; cc += 4) {   // 32 features at a time
          uint4 ov[4];
#pragma unroll
          for (int hf = 0; hf < 2; ++hf) {     // 32 columns = 16 features: bounded register use
            uint32_t acc[32];
            tc_ld_32x32(t_row + cc * 64 + hf * 32, acc);
            const int nb = n0 + cc * 64 + hf * 32;
            uint4 bv[4];                       // 4 gate biases, then 4 value biases
#pragma unroll
            for (int j = 0; j < 4; ++j) bv[j] = nb + 8 * j < N ? *reinterpret_cast<const uint4*>(bias + nb + 8 * j)
                                                               : make_uint4(0u, 0u, 0u, 0u);
            tc_wait_ld();
            uint32_t o[8];
#pragma unroll
            for (int j = 0; j < 4; ++j) {
#pragma unroll
              for (int p = 0; p < 2; ++p) {
                const int n = j * 8 + p * 2;
                const uint32_t g2 = badd2(pack_bf16x2(__uint_as_float(acc[n]), __uint_as_float(acc[n + 1])),
                                          p == 0 ? bv[j].x : bv[j].y);
                const uint32_t v2 = badd2(pack_bf16x2(__uint_as_float(acc[n + 4]), __uint_as_float(acc[n + 5])),
                                          p == 0 ? bv[j].z : bv[j].w);
                const uint32_t a2 = pack_bf16x2(gelu_tanh_<true>(bf16_lo(g2)), gelu_tanh_<true>(bf16_hi(g2)));
                o[j * 2 + p] = bmul2(a2, v2);
              }
            }
            ov[hf * 2] = make_uint4(o[0], o[1], o[2], o[3]);
            ov[hf * 2 + 1] = make_uint4(o[4], o[5], o[6], o[7]);
          }
#pragma unroll
          for (int j = 0; j < 4; ++j)
            *reinterpret_cast<uint4*>(stage + lane * 64 + ((j ^ ((lane >> 1) & 3)) << 4)) = ov[j];
          __syncwarp();
#pragma unroll
          for (int k = 0; k < 4; ++k) {
            const int r = (lane >> 2) + 8 * k, piece = lane & 3;
            const uint4 v = *reinterpret_cast<const uint4*>(stage + r * 64 + ((piece ^ ((r >> 1) & 3)) << 4));
            const int64_t grow = m0 + lane_base + r;
            const int gcol = oc0 + cc * 32 + piece * 8;
            if (grow < M && gcol < n_out) *reinterpret_cast<uint4*>(out + grow * n_out + gcol) = v;
          }
          __syncwarp();
        }
      } else {
#pragma unroll 1
      for (int cc = col_group; cc < bn / 32; cc += 4) {
        uint32_t acc[32];
        tc_ld_32x32(t_row + cc * 32, acc);
        const int nc = n0 + cc * 32;         // first output column of this chunk
        tc_wait_ld();
        uint4 ov[4];
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          uint32_t o[4];
#pragma unroll
          for (int p = 0; p < 4; ++p) {
            const int n = j * 8 + p * 2;
            const uint32_t b2 = bv[j * 4 + p];
            float v0 = __uint_as_float(acc[n]) + bf16_lo(b2), v1 = __uint_as_float(acc[n + 1]) + bf16_hi(b2);
            uint32_t pk = pack_bf16x2(v0, v1);
            if (kMode == 1 && mi == 0) pk = pack_bf16x2(gelu_tanh_<true>(bf16_lo(pk)), gelu_tanh_<true>(bf16_hi(pk)));
            if constexpr (kMode == 4) {
              const float cap = a.cap;
              uint32_t t = pack_bf16x2(__fdiv_rn(bf16_lo(pk), cap), __fdiv_rn(bf16_hi(pk), cap));
              t = pack_bf16x2(tanhf(bf16_lo(t)), tanhf(bf16_hi(t)));
              pk = pack_bf16x2(bf16_lo(t) * cap, bf16_hi(t) * cap);
            }
            o[p] = pk;
          }
          ov[j] = make_uint4(o[0], o[1], o[2], o[3]);
        }
        // 32 x 32 transposition through the warp's staging buffer (see gates_tc.cu), then stores of
        // 8 rows x 64 contiguous bytes per instruction.
#pragma unroll
        for (int j = 0; j < 4; ++j)
          *reinterpret_cast<uint4*>(stage + lane * 64 + ((j ^ ((lane >> 1) & 3)) << 4)) = ov[j];
        __syncwarp();
#pragma unroll
        for (int k = 0; k < 4; ++k) {
          const int r = (lane >> 2) + 8 * k, piece = lane & 3;
          uint4 v = *reinterpret_cast<const uint4*>(stage + r * 64 + ((piece ^ ((r >> 1) & 3)) << 4));
          const int64_t grow = m0 + lane_base + r;
          const int gcol = nc + piece * 8;
          if (grow < M && gcol < N) {
            if constexpr (kMode == 2) {
              // the residual stream joins here: round(round(acc + bias) + residual), the two tensor
              // operations of the reference (torch/modules.py:899-902)
              v = make_uint4(badd2(v.x, rv[k].x), badd2(v.y, rv[k].y), badd2(v.z, rv[k].z),
                             badd2(v.w, rv[k].w));
            }
            *reinterpret_cast<uint4*>(out + grow * N + gcol) = v;
          }
        }
        if (cc + 4 < bn / 32) load_chunk(cc + 4);
        __syncwarp();
      }
      }
      tc_fence_before();
      __syncwarp();
      if (lane == 0) {
        if constexpr (kCtas == 2) mbar_arrive_cluster(peer_smem(bar_acc_empty(as), 0));
        else mbar_arrive(bar_acc_empty(as));
      }
    }
  }

  tc_fence_before();
  __syncthreads();
  if (threadIdx.x == 0 && *s_abort && status != nullptr) atomicExch(status, kStatusTimeout);
  if constexpr (kCtas == 2) {
    cluster_arrive();
    cluster_wait();                                // the peer signals this CTA no more
  }
  if (warp == kEpi + 1) {
    tc_fence_after();
    if constexpr (kCtas == 2)
      asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" :: "r"(tmem_base), "r"(512)
                   : "memory");
    else
      asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" :: "r"(tmem_base), "r"(512)
                   : "memory");
  }
}

// ffw_up of the MLP block: w [2, D, X] (in, out) and b [2, X] into the K-major, gate/value
// interleaved layout of mode 3: packed row g*8 + c*4 + i = column (feature) g*4 + i of w[c].
__global__ void pack_mlp_up_kernel(const __nv_bfloat16* __restrict__ w, const __nv_bfloat16* __restrict__ b,
                                   int D, int X, __nv_bfloat16* __restrict__ packed_w,
                                   __nv_bfloat16* __restrict__ packed_b) {
  __shared__ __nv_bfloat16 tile[32][33];
  // grid: (D / 32 rounded up, X / 32, 2); block 32 x 8
  const int c = blockIdx.z, k0 = blockIdx.x * 32, f0 = blockIdx.y * 32;
  const __nv_bfloat16* src = w + (int64_t)c * D * X;
  for (int r = threadIdx.y; r < 32; r += 8) {                      // r walks k, x walks features
    const int k = k0 + r, f = f0 + threadIdx.x;
    tile[r][threadIdx.x] = (k < D && f < X) ? src[(int64_t)k * X + f] : __float2bfloat16(0.0f);
  }
  __syncthreads();
  for (int r = threadIdx.y; r < 32; r += 8) {                      // r walks features, x walks k
    const int f = f0 + r, k = k0 + threadIdx.x;
    if (f < X && k < D) {
      const int64_t row = (int64_t)(f / 4) * 8 + c * 4 + (f % 4);
      packed_w[row * D + k] = tile[threadIdx.x][r];
      if (k == 0) packed_b[row] = b[(int64_t)c * X + f];
    }
  }
}



// Columns of a tile: the width with the least expected time.  A wave (one tile per pair) takes, per 40
// K blocks, 8.2, 8.6, 9.3 and 12.5 us at 64, 128, 192 and 256 columns - up to 192 the time to fetch
// the operands from L2 (16 KB of x whatever the width), from there on the MMAs themselves.  So a tall
// problem takes 256, and a short one the width that fills the last wave.  The GeGLU epilogue works on
// 64 columns at a time, the others on 32.
int tile_columns(int64_t m_tiles, const RowsMatrix* mats, int n_mats, int pairs, int step) {
  int best = kBnMax;
  double least = 1e300;
  for (int bn = kBnMax; bn >= 64; bn -= step) {
    int64_t tiles = 0;
    for (int i = 0; i < n_mats; ++i) tiles += (mats[i].n + bn - 1) / bn;
    tiles *= m_tiles;
    const double wave = bn <= 192 ? 7.7 + bn / 120.0 : 9.3 + (bn - 192) / 20.0;
    const double t = (double)((tiles + pairs - 1) / pairs) * wave;
    if (t < least) { least = t; best = bn; }
  }
  return best;
}

// Rows of tiles that a group takes: the pairs running together then read about as many rows of x as
// of W, where the same number of tiles in one row would read all of W for each of them (2560 -> 15360
// at 3002 rows 180 -> 162 us, at 8192 445 -> 405 us; 8 to 16 make no difference).
constexpr int kGroupRows = 12;

}  // namespace

bool dense_tc_supported(int dtype, int64_t M, int64_t K, int64_t N) {
  return dtype == 1 && M >= 1 && M < ((int64_t)1 << 31) && K >= 8 && K % 8 == 0 && N >= 8 &&
         N % 8 == 0 && K < (1 << 24) && N < (1 << 24);
}

cudaError_t launch_dense_tc(const void* x, const RowsMatrix* mats, int n_mats, const void* residual, int64_t M,
                            int K, int act, int* status, cudaStream_t s, float cap) {
  if (M == 0) return cudaSuccess;
  if (n_mats < 1 || n_mats > 3 || (n_mats > 1 && (act == 2 || residual != nullptr || cap != 0.0f)))
    return cudaErrorInvalidValue;
  if ((act != 0) + (residual != nullptr) > 1) return cudaErrorInvalidValue;
  if (cap != 0.0f && (act != 0 || residual != nullptr || mats[0].bias != nullptr)) return cudaErrorInvalidValue;
  static PerDeviceOnce once;
  int num_sms = 0;
  cudaError_t e = once.run([] {
    cudaError_t r = cudaSuccess;
    auto set = [&](auto* kernel) {
      if (r == cudaSuccess)
        r = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmemG);
    };
    set(gemm_tc_kernel<0, 2>);
    set(gemm_tc_kernel<1, 2>);
    set(gemm_tc_kernel<2, 2>);
    set(gemm_tc_kernel<3, 2>);
    set(gemm_tc_kernel<4, 2>);
    set(gemm_tc_kernel<0, 1>);
    set(gemm_tc_kernel<4, 1>);
    return r;
  }, &num_sms);
  if (e != cudaSuccess) return e;
  // One tile of 128 rows is left to single CTAs where nothing but the cap follows the contraction: half of a
  // pair would work on rows that do not exist, and a pair has 96 KB of weights in flight an SM where a CTA
  // by itself has 128 (logits of 64 rows over 256000 tokens 306 -> 226 us, over 32000 53 -> 42).
  const int ctas = M <= BM && n_mats == 1 && act == 0 && residual == nullptr ? 1 : 2;
  const int64_t m_tiles = (M + ctas * BM - 1) / (ctas * BM);
  DenseArgs a = {};
  a.bn = tile_columns(m_tiles, mats, n_mats, num_sms / ctas, act == 2 ? 64 : 32);
  int64_t n_tiles = 0;
  CUtensorMap map_x, map_w[3];
  // rows that do not exist are not asked for where there is one tile of rows: filling them with zeros slows
  // the loads (16 rows of the above 298 -> 219 us), and what the instruction reads in their place reaches
  // only rows that are not stored
  const int box_m = ctas == 1 ? (int)M : BM;
  a.load_bytes = (box_m + a.bn / ctas) * (BK * 2);
  if (!tensor_map_2d(&map_x, x, (uint64_t)M, (uint64_t)K, (uint32_t)box_m, BK, true)) return cudaErrorInvalidValue;
  for (int i = 0; i < n_mats; ++i) {
    a.mat[i] = {static_cast<const __nv_bfloat16*>(mats[i].bias), static_cast<__nv_bfloat16*>(mats[i].out),
                mats[i].n, (int)n_tiles};
    n_tiles += (mats[i].n + a.bn - 1) / a.bn;
    if (!tensor_map_2d(&map_w[i], mats[i].w, (uint64_t)mats[i].n, (uint64_t)K, (uint32_t)(a.bn / ctas), BK, true))
      return cudaErrorInvalidValue;
  }
  for (int i = n_mats; i < 3; ++i) {
    a.mat[i].tile0 = 0x7fffffff;
    map_w[i] = map_w[0];
  }
  if (m_tiles * n_tiles > 0x7fffffff) return cudaErrorInvalidValue;
  const int64_t total = m_tiles * n_tiles, groups = (m_tiles + kGroupRows - 1) / kGroupRows;
  a.residual = static_cast<const __nv_bfloat16*>(residual);
  a.M = M;
  a.k_blocks = (K + BK - 1) / BK;
  a.m_tiles = (int)m_tiles;
  a.n_tiles = (int)n_tiles;
  a.group = (int)((m_tiles + groups - 1) / groups);
  a.cap = cap;
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  attr[1].id = cudaLaunchAttributeClusterDimension;
  attr[1].val.clusterDim.x = 2;
  attr[1].val.clusterDim.y = attr[1].val.clusterDim.z = 1;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)(ctas * (total < num_sms / ctas ? total : num_sms / ctas)));
  cfg.blockDim = dim3(kThreadsG);
  cfg.dynamicSmemBytes = kSmemG;
  cfg.stream = s;
  cfg.attrs = attr;
  cfg.numAttrs = ctas;                             // (a CTA by itself has no cluster)
#define RGK_GEMM(MODE, CTAS) \
  cudaLaunchKernelEx(&cfg, gemm_tc_kernel<MODE, CTAS>, map_x, map_w[0], map_w[1], map_w[2], a, status)
  if (ctas == 1) e = cap != 0.0f ? RGK_GEMM(4, 1) : RGK_GEMM(0, 1);
  else e = cap != 0.0f ? RGK_GEMM(4, 2) : act == 2 ? RGK_GEMM(3, 2) : act == 1 ? RGK_GEMM(1, 2)
                       : residual != nullptr ? RGK_GEMM(2, 2) : RGK_GEMM(0, 2);
#undef RGK_GEMM
  return e != cudaSuccess ? e : cudaGetLastError();
}

cudaError_t launch_pack_mlp_up(const void* w, const void* b, int D, int X, void* packed_w,
                               void* packed_b, cudaStream_t s) {
  using T_ = __nv_bfloat16;
  const dim3 grid((unsigned)((D + 31) / 32), (unsigned)((X + 31) / 32), 2), block(32, 8);
  pack_mlp_up_kernel<<<grid, block, 0, s>>>((const T_*)w, (const T_*)b, D, X, (T_*)packed_w,
                                           (T_*)packed_b);
  return cudaGetLastError();
}

}  // namespace rgk
