// Block-diagonal gate projections of the RG-LRU in float32 on the 5th-generation tensor cores,
// fused with the gate arithmetic (recurrentgemma torch/layers.py:127-137, 338-353), for heads of
// width 256.
//
// The tensor cores have no float32 multiply; kind::tf32 reads the upper 19 bits of a float32
// (10 mantissa bits).  A float32 product is recovered to well below the 1e-5 parity bar from three
// TF32 products with a float32 accumulator ("3xTF32"):
//     x w  ~  x_hi w_hi + x_lo w_hi + x_hi w_lo,     v_hi = v with the low 13 mantissa bits cleared,
//                                                    v_lo = v - v_hi (exact in float32)
// (the dropped x_lo w_lo term is below 2^-22 of the product).  The activations are split on chip, per
// K-slice, by the warps that later run the epilogue (hi written back over the slice the copy engine
// delivered, lo beside it); the weights are split by a packing kernel into two K-major arrays.
//
// A CTA takes 128 tokens x kTN accumulator columns: the x-gate and the a-gate outputs of kTN / 2
// channels, so that an epilogue thread finds both gates of a channel in its own TMEM lane.  K = 256
// arrives in sixteen slices of 16 (64-byte rows, 64-byte swizzle) through a ring: activations 8 KiB, their
// low part 8 KiB (written by the helper warps), weights hi and lo 16 KiB each (kTN = 256) - the
// per-slice hand-offs (copy engine -> split -> tensor core -> release) of a CTA are serial, so more and
// smaller stages in flight hide them.  One warp runs the MMA loop, an elected lane issues three
// tcgen05.mma.cta_group::1.kind::tf32 (M 128, N kTN, K 8) per K step.  The epilogue (TMEM lane quarter x 32-channel chunks per warp) reads the
// accumulators, applies the float32-accurate gate arithmetic and writes a and the normalised input for
// the scan kernel.
//
// A tile costs some 640 KB of fetches, 6 us of contraction and 8 us of arithmetic (a hundred instructions
// an element); with several tiles per SM two CTAs share it and overlap them (launch_gates_tf32).  (A
// persistent form on pairs of CTAs, with warps of its own for the split, was slower: 1 us per slice.)
//
// Every mbarrier wait is bounded; on expiry WsHeader::status is raised and the CTA leaves.
#include <cuda.h>

#include "rgk_common.cuh"
#include "rgk_internal.h"
#include "tc_common.cuh"

namespace rgk {
namespace {

constexpr int kHW = 256;                 // head width = K
constexpr int kTM = 128;                 // tokens per tile (MMA M)
constexpr int kHalf = 128;               // channels of a group of packed weights (256 rows: both gates)
constexpr int kKS = 16;                  // K per slice: 16 float32 = 64 bytes (64-byte swizzle)
constexpr int kSlices = kHW / kKS;
constexpr int kABytes = kTM * kKS * 4;
// kTN = 256 or 128 accumulator columns: both gates of kTN / 2 channels; kPerSm CTAs share an SM
template <int kTN, int kPerSm>
struct Cfg {
  static constexpr int kEpi = kPerSm == 1 ? 16 : 8;
  static constexpr int kThreads = (kEpi + 2) * 32;
  static constexpr int kStages = kPerSm == 1 ? 4 : (kTN == 256 ? 2 : 3);
  static constexpr int kBBytes = kTN * kKS * 4;
  static constexpr int kStageBytes = 2 * kABytes + 2 * kBBytes;     // A, A_lo, B_hi, B_lo
  static constexpr int kOffSp = kStages * kStageBytes;              // float [3][kTN / 2]: softplus(a_param), gate biases
  static constexpr int kOffBar = kOffSp + 3 * (kTN / 2) * 4;        // full, lo_full, empty [stage], acc_full
  static constexpr int kOffTmem = kOffBar + (3 * kStages + 1) * 8;
  static constexpr int kOffAbort = kOffTmem + 4;
  static constexpr int kSmem = kOffAbort + 4 + 1024;
  static_assert(kPerSm * (kSmem + 1024) <= 233472, "too much shared memory");
  static_assert(kEpi * 8192 <= kStages * kStageBytes, "the epilogue's blocks lie over the ring");
};

// Instruction descriptor of tcgen05.mma kind::tf32: D float32, A and B TF32, both K-major.
constexpr uint32_t tc_idesc_tf32(int m, int n) {
  return (1u << 4) | (2u << 7) | (2u << 10) | ((uint32_t)(n >> 3) << 17) | ((uint32_t)(m >> 4) << 24);
}

__device__ __forceinline__ void tc_mma_tf32(uint32_t d_tmem, uint64_t a_desc, uint64_t b_desc,
                                            uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::tf32 [%0], %1, %2, %3, p;\n\t}"
      :: "r"(d_tmem), "l"(a_desc), "l"(b_desc), "r"(idesc), "r"(accumulate) : "memory");
}

// The place of a launch among those that share the tiles of a call.
enum { kAlone = 0, kFirst = 1, kSecond = 2 };

// v with the low 13 mantissa bits cleared (an exact TF32 value), and the rest of v (exact).
__device__ __forceinline__ float tf32_high_part(float v) {
  return __uint_as_float(__float_as_uint(v) & 0xffffe000u);
}
__device__ __forceinline__ float tf32_low_part(float v) { return v - tf32_high_part(v); }

template <int kTN, int kPerSm>
__global__ void __launch_bounds__((Cfg<kTN, kPerSm>::kThreads), kPerSm)
gates_tf32_kernel(const __grid_constant__ CUtensorMap map_x, const __grid_constant__ CUtensorMap map_wh,
                  const __grid_constant__ CUtensorMap map_wl, const float* x,
                  const void* pos, int pos64, const float* __restrict__ a_param,
                  const float* __restrict__ bias_x, const float* __restrict__ bias_a, int64_t M,
                  int E, float* __restrict__ a_out, float* __restrict__ xn_out, WsHeader* hdr, const ScanPrep prep,
                  int first_tile, int order) {
  using C = Cfg<kTN, kPerSm>;
  constexpr int kEpi = C::kEpi;
  constexpr int kStages = C::kStages, kBBytes = C::kBBytes, kStageBytes = C::kStageBytes;
  constexpr int kChans = kTN / 2;
  constexpr uint32_t kIdescF = tc_idesc_tf32(kTM, kTN);
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = smem_raw + ((1024u - (smem_u32(smem_raw) & 1023u)) & 1023u);
  const uint32_t s_base = smem_u32(smem);
  const uint32_t bar0 = s_base + C::kOffBar;
  auto bar_full = [&](int s) { return bar0 + 8u * s; };
  auto bar_lo = [&](int s) { return bar0 + 8u * (kStages + s); };
  auto bar_empty = [&](int s) { return bar0 + 8u * (2 * kStages + s); };
  const uint32_t bar_acc = bar0 + 8u * (3 * kStages);
  float* s_sp = reinterpret_cast<float*>(smem + C::kOffSp);
  volatile uint32_t* s_tmem = reinterpret_cast<volatile uint32_t*>(smem + C::kOffTmem);
  volatile int* s_abort = reinterpret_cast<volatile int*>(smem + C::kOffAbort);

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int n_tiles = E / kChans, index = first_tile + blockIdx.x;
  const int tile = index / n_tiles, chan0 = (index - tile * n_tiles) * kChans;
  const int head = chan0 / kHW;
  const int wrow = chan0 / kHalf * (2 * kHalf) + chan0 % kHalf;      // packed rows: x-gate, kHalf behind a-gate

  if (threadIdx.x == 0) {
    *s_abort = 0;
    for (int s = 0; s < kStages; ++s) {
      mbar_init(bar_full(s), 1);
      mbar_init(bar_lo(s), kEpi);
      mbar_init(bar_empty(s), 1);
    }
    mbar_init(bar_acc, 1);
    mbar_fence_init();
  }
  if (warp == kEpi + 1) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;"
                 :: "r"(s_base + C::kOffTmem), "r"(kTN) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  // (the second of two launches starts when every CTA of the first has passed its own wait)
  if (order != kSecond) grid_dependency_wait();
  if (order == kFirst) grid_launch_dependents();
  if (prep.ticket != nullptr) {                              // for the scan kernel behind
    if (blockIdx.x == 0 && threadIdx.x == 0) *prep.ticket = 0u;
    for (int64_t i = (int64_t)blockIdx.x * C::kThreads + threadIdx.x; i < prep.n_zero;
         i += (int64_t)gridDim.x * C::kThreads)
      prep.zero[i] = make_uint4(0u, 0u, 0u, 0u);
  }
  if (threadIdx.x < kChans) {
    s_sp[threadIdx.x] = softplus_(a_param[chan0 + threadIdx.x]);
    s_sp[kChans + threadIdx.x] = bias_x[chan0 + threadIdx.x];
    s_sp[2 * kChans + threadIdx.x] = bias_a[chan0 + threadIdx.x];
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *s_tmem;

  if (warp == kEpi) {
    // ------------------------------ TMA producer --------------------------------------------------
    if (lane == 0) {
      bool ok = true;
      for (int kb = 0; kb < kSlices && ok; ++kb) {
        const int s = kb % kStages;
        ok = mbar_wait(bar_empty(s), ((kb / kStages) & 1) ^ 1, s_abort);
        if (!ok) break;
        const uint32_t st = s_base + s * kStageBytes;
        mbar_expect_tx(bar_full(s), kABytes + 2 * kBBytes);
        tma_load_2d(st, &map_x, head * kHW + kb * kKS, tile * kTM, bar_full(s));
#pragma unroll
        for (int g = 0; g < 2; ++g) {                      // x-gate rows, a-gate rows
          const uint32_t w = st + 2 * kABytes + g * (kBBytes / 2);
          tma_load_2d(w, &map_wh, kb * kKS, wrow + g * kHalf, bar_full(s));
          tma_load_2d(w + kBBytes, &map_wl, kb * kKS, wrow + g * kHalf, bar_full(s));
        }
      }
    }
  } else if (warp == kEpi + 1) {
    // ------------------------------ MMA issue -----------------------------------------------------
    // (the whole warp runs the loop, one elected lane issues: see mma_ring)
    const uint64_t desc_a = smem_desc_sw64(s_base), desc_b = smem_desc_sw64(s_base + 2 * kABytes);
    bool ok = true;
    int s = 0;
    uint32_t phase = 0;
    for (int kb = 0; kb < kSlices; ++kb) {
      ok = mbar_wait(bar_full(s), phase, s_abort);
      if (ok) ok = mbar_wait(bar_lo(s), phase, s_abort);
      ok = __all_sync(0xffffffffu, ok);
      if (!ok) break;
      tc_fence_after();
      if (elect_one()) {
        const uint64_t st = (uint64_t)(s * (kStageBytes >> 4));
        const uint64_t dah = desc_a + st, dal = dah + (kABytes >> 4), dbh = desc_b + st, dbl = dbh + (kBBytes >> 4);
#pragma unroll
        for (int ks = 0; ks < kKS / 8; ++ks) {
          tc_mma_tf32(tmem_base, dah + 2 * ks, dbh + 2 * ks, kIdescF, (kb | ks) != 0 ? 1u : 0u);
          tc_mma_tf32(tmem_base, dal + 2 * ks, dbh + 2 * ks, kIdescF, 1u);
          tc_mma_tf32(tmem_base, dah + 2 * ks, dbl + 2 * ks, kIdescF, 1u);
        }
        tc_commit(bar_empty(s));
        if (kb == kSlices - 1) tc_commit(bar_acc);
      }
      __syncwarp();
      if (++s == kStages) { s = 0; phase ^= 1; }
    }
  } else {
    // ------------------------------ helper, then epilogue ------------------------------------------
    // During the main loop: the low parts of the activation slice (element-wise, so the swizzled
    // layout carries over address for address).  512 threads cover one 128-token slice.
    bool ok = true;
    for (int kb = 0; kb < kSlices && ok; ++kb) {
      const int s = kb % kStages;
      ok = mbar_wait(bar_full(s), (kb / kStages) & 1, s_abort);
      if (!ok) break;
      constexpr int kPer = kABytes / 16 / (kEpi * 32);          // 16-byte pieces per thread
      float4* src = reinterpret_cast<float4*>(smem + s * kStageBytes) + threadIdx.x * kPer;
      float4* dst = reinterpret_cast<float4*>(smem + s * kStageBytes + kABytes) + threadIdx.x * kPer;
#pragma unroll
      for (int i = 0; i < kPer; ++i) {
        const float4 v = src[i];
        dst[i] = make_float4(tf32_low_part(v.x), tf32_low_part(v.y), tf32_low_part(v.z),
                             tf32_low_part(v.w));
        // the high part is written back explicitly, so that the split does not depend on how the
        // tensor core narrows a float32 operand (an exact TF32 value passes unchanged either way)
        src[i] = make_float4(tf32_high_part(v.x), tf32_high_part(v.y), tf32_high_part(v.z),
                             tf32_high_part(v.w));
      }
      fence_proxy_async();                  // the tensor core reads this through the async proxy
      __syncwarp();
      if (lane == 0) mbar_arrive(bar_lo(s));
    }
    // Epilogue: thread = token row of the warp's TMEM lane quarter, 32 channels of the half.
    // Global traffic goes through two per-warp 32 x 32 float32 blocks in the (now idle) ring, so that
    // a load or store instruction moves four rows x 128 contiguous bytes instead of 32 rows x 16
    // bytes: 16-byte piece j of row r sits at piece j ^ (r & 7), conflict-free both for the row
    // owner (lane = row) and for the copy pattern (8 lanes per row).
    const int lane_base = (warp & 3) * 32;
    const int64_t row0 = (int64_t)tile * kTM + lane_base;
    const int64_t row = row0 + lane;
    const bool is_reset = row < M && pos_is_zero(pos, pos64, row);
    uint8_t* blk_a = smem + warp * 8192;                     // conv values in, a out
    uint8_t* blk_x = blk_a + 4096;                           // normalised input out
    const int cr = lane >> 3, cp = lane & 7;                 // copy pattern: row cr + 4 k, piece cp
    // (a warp takes the 32-channel chunks warp / 4 and, with eight warps, every second behind it)
#pragma unroll 1
    for (int cq = warp >> 2; cq < kChans / 32; cq += kEpi / 4) {
      const int e0 = chan0 + cq * 32;
      // the conv values of the warp's block are asked for while the last MMAs run
      float4 cin[8];
#pragma unroll
      for (int k = 0; k < 8; ++k) {
        const int r = cr + 4 * k;
        cin[k] = make_float4(0.f, 0.f, 0.f, 0.f);
        if (row0 + r < M) cin[k] = *reinterpret_cast<const float4*>(x + (row0 + r) * E + e0 + cp * 4);
      }
      if (ok) ok = mbar_wait(bar_acc, 0, s_abort);             // every MMA has read the ring by now
      __syncwarp();
      tc_fence_after();
#pragma unroll
      for (int k = 0; k < 8; ++k) {
        const int r = cr + 4 * k;
        *reinterpret_cast<float4*>(blk_a + r * 128 + ((cp ^ (r & 7)) << 4)) = cin[k];
      }
      __syncwarp();
      const uint32_t t_row = tmem_base + (static_cast<uint32_t>(lane_base) << 16) + cq * 32;
#pragma unroll
      for (int cc = 0; cc < 2; ++cc) {
        uint32_t zx[16], za[16];
        tc_ld_32x16(t_row + cc * 16, zx);
        tc_ld_32x16(t_row + kChans + cc * 16, za);
        tc_wait_ld();
#pragma unroll
        for (int q = 0; q < 4; ++q) {
          const int piece = (cc * 4 + q) ^ (lane & 7);
          const float4 cv = *reinterpret_cast<const float4*>(blk_a + lane * 128 + (piece << 4));
          const float cvv[4] = {cv.x, cv.y, cv.z, cv.w};
          float av[4], xv[4];
#pragma unroll
          for (int j = 0; j < 4; ++j) {
            const int n = q * 4 + j;
            const int ch = cq * 32 + cc * 16 + n;            // channel within the tile
            gate_math<false, true>(cvv[j], __uint_as_float(zx[n]), __uint_as_float(za[n]), s_sp[kChans + ch],
                             s_sp[2 * kChans + ch], s_sp[ch], is_reset, av[j], xv[j]);
          }
          *reinterpret_cast<float4*>(blk_a + lane * 128 + (piece << 4)) = make_float4(av[0], av[1], av[2], av[3]);
          *reinterpret_cast<float4*>(blk_x + lane * 128 + (piece << 4)) = make_float4(xv[0], xv[1], xv[2], xv[3]);
        }
      }
      __syncwarp();
      if (ok) {
#pragma unroll
        for (int k = 0; k < 8; ++k) {
          const int r = cr + 4 * k;
          if (row0 + r < M) {
            const int off = r * 128 + ((cp ^ (r & 7)) << 4);
            *reinterpret_cast<float4*>(a_out + (row0 + r) * E + e0 + cp * 4) =
                *reinterpret_cast<const float4*>(blk_a + off);
            *reinterpret_cast<float4*>(xn_out + (row0 + r) * E + e0 + cp * 4) =
                *reinterpret_cast<const float4*>(blk_x + off);
          }
        }
      }
      __syncwarp();
    }
  }

  // ------------------------------ teardown --------------------------------------------------------
  if (order == kSecond) grid_dependency_wait();            // whoever waits for this launch waits for the first too
  tc_fence_before();
  __syncthreads();
  if (threadIdx.x == 0 && *s_abort) atomicExch(&hdr->status, kStatusTimeout);
  if (warp == kEpi + 1) {
    tc_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" :: "r"(tmem_base), "r"(kTN)
                 : "memory");
  }
}

template <int kTN, int kPerSm>
cudaError_t set_smem() {
  return cudaFuncSetAttribute(gates_tf32_kernel<kTN, kPerSm>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                              Cfg<kTN, kPerSm>::kSmem);
}

template <int kTN, int kPerSm>
cudaError_t launch_gates_t(const float* c, const void* pos, int pos64, const float* a_param, const float* bx,
                           const float* ba, int64_t M, int E, const float* hi, const float* lo, float* a_out,
                           float* xn_out, WsHeader* hdr, cudaStream_t s, const ScanPrep& prep, int64_t first_tile,
                           int64_t n_tiles, int order) {
  const uint64_t w_rows = (uint64_t)E / kHalf * (2 * kHalf);
  CUtensorMap map_x, map_wh, map_wl;
  if (!tensor_map_2d(&map_x, c, (uint64_t)M, (uint64_t)E, kTM, kKS, false, 4, true) ||
      !tensor_map_2d(&map_wh, hi, w_rows, kHW, kTN / 2, kKS, false, 4, true) ||
      !tensor_map_2d(&map_wl, lo, w_rows, kHW, kTN / 2, kKS, false, 4, true))
    return cudaErrorInvalidValue;
  return launch_dependent(gates_tf32_kernel<kTN, kPerSm>, dim3((unsigned)n_tiles), dim3(Cfg<kTN, kPerSm>::kThreads),
                          (size_t)Cfg<kTN, kPerSm>::kSmem, s, map_x, map_wh, map_wl, c, pos, pos64, a_param, bx, ba,
                          M, E, a_out, xn_out, hdr, prep, (int)first_tile, order);
}

// Splits the two gate weights [H, 256 (k), 256 (n)] float32 into K-major groups
// [H, 2, 256 (n'), 256 (k)] (rows 0-127 of a group: the x-gate columns of its 128 channels, rows
// 128-255 the a-gate ones), once with the low 13 mantissa bits cleared and once as what they held.
__global__ void pack_gate_weights_tf32_kernel(const float* __restrict__ wx, const float* __restrict__ wa,
                                              int H, float* __restrict__ hi, float* __restrict__ lo) {
  __shared__ float tile[32][33];
  const int group = blockIdx.z, head = group >> 1, half = group & 1;
  const int k0 = blockIdx.x * 32, n0 = blockIdx.y * 32;          // n' in [0, 256)
  const float* src = (n0 < kHalf ? wx : wa) + (int64_t)head * kHW * kHW;
  const int chan = half * kHalf + (n0 % kHalf);
  for (int r = threadIdx.y; r < 32; r += 8)                        // r walks k, x walks n
    tile[r][threadIdx.x] = src[(int64_t)(k0 + r) * kHW + chan + threadIdx.x];
  __syncthreads();
  const int64_t base = (int64_t)group * 2 * kHalf * kHW;
  for (int r = threadIdx.y; r < 32; r += 8) {                      // r walks n', x walks k
    const float v = tile[threadIdx.x][r];
    const float h = __uint_as_float(__float_as_uint(v) & 0xffffe000u);
    hi[base + (int64_t)(n0 + r) * kHW + k0 + threadIdx.x] = h;
    lo[base + (int64_t)(n0 + r) * kHW + k0 + threadIdx.x] = v - h;
  }
}

}  // namespace

size_t gates_tf32_packed_bytes(int H) { return (size_t)H * 2 * 2 * kHalf * kHW * 4 * 2; }

bool gates_tf32_supported(int dtype, int bw, int64_t M) {
  return dtype == 0 && bw == kHW && M >= 1 && M < ((int64_t)1 << 31);
}

cudaError_t launch_pack_gate_weights_tf32(const void* wx, const void* wa, int H, void* packed_w,
                                          cudaStream_t s) {
  float* hi = static_cast<float*>(packed_w);
  float* lo = hi + (size_t)H * 2 * 2 * kHalf * kHW;
  pack_gate_weights_tf32_kernel<<<dim3(kHW / 32, 2 * kHalf / 32, 2 * H), dim3(32, 8), 0, s>>>(
      (const float*)wx, (const float*)wa, H, hi, lo);
  return cudaGetLastError();
}

cudaError_t launch_gates_tf32(const void* c, const void* pos, int pos64, const void* a_param,
                              const void* wx, const void* bx, const void* wa, const void* ba,
                              int64_t M, int H, void* packed_w, bool packed_valid, void* a_out,
                              void* xn_out, void* ws_header, cudaStream_t s, const ScanPrep& prep) {
  if (M == 0) return cudaSuccess;
  const int E = H * kHW;
  float* hi = static_cast<float*>(packed_w);
  float* lo = hi + (size_t)H * 2 * 2 * kHalf * kHW;
  if (!packed_valid) {
    cudaError_t err = launch_pack_gate_weights_tf32(wx, wa, H, packed_w, s);
    if (err != cudaSuccess) return err;
  }

  static PerDeviceOnce once;
  int num_sms = 0;
  cudaError_t e0 = once.run([] {
    cudaError_t e = set_smem<256, 1>();
    if (e == cudaSuccess) e = set_smem<256, 2>();
    if (e == cudaSuccess) e = set_smem<128, 2>();
    return e;
  }, &num_sms);
  if (e0 != cudaSuccess) return e0;
  // One tile an SM as long as there are no more: 700 tokens of 2560 channels 34 us, as two CTAs an SM 39.
  // From there on two an SM, so that one's arithmetic runs under the other's contraction: 32768 tokens
  // 829 -> 737 us with the scan behind.  Few tiles are cut in half: 200 tokens 29 -> 25 us.
  const int64_t m_tiles = (M + kTM - 1) / kTM, tiles = m_tiles * (E / kHalf);
  if (2 * tiles > 0x7fffffff) return cudaErrorInvalidValue;
  auto run = [&](auto launch, int64_t first, int64_t n, int order) {
    return launch((const float*)c, pos, pos64, (const float*)a_param, (const float*)bx, (const float*)ba, M, E, hi,
                  lo, (float*)a_out, (float*)xn_out, reinterpret_cast<WsHeader*>(ws_header), s,
                  order == kSecond ? ScanPrep() : prep, first, n, order);
  };
  if (2 * tiles <= num_sms) return run(launch_gates_t<128, 2>, 0, 2 * tiles, kAlone);
  if (tiles <= num_sms) return run(launch_gates_t<256, 1>, 0, tiles, kAlone);
  // A last wave that half tiles, one an SM, can carry becomes a second launch of those, whose CTAs start as
  // the first's leave: 2048 tokens (24 of 320 tiles) 71 -> 66 us with the scan, 4096 (48 of 640) 131 -> 124;
  // with 96 of 1280 tiles left over 234.5 -> 236, with 204 of 500 94 -> 98.
  const int64_t slots = 2 * (int64_t)num_sms, rest = tiles > slots ? tiles % slots : 0;
  if (rest == 0 || 2 * rest > num_sms) return run(launch_gates_t<256, 2>, 0, tiles, kAlone);
  e0 = run(launch_gates_t<256, 2>, 0, tiles - rest, kFirst);
  return e0 != cudaSuccess ? e0 : run(launch_gates_t<128, 2>, 2 * (tiles - rest), 2 * rest, kSecond);
}

}  // namespace rgk
