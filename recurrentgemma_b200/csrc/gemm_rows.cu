// Dense projections of a handful of rows (M <= 8: a decode step of a few sequences), with what
// surrounds them in the blocks: RMSNorm of the rows in front (torch/layers.py:65-73), bias, gelu,
// GeGLU, residual add or the logits soft cap behind (recurrentgemma torch/modules.py:531-548,
// 626-647, 749-752, 897-911, 1001-1003; torch/griffin.py:183-185).
//
// Bound: the weights are streamed from HBM once (26 MB for linear_y | linear_x at 2B dims, 4.1 us
// at 6.45 TB/s) and nothing else matters much, so the kernel is built around keeping loads in
// flight and around starting early.  A unit of work is 8 output features over the whole K: its
// 8 x K weights are the B operand of mma.sync.m16n8k16 and go from global memory straight into
// registers - lane (g, t) of a warp holds 16-byte pieces of feature g - with K divided over the 8
// warps of a CTA; at K = 2560 that is ten 16-byte loads per lane, all issued before the first use and
// before the dependency wait of a programmatic dependent launch (the weights depend on no kernel
// that signals early).  The rows of x are the A operand, its upper 8 rows empty.  Against the 128-feature tcgen05
// tiles of gemm_small_tc.cu there is no tensor-memory or barrier set-up, no K split over CTAs and
// no exchange of partial sums, and 8-feature units fill every SM evenly.  The contraction index is permuted the same way in both operands, so that a lane
// feeds two instructions from one 16-byte piece (elements 0-3, then 4-7).
//
// CTAs are persistent over units (three per SM), refilling each weight register as soon as its
// value has been used.  x (normalised, if asked) is staged once per CTA in shared memory; where M x K
// is too large for that, fragments of x are read from L2 as they are needed.
//
// From 9 rows on the upper half of the A operand would have to be there too (its registers cost the weights
// in flight) and x be read again for every 8 features, where the tcgen05 kernel reads it once per 128:
// 2560 x 2560 at 9 rows 7.0 us this way, 6.5 that.
#include "rgk_common.cuh"
#include "rgk_internal.h"
#include "tc_common.cuh"

namespace rgk {
namespace {

constexpr int kRowsWarps = 8;
constexpr int kRowsThreads = kRowsWarps * 32;
constexpr int kU = 10;                    // 16-byte weight pieces in flight per lane
constexpr int kCtasPerSm = 3;
constexpr int kXBudget = 84 * 1024;       // staged x per CTA: 8 rows of 5120
constexpr int kXThree = 71 * 1024;        // up to here there is room for three CTAs per SM, above that for two
// Without a norm to apply, larger rows are better read from L2 as they are needed (four rows of 7680: 12.6 us
// staged, while eight rows read from L2 take 10.4 us).
constexpr int kXStage = 48 * 1024;

struct RowsArgs {
  const __nv_bfloat16 *x, *scale, *residual;
  RowsMatrix mat[3];                      // up to three projections of the same rows
  int unit1, unit2;                       // the first units of the second and third
  int M, K;
  int units, chunks, blocks_per_warp;     // 8-feature units; chunks of kU K blocks per warp
  int pitch;                              // bytes between rows of the staged x
  float eps, cap;
  int early;                              // the kernel in front does not write weights
};

__device__ __forceinline__ float to_float(__nv_bfloat16 v) { return __bfloat162float(v); }

// kMode: 0 bias, 1 gelu of the first matrix as well, residual if given; 2 GeGLU over the packed up-projection; 4 soft cap.
// kStaged: x lies in shared memory (normalised if `scale` is given).
// kFull: K is exactly 8 warps x chunks x kU blocks of 32 (2560, 7680), so no piece needs a test.
enum { kPlain = 0, kGeluRows = 1, kGeglu = 2, kCap = 4 };

template <int kMode, bool kStaged, bool kFull>
__global__ void __launch_bounds__(kRowsThreads, kCtasPerSm)
gemm_rows_kernel(const RowsArgs a) {
  extern __shared__ __align__(16) uint8_t s_x[];
  __shared__ float s_red[kRowsWarps][8][8];
  __shared__ float s_sum[kRowsWarps];
  __shared__ uint32_t s_r[8];
  // (the warp's number from a lane, so that the compiler knows it to be the same in the whole warp: 0.8 % of a block's
  // decode step of one row, about 1 % of a generated token of one sequence)
  const int tid = threadIdx.x, warp = __shfl_sync(0xffffffffu, tid >> 5, 0), lane = tid & 31;
  const int g = lane >> 2, t = lane & 3;
  const int M = a.M, K = a.K;
  const int kb0 = warp * a.blocks_per_warp;

  // this lane's feature row of a unit, and the 16-byte piece of K block kb in it
  auto weight_row = [&](int unit) -> const __nv_bfloat16* {
    // (GeGLU: a unit is one group of the packed up-projection, 4 gate rows and their 4 value rows)
    const int i = (unit >= a.unit1) + (unit >= a.unit2);
    const int first = i == 0 ? 0 : (i == 1 ? a.unit1 : a.unit2);
    return static_cast<const __nv_bfloat16*>(a.mat[i].w) + (int64_t)((unit - first) * 8 + g) * K;
  };
  auto piece = [&](const __nv_bfloat16* row, int kb) -> uint4 {
    const int k = kb * 32 + t * 8;
    return (kFull || (kb < kb0 + a.blocks_per_warp && k < K)) ? ld_stream(row + k) : make_uint4(0u, 0u, 0u, 0u);
  };

  // ---- weights of the first chunk, before anything that depends on the kernel in front -----------
  uint4 w[kU];
  int unit = blockIdx.x;                  // grid <= units
  const __nv_bfloat16* row = weight_row(unit);
  auto first_chunk = [&] {
#pragma unroll
    for (int i = 0; i < kU; ++i) w[i] = piece(row, kb0 + i);
  };
  if (a.early) {
    first_chunk();
    grid_launch_dependents();
    grid_dependency_wait();
  } else {
    // The kernel in front may have written the weights: until it has completed they are only asked
    // into L2 (the point of coherence), and the next kernel is not let loose on them either.
    if (t == 0) {
#pragma unroll
      for (int i = 0; i < kU; i += 2) {
        if (kFull || (kb0 + i) * 32 < K)
          asm volatile("prefetch.global.L2 [%0];" :: "l"(row + (kb0 + i) * 32));
      }
    }
    grid_dependency_wait();
    grid_launch_dependents();
    first_chunk();
  }

  // ---- x into shared memory, normalised on the way ------------------------------------------------
  if constexpr (kStaged) {
    const int packs = K / 8;
    if (a.scale != nullptr) {
      // the sum over the bfloat16-rounded squares of a row, every rounding of the reference; all 8
      // warps at work whatever M is
      constexpr int kS = 2;               // scale packs kept in registers while the sums are formed
      uint4 sc[kS];
#pragma unroll
      for (int j = 0; j < kS; ++j)
        sc[j] = tid + j * kRowsThreads < packs
                    ? *reinterpret_cast<const uint4*>(a.scale + (tid + j * kRowsThreads) * 8)
                    : make_uint4(0u, 0u, 0u, 0u);
      const int wpr = M == 1 ? 8 : (M == 2 ? 4 : (M <= 4 ? 2 : 1));     // warps per row
      const int m = warp / wpr;
      float sum = 0.0f;
      if (m < M) {
#pragma unroll 5
        for (int p = (warp % wpr) * 32 + lane; p < packs; p += 32 * wpr) {
          const uint4 v = *reinterpret_cast<const uint4*>(a.x + (int64_t)m * K + p * 8);
          *reinterpret_cast<uint4*>(s_x + m * a.pitch + p * 16) = v;
          const uint32_t q[4] = {bmul2(v.x, v.x), bmul2(v.y, v.y), bmul2(v.z, v.z), bmul2(v.w, v.w)};
#pragma unroll
          for (int k = 0; k < 4; ++k) sum += bf16_lo(q[k]) + bf16_hi(q[k]);
        }
      }
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
      if (lane == 0) s_sum[warp] = sum;
      __syncthreads();
      if (tid < M) {
        float total = 0.0f;
        for (int i = 0; i < wpr; ++i) total += s_sum[tid * wpr + i];
        const float var = round_bf16(total / (float)K);
        const float r = round_bf16(1.0f / sqrtf(round_bf16(var + a.eps)));
        s_r[tid] = pack_bf16x2(r, r);
      }
      __syncthreads();
      constexpr uint32_t kOne = 0x3f803f80u;
      auto scale_pack = [&](int p, uint4 v) {
        const uint4 s1 = make_uint4(badd2(v.x, kOne), badd2(v.y, kOne), badd2(v.z, kOne), badd2(v.w, kOne));
        for (int m = 0; m < M; ++m) {
          uint4* at = reinterpret_cast<uint4*>(s_x + m * a.pitch + p * 16);
          const uint32_t r2 = s_r[m];
          const uint4 u = *at;
          *at = make_uint4(bmul2(bmul2(u.x, r2), s1.x), bmul2(bmul2(u.y, r2), s1.y),
                           bmul2(bmul2(u.z, r2), s1.z), bmul2(bmul2(u.w, r2), s1.w));
        }
      };
#pragma unroll
      for (int j = 0; j < kS; ++j)
        if (tid + j * kRowsThreads < packs) scale_pack(tid + j * kRowsThreads, sc[j]);
      for (int p = tid + kS * kRowsThreads; p < packs; p += kRowsThreads)
        scale_pack(p, *reinterpret_cast<const uint4*>(a.scale + p * 8));
    } else {
#pragma unroll 4
      for (int i = tid; i < M * packs; i += kRowsThreads) {
        const int m = i / packs, p = i - m * packs;
        *reinterpret_cast<uint4*>(s_x + m * a.pitch + p * 16) =
            *reinterpret_cast<const uint4*>(a.x + (int64_t)m * K + p * 8);
      }
    }
    __syncthreads();
  }
  // a fragment of x: 16 bytes of row m of K block kb
  auto x_piece = [&](int m, int kb) -> uint4 {
    const int k = kb * 32 + t * 8;
    if (m >= M || (!kFull && k >= K)) return make_uint4(0u, 0u, 0u, 0u);
    if constexpr (kStaged) return *reinterpret_cast<const uint4*>(s_x + m * a.pitch + k * 2);
    else return *reinterpret_cast<const uint4*>(a.x + (int64_t)m * K + k);
  };

  for (; unit < a.units; unit += gridDim.x) {
    float acc[2][4] = {};                 // two chains of accumulation
    // The bias and the residual of the epilogue are asked for here (and kept as loaded: a conversion
    // would wait for them) where the contraction reads nothing else from global memory; behind
    // fragment loads of x they would only lengthen the queue.
    const int em = tid >> 3, ef = tid & 7;
    const bool e_ok = em < M && (kMode != kGeglu || ef < 4);
    const int mi = (unit >= a.unit1) + (unit >= a.unit2);
    const int col = kMode == kGeglu ? unit * 4 + ef
                                    : (unit - (mi == 0 ? 0 : (mi == 1 ? a.unit1 : a.unit2))) * 8 + ef;
    __nv_bfloat16 e_bias = __ushort_as_bfloat16(0), e_other = e_bias;   // other: value's bias, or residual
    auto epilogue_operands = [&] {
      if (kMode == kCap || !e_ok) return;
      const __nv_bfloat16* bias = static_cast<const __nv_bfloat16*>(a.mat[mi].bias);
      const int bc = kMode == kGeglu ? unit * 8 + ef : col;
      if (bias != nullptr) e_bias = bias[bc];
      if constexpr (kMode == kGeglu) e_other = bias[bc + 4];
      else if (a.residual != nullptr) e_other = a.residual[(int64_t)em * a.mat[0].n + col];
    };
    if constexpr (kStaged) epilogue_operands();
    for (int c = 0; c < a.chunks; ++c) {
      const int kb = kb0 + c * kU;
      // what refills the registers: the next chunk of this unit, or the first of the next unit
      const bool last = c + 1 == a.chunks;
      const int next_unit = last ? unit + (int)gridDim.x : unit;
      const int next_kb = last ? kb0 : kb + kU;
      const bool more = next_unit < a.units;
      if (last && more) row = weight_row(next_unit);
      constexpr int kX = kStaged ? 1 : 5;      // pieces of x in flight (registers)
#pragma unroll
      for (int h = 0; h < kU; h += kX) {
        uint4 xa[kX];
#pragma unroll
        for (int i = 0; i < kX; ++i) xa[i] = x_piece(g, kb + h + i);
#pragma unroll
        for (int i = 0; i < kX; ++i) {
          const uint4 b = w[h + i];
          mma_16816(acc[0], xa[i].x, 0u, xa[i].y, 0u, b.x, b.y);
          mma_16816(acc[1], xa[i].z, 0u, xa[i].w, 0u, b.z, b.w);
          if (more) w[h + i] = piece(row, next_kb + h + i);
        }
      }
    }
    // ---- the warps' sums, then the epilogue ----------------------------------------------------------
    *reinterpret_cast<float2*>(&s_red[warp][g][2 * t]) =
        make_float2(acc[0][0] + acc[1][0], acc[0][1] + acc[1][1]);
    __syncthreads();
    {
      if constexpr (!kStaged) epilogue_operands();
      if (e_ok) {
        float sum = 0.0f;
#pragma unroll
        for (int i = 0; i < kRowsWarps; ++i) sum += s_red[i][em][ef];
        __nv_bfloat16* out = static_cast<__nv_bfloat16*>(a.mat[mi].out);
        if constexpr (kMode == kGeglu) {
          float val = 0.0f;
#pragma unroll
          for (int i = 0; i < kRowsWarps; ++i) val += s_red[i][em][ef + 4];
          // the contraction and the bias add are two tensor operations
          const float gate = round_bf16(round_bf16(sum) + to_float(e_bias));
          const float value = round_bf16(round_bf16(val) + to_float(e_other));
          out[(int64_t)em * (a.mat[0].n / 2) + col] =
              __float2bfloat16_rn(round_bf16(gelu_tanh_<true>(gate)) * value);
        } else if constexpr (kMode == kCap) {
          const float q = round_bf16(__fdiv_rn(round_bf16(sum), a.cap));
          out[(int64_t)em * a.mat[0].n + col] = __float2bfloat16_rn(round_bf16(tanhf(q)) * a.cap);
        } else {
          float y = round_bf16(sum + to_float(e_bias));
          if (kMode == kGeluRows && mi == 0) y = round_bf16(gelu_tanh_<true>(y));
          if (a.residual != nullptr) y = y + to_float(e_other);
          out[(int64_t)em * a.mat[mi].n + col] = __float2bfloat16_rn(y);
        }
      }
    }
    __syncthreads();
  }
}

template <int kMode>
cudaError_t launch_rows_t(const cudaLaunchConfig_t& cfg, bool staged, const RowsArgs& a) {
  if (a.K == kRowsWarps * a.chunks * kU * 32)
    return staged ? cudaLaunchKernelEx(&cfg, gemm_rows_kernel<kMode, true, true>, a)
                  : cudaLaunchKernelEx(&cfg, gemm_rows_kernel<kMode, false, true>, a);
  return staged ? cudaLaunchKernelEx(&cfg, gemm_rows_kernel<kMode, true, false>, a)
                : cudaLaunchKernelEx(&cfg, gemm_rows_kernel<kMode, false, false>, a);
}

template <int kMode>
cudaError_t set_smem() {
  cudaError_t e = cudaSuccess;
  auto set = [&](auto* kernel) {
    if (e == cudaSuccess)
      e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kXBudget);
  };
  set(gemm_rows_kernel<kMode, true, true>);
  set(gemm_rows_kernel<kMode, true, false>);
  return e;
}

int x_pitch(int K) { return (K * 2 + 127) / 128 * 128 + 64; }   // an odd half of 128: conflict-free pieces

}  // namespace

// Rows read from L2 as they are needed cost the general form too much: its pieces have tests of their own and
// its last chunk is partly empty (4096 -> 4096 18 us at 6 to 8 rows, 12288 -> 4096 39 us at two, where
// gemm_small_tc.cu takes 9.5 and 20).
bool rows_gemm_suits(int64_t M, int64_t K) {
  return K % (kRowsWarps * kU * 32) == 0 || M * x_pitch((int)K) <= kXStage;
}

bool rows_gemm_supported(int dtype, int64_t M, int64_t K, int64_t N, bool norm) {
  return dtype == 1 && M >= 1 && M <= 8 && K >= 8 && N >= 8 && K % 8 == 0 && N % 8 == 0 &&
         K < (1 << 28) && N < (1 << 30) && (!norm || M * x_pitch((int)K) <= kXBudget);
}

cudaError_t launch_rows_gemm(const void* x, const void* norm_scale, float eps, const RowsMatrix* mats,
                             int n_mats, const void* residual, int64_t M, int K, int act, float cap,
                             bool early, cudaStream_t s) {
  static PerDeviceOnce once;
  int num_sms = 0;
  cudaError_t e0 = once.run([] {
    cudaError_t e = set_smem<kPlain>();
    if (e == cudaSuccess) e = set_smem<kGeluRows>();
    if (e == cudaSuccess) e = set_smem<kGeglu>();
    if (e == cudaSuccess) e = set_smem<kCap>();
    return e;
  }, &num_sms);
  if (e0 != cudaSuccess) return e0;
  if (n_mats < 1 || n_mats > 3 || M < 1 || M > 8) return cudaErrorInvalidValue;
  RowsArgs a;
  a.x = (const __nv_bfloat16*)x;
  a.scale = (const __nv_bfloat16*)norm_scale;
  a.residual = (const __nv_bfloat16*)residual;
  a.units = 0;
  for (int i = 0; i < 3; ++i) {
    a.mat[i] = mats[i < n_mats ? i : 0];
    if (i == 1) a.unit1 = a.units;
    if (i == 2) a.unit2 = a.units;
    if (i < n_mats) {
      if (mats[i].n % 8 != 0) return cudaErrorInvalidValue;
      a.units += mats[i].n / 8;
    }
  }
  if (act == 2 && (n_mats != 1 || residual != nullptr || mats[0].bias == nullptr || mats[0].n % 128 != 0))
    return cudaErrorInvalidValue;
  if (n_mats > 1 && residual != nullptr) return cudaErrorInvalidValue;
  if (cap != 0.0f && (n_mats != 1 || residual != nullptr || mats[0].bias != nullptr || act != 0))
    return cudaErrorInvalidValue;
  a.M = (int)M; a.K = K;
  a.early = early ? 1 : 0;
  const int blocks = (K + 31) / 32;
  a.blocks_per_warp = (blocks + kRowsWarps - 1) / kRowsWarps;
  a.chunks = (a.blocks_per_warp + kU - 1) / kU;
  a.pitch = x_pitch(K);
  a.eps = eps; a.cap = cap;
  const bool staged = (int64_t)M * a.pitch <= (norm_scale != nullptr ? kXBudget : kXStage);
  if (norm_scale != nullptr && !staged) return cudaErrorInvalidValue;

  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cudaLaunchConfig_t cfg = {};
  const int per_sm = staged && (int64_t)M * a.pitch > kXThree ? 2 : kCtasPerSm;
  const int slots = num_sms * per_sm;
  attr[1] = smem_carveout(per_sm * ((staged ? (size_t)M * a.pitch : 0) + 6 * 1024));
  cfg.gridDim = dim3((unsigned)(a.units < slots ? a.units : slots));
  cfg.blockDim = dim3(kRowsThreads);
  cfg.dynamicSmemBytes = staged ? (size_t)M * a.pitch : 0;
  cfg.stream = s;
  cfg.attrs = attr;
  cfg.numAttrs = 2;
#define RGK_ROWS(MODE) launch_rows_t<MODE>(cfg, staged, a)
  cudaError_t e;
  if (cap != 0.0f) e = RGK_ROWS(kCap);
  else if (act == 2) e = RGK_ROWS(kGeglu);
  else if (act == 1) e = RGK_ROWS(kGeluRows);
  else e = RGK_ROWS(kPlain);
#undef RGK_ROWS
  return e != cudaSuccess ? e : cudaGetLastError();
}

}  // namespace rgk
