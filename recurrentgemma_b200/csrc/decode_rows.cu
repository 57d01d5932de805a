// One decode step of the RG-LRU + Conv1D sub-path for small batches as a single kernel (bfloat16,
// heads of width 256): recurrentgemma torch/layers.py:469-550 (Conv1D with a cache), 338-353
// (gates), 170-177 (rnn_scan with one token) and the join of torch/modules.py:627-628, 646.
//
// Bound: latency.  The step of a 2B layer reads 2.6 MB of gate weights and a few kilobytes per
// row; what counts is the chain loads -> conv -> contraction -> gate arithmetic -> stores.  The
// 128-row tile of decode_tc.cu pays for tensor-memory set-up, a weight tile through shared
// memory and an exchange of conv slices between CTAs whatever the batch is; here a CTA serves 16
// rows x 32 channels: a thread convolves 8 channels of one row (the whole head's 256 channels, so
// that nothing is exchanged: eight times the loads, which at 16 rows is 2.6 MB of L2 traffic), the
// gate weights go from global memory straight into the B fragments of mma.sync.m16n8k16 before the
// activations are there, and 16 warps = 4 groups of 8 channels x 4 quarters of K keep that to four
// 16-byte loads and eight instructions per warp.
//
// The eight CTAs of a head are a cluster: when the conv window is updated in place, each waits for
// the other seven to have read it.
#include "rgk_common.cuh"
#include "rgk_internal.h"
#include "tc_common.cuh"

namespace rgk {
namespace {

constexpr int kHeadR = 256;
constexpr int kRowsR = 16;                       // batch rows per CTA
constexpr int kThreadsR = 512;
constexpr int kPitchR = kHeadR * 2 + 64;         // conv rows in shared memory: conflict-free pieces
__device__ __forceinline__ uint4 mul4r(const uint4& a, const uint4& b) {
  return make_uint4(bmul2(a.x, b.x), bmul2(a.y, b.y), bmul2(a.z, b.z), bmul2(a.w, b.w));
}
__device__ __forceinline__ uint4 add4r(const uint4& a, const uint4& b) {
  return make_uint4(badd2(a.x, b.x), badd2(a.y, b.y), badd2(a.z, b.z), badd2(a.w, b.w));
}

struct DecodeRowsArgs {
  const __nv_bfloat16 *xb, *yb, *conv_w, *conv_b, *a_param, *bias_x, *bias_a, *cache_in, *packed;
  const void* pos;
  const float* h_in;
  __nv_bfloat16 *out, *cache_out;
  float* h_out;
  int pos64, M, E;
  int ordered;            // the CTAs of a head must all have read before any of them writes
  int early;              // the kernel in front does not write weights: fetch them before it ends
};

// kCG: groups of 8 channels per warp, a CTA owns 32 x kCG channels.
template <bool kMul, int kMath, int kCG>
__global__ void __launch_bounds__(kThreadsR, 2)
decode_rows_kernel(const DecodeRowsArgs a) {
  constexpr int kChansR = 32 * kCG;              // channels per CTA
  constexpr int kCtasR = kHeadR / kChansR;       // per head: the cluster
  constexpr int kZPitch = kChansR + 4;
  __shared__ __align__(16) uint8_t s_conv[kRowsR * kPitchR];
  __shared__ float s_z[4][2][kRowsR][kZPitch];   // [quarter of K][gate][row][channel]
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, g = lane >> 2, t = lane & 3;
  const int head = blockIdx.x / kCtasR, part = blockIdx.x % kCtasR;
  const int row0 = blockIdx.y * kRowsR;
  const int E = a.E;
  const int chan0 = head * kHeadR + part * kChansR;

  // ---- gate weights: K-major rows of the packed copy ([head][half][128 x-gate | 128 a-gate][256]) --
  const int grp = warp & 3, kq = warp >> 2;      // 8 kCG channels; 64 of the 256 contraction indices
  const __nv_bfloat16* wrow[kCG];
#pragma unroll
  for (int c = 0; c < kCG; ++c) {
    const int ch = part * kChansR + (c * 4 + grp) * 8 + g;       // channel within the head
    wrow[c] = a.packed + ((int64_t)(head * 2 + (ch >> 7)) * 256 + (ch & 127)) * kHeadR + kq * 64 + t * 8;
  }
  uint4 wx[kCG][2], wa[kCG][2];
  auto load_weights = [&] {
#pragma unroll
    for (int c = 0; c < kCG; ++c) {
#pragma unroll
      for (int i = 0; i < 2; ++i) {
        wx[c][i] = ld_stream(wrow[c] + i * 32);
        wa[c][i] = ld_stream(wrow[c] + 128 * kHeadR + i * 32);
      }
    }
  };
  // What comes from HBM and may have been written by the kernel in front is only asked into L2 before
  // the wait (L2 is the point of coherence).
  const int ec = head * kHeadR + lane * 8;       // conv: a warp is a row, a lane 8 channels
  const int m = row0 + warp;
  const bool row_ok = m < a.M;
  const __nv_bfloat16* cr = a.cache_in + (int64_t)(row_ok ? m : 0) * 3 * E + ec;
  if (a.early) {
    load_weights();
  } else if (t == 0) {
#pragma unroll
    for (int c = 0; c < kCG; ++c) {
      asm volatile("prefetch.global.L2 [%0];" :: "l"(wrow[c]));
      asm volatile("prefetch.global.L2 [%0];" :: "l"(wrow[c] + 128 * kHeadR));
    }
  }
  if (row_ok && (lane & 7) == 0) {
    asm volatile("prefetch.global.L2 [%0];" :: "l"(cr));
    asm volatile("prefetch.global.L2 [%0];" :: "l"(cr + E));
    asm volatile("prefetch.global.L2 [%0];" :: "l"(cr + 2 * (int64_t)E));
  }
  // epilogue threads: one row, two channels
  const int er = tid / (kChansR / 2), ep = tid % (kChansR / 2);
  const int e0 = chan0 + 2 * ep, me = row0 + er;
  const bool epi = tid < kRowsR * kChansR / 2 && me < a.M;
  if (epi && ep % 16 == 0) asm volatile("prefetch.global.L2 [%0];" :: "l"(a.h_in + (int64_t)me * E + e0));
  uint4 cw[4], cb;
  uint32_t bx2 = 0, ba2 = 0, m8 = 0;
  auto load_constants = [&] {
#pragma unroll
    for (int k = 0; k < 4; ++k) cw[k] = *reinterpret_cast<const uint4*>(a.conv_w + (int64_t)k * E + ec);
    cb = *reinterpret_cast<const uint4*>(a.conv_b + ec);
    if (epi) {
      bx2 = *reinterpret_cast<const uint32_t*>(a.bias_x + e0);
      ba2 = *reinterpret_cast<const uint32_t*>(a.bias_a + e0);
      const uint32_t ap = *reinterpret_cast<const uint32_t*>(a.a_param + e0);
      m8 = pack_bf16x2(-8.0f * round_bf16(softplus_(bf16_lo(ap))), -8.0f * round_bf16(softplus_(bf16_hi(ap))));
    }
  };
  if (a.early) {
    load_constants();
    grid_launch_dependents();
    grid_dependency_wait();
  } else {
    // the next kernel may fetch weights as soon as it starts: not before the kernel in front of
    // this one, which may have written them, has completed
    grid_dependency_wait();
    grid_launch_dependents();
    load_weights();
    load_constants();
  }

  // ---- conv: newest tap first (torch/layers.py:491-517 with prompt_len = 3), then the bias ---------
  uint4 x1, x2, x3, cv = make_uint4(0u, 0u, 0u, 0u);
  if (row_ok) {
    const uint4 x0 = *reinterpret_cast<const uint4*>(cr);
    x1 = *reinterpret_cast<const uint4*>(cr + E);
    x2 = *reinterpret_cast<const uint4*>(cr + 2 * (int64_t)E);
    x3 = *reinterpret_cast<const uint4*>(a.xb + (int64_t)m * E + ec);
    cv = mul4r(x3, cw[3]);
    cv = add4r(cv, mul4r(x2, cw[2]));
    cv = add4r(cv, mul4r(x1, cw[1]));
    cv = add4r(cv, mul4r(x0, cw[0]));
    cv = add4r(cv, cb);
  }
  // the state and the other branch, in flight during the contraction
  float2 h = make_float2(0.f, 0.f);
  uint32_t y2 = 0;
  bool is_reset = false;
  if (epi) {
    h = *reinterpret_cast<const float2*>(a.h_in + (int64_t)me * E + e0);
    if constexpr (kMul) y2 = *reinterpret_cast<const uint32_t*>(a.yb + (int64_t)me * E + e0);
    is_reset = pos_is_zero(a.pos, a.pos64, me);
  }
  *reinterpret_cast<uint4*>(s_conv + warp * kPitchR + lane * 16) = cv;
  __syncthreads();
  if (a.ordered) asm volatile("barrier.cluster.arrive.aligned;" ::: "memory");

  // ---- both gates: 16 rows x 8 kCG channels x 64 contraction indices per warp -----------------------
  uint4 lo[2], hi[2];
#pragma unroll
  for (int i = 0; i < 2; ++i) {
    const uint8_t* src = s_conv + g * kPitchR + (kq * 64 + i * 32 + t * 8) * 2;
    lo[i] = *reinterpret_cast<const uint4*>(src);
    hi[i] = *reinterpret_cast<const uint4*>(src + 8 * kPitchR);
  }
#pragma unroll
  for (int c = 0; c < kCG; ++c) {
    float zx[4] = {}, za[4] = {};
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      mma_16816(zx, lo[i].x, hi[i].x, lo[i].y, hi[i].y, wx[c][i].x, wx[c][i].y);
      mma_16816(za, lo[i].x, hi[i].x, lo[i].y, hi[i].y, wa[c][i].x, wa[c][i].y);
      mma_16816(zx, lo[i].z, hi[i].z, lo[i].w, hi[i].w, wx[c][i].z, wx[c][i].w);
      mma_16816(za, lo[i].z, hi[i].z, lo[i].w, hi[i].w, wa[c][i].z, wa[c][i].w);
    }
    const int zc = (c * 4 + grp) * 8 + 2 * t;
    *reinterpret_cast<float2*>(&s_z[kq][0][g][zc]) = make_float2(zx[0], zx[1]);
    *reinterpret_cast<float2*>(&s_z[kq][0][g + 8][zc]) = make_float2(zx[2], zx[3]);
    *reinterpret_cast<float2*>(&s_z[kq][1][g][zc]) = make_float2(za[0], za[1]);
    *reinterpret_cast<float2*>(&s_z[kq][1][g + 8][zc]) = make_float2(za[2], za[3]);
  }
  __syncthreads();
  if (a.ordered) asm volatile("barrier.cluster.wait.aligned;" ::: "memory");

  // ---- shifted conv window: this CTA's own channels ---------------------------------------------------
  if (a.cache_out != nullptr && row_ok && lane / (kChansR / 8) == part) {
    __nv_bfloat16* co = a.cache_out + (int64_t)m * 3 * E + ec;
    *reinterpret_cast<uint4*>(co) = x1;
    *reinterpret_cast<uint4*>(co + E) = x2;
    *reinterpret_cast<uint4*>(co + 2 * (int64_t)E) = x3;
  }
  // ---- gate arithmetic, state update, join --------------------------------------------------------------
  if (epi) {
    float2 sx = make_float2(0.f, 0.f), sa = sx;
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      const float2 px = *reinterpret_cast<const float2*>(&s_z[k][0][er][2 * ep]);
      const float2 pa = *reinterpret_cast<const float2*>(&s_z[k][1][er][2 * ep]);
      sx.x += px.x; sx.y += px.y; sa.x += pa.x; sa.y += pa.y;
    }
    const uint32_t c2 = *reinterpret_cast<const uint32_t*>(s_conv + er * kPitchR + (part * kChansR + 2 * ep) * 2);
    uint32_t a2, xn2;
    if constexpr (kMath == kMathFast) {
      uint32_t gx2, mult2;
      gate_tokens<kMathFast>(sx.x, sx.y, sa.x, sa.y, bx2, ba2, bmul2(bx2, 0x3f003f00u), m8, a2, gx2, mult2);
      if (is_reset) {
        mult2 = 0x3f803f80u;
        a2 = 0u;
      }
      xn2 = bmul2(bmul2(c2, gx2), mult2);
    } else {
      gate_pair(sx.x, sx.y, sa.x, sa.y, bx2, ba2, m8, c2, is_reset, a2, xn2);
    }
    // h = a h + x in float32; the state keeps the unrounded value (torch/layers.py:176-177)
    h = make_float2(fmaf(bf16_lo(a2), h.x, bf16_lo(xn2)), fmaf(bf16_hi(a2), h.y, bf16_hi(xn2)));
    uint32_t o = pack_bf16x2(h.x, h.y);
    if constexpr (kMul) {
      if constexpr (kMath == kMathFast) {
        o = join_gelu2<kMathFast>(o, y2);
      } else {
        o = bmul2(o, pack_bf16x2(gelu_tanh_<true>(bf16_lo(y2)), gelu_tanh_<true>(bf16_hi(y2))));
      }
    }
    *reinterpret_cast<float2*>(a.h_out + (int64_t)me * E + e0) = h;
    *reinterpret_cast<uint32_t*>(a.out + (int64_t)me * E + e0) = o;
  }
}

}  // namespace

cudaError_t launch_path_decode_rows(const void* xb, const void* yb, const void* pos, int pos64,
                                    const void* conv_w, const void* conv_b, const void* a_param,
                                    const void* bx, const void* ba, const void* packed_w,
                                    const float* h_in, const void* cache_in, int64_t B, int H,
                                    void* out, float* h_out, void* cache_out, cudaStream_t s,
                                    int math, bool early) {
  if (B == 0) return cudaSuccess;
  using T_ = const __nv_bfloat16*;
  DecodeRowsArgs a;
  a.xb = (T_)xb; a.yb = (T_)yb; a.conv_w = (T_)conv_w; a.conv_b = (T_)conv_b; a.a_param = (T_)a_param;
  a.bias_x = (T_)bx; a.bias_a = (T_)ba; a.cache_in = (T_)cache_in; a.packed = (T_)packed_w;
  a.pos = pos; a.h_in = h_in; a.out = (__nv_bfloat16*)out; a.cache_out = (__nv_bfloat16*)cache_out;
  a.h_out = h_out; a.pos64 = pos64; a.M = (int)B; a.E = H * kHeadR;
  a.ordered = cache_out == cache_in || out == xb;
  a.early = early;
  // 32 channels per CTA while all CTAs then run at once (two per SM, in clusters of eight), 64 from
  // there on: half the conv work in all, and twice the rest per CTA
  const int cg = B <= 48 ? 1 : 2, ctas = kHeadR / (32 * cg);
  cudaLaunchAttribute attr[3];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  attr[1].id = cudaLaunchAttributeClusterDimension;      // the channel groups of a head
  attr[1].val.clusterDim.x = (unsigned)ctas;
  attr[1].val.clusterDim.y = 1;
  attr[1].val.clusterDim.z = 1;
  attr[2] = smem_carveout(2 * 30 * 1024);                // two CTAs
  cudaLaunchConfig_t cfg = {};
  const unsigned row_tiles = (unsigned)((B + kRowsR - 1) / kRowsR);
  cfg.gridDim = dim3((unsigned)(H * ctas), row_tiles);
  cfg.blockDim = dim3(kThreadsR);
  cfg.stream = s;
  cfg.attrs = attr;
  cfg.numAttrs = 3;
  cudaError_t e;
#define RGK_DEC(MUL, MATH)                                                        \
  (cg == 1 ? cudaLaunchKernelEx(&cfg, decode_rows_kernel<MUL, MATH, 1>, a)        \
           : cudaLaunchKernelEx(&cfg, decode_rows_kernel<MUL, MATH, 2>, a))
  if (math == kMathExact) e = yb ? RGK_DEC(true, kMathExact) : RGK_DEC(false, kMathExact);
  else e = yb ? RGK_DEC(true, kMathFast) : RGK_DEC(false, kMathFast);
#undef RGK_DEC
  return e != cudaSuccess ? e : cudaGetLastError();
}

}  // namespace rgk
