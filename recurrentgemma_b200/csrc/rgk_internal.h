// Launchers implemented by the .cu files of librgk; called only from api.cu, which validates
// arguments first.  Each returns the cudaError_t of its last launch.
#pragma once

#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <stddef.h>
#include <stdint.h>

#include <mutex>

namespace rgk {

// One-time set-up per device.  cudaFuncSetAttribute applies to the function on the CURRENT device
// only, so a launcher that needs more than the default dynamic shared memory runs its set-up the
// first time it sees each device (a process may drive several), under a lock, and caches that
// device's SM count.  A failed set-up is retried by the next call.
class PerDeviceOnce {
 public:
  template <typename F>
  cudaError_t run(F&& setup, int* num_sms = nullptr) {
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return e;
    if (dev < 0 || dev >= kMaxDevices) return cudaErrorInvalidDevice;
    std::lock_guard<std::mutex> lock(mu_);
    if (sms_[dev] == 0) {
      int n = 0;
      if ((e = cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev)) != cudaSuccess) return e;
      if ((e = setup()) != cudaSuccess) return e;
      sms_[dev] = n;
    }
    if (num_sms != nullptr) *num_sms = sms_[dev];
    return cudaSuccess;
  }

 private:
  static constexpr int kMaxDevices = 64;
  std::mutex mu_;
  int sms_[kMaxDevices] = {};
};

// A launch that may be placed while the kernel in front still runs (programmatic dependent launch): every
// CTA of `kernel` executes griddepcontrol.wait before it touches memory that a kernel may have written
// or still reads.  Such a kernel promises of nothing but weights that it does not change while it runs: no
// __restrict__ on other pointers that it reads, no __ldg, no ld.global.nc.
template <typename... P, typename... A>
cudaError_t launch_dependent(void (*kernel)(P...), dim3 grid, dim3 block, size_t smem, cudaStream_t s, A... args) {
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = block;
  cfg.dynamicSmemBytes = smem;
  cfg.stream = s;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  const cudaError_t e = cudaLaunchKernelEx(&cfg, kernel, static_cast<P>(args)...);
  return e != cudaSuccess ? e : cudaGetLastError();
}

// What rglru_chan_kernel finds prepared: the words that states (and maps) arrive in without their tokens,
// and -8 softplus(a_param).  The kernel in front does it on the side (launch_conv1d_prefill), or a small
// one of its own.
struct ChanPrep {
  uint4* zero = nullptr;
  int64_t n_zero = 0;                    // in packs of 16 bytes
  const __nv_bfloat16* a_param = nullptr;
  __nv_bfloat16* m8sp = nullptr;
  int E = 0;
  int early = 0;                         // the kernel behind is let in at once: it has a unit a CTA at most
};

// What scan_kernel finds cleared: its ticket and its flags.  The gate kernel in front does it on the side
// (launch_gates_tf32), or a memset.
struct ScanPrep {
  unsigned* ticket = nullptr;
  uint4* zero = nullptr;
  int64_t n_zero = 0;                    // in packs of 16 bytes
};

// The share of an SM's 228 KB that a launch asks to be shared memory rather than L1, for kernels that
// stream through L1: without it they inherit whatever the kernel in front left, and behind one that used
// all of it the projections of one row took 26 us instead of 11.5 (28 KB of L1 for 120 KB of loads in
// flight).  `bytes`: shared memory of the CTAs of an SM; 64 KB at least, so that the kernels of a decode
// step of a few sequences agree and the SMs are not reconfigured between them.
inline cudaLaunchAttribute smem_carveout(size_t bytes) {
  cudaLaunchAttribute a = {};
  a.id = cudaLaunchAttributePreferredSharedMemoryCarveout;
  const size_t kb = bytes > 64 * 1024 ? (bytes + 1023) / 1024 : 64;
  a.val.sharedMemCarveout = kb >= 228 ? 100 : (unsigned)((kb * 100 + 227) / 228);
  return a;
}

// How the fused RG-LRU kernel evaluates the two sigmoids of the gates and the gelu of the join.
//   kMathExact  sigmoids as 1 / (1 + 2^(-z log2 e)) in float32 with one reciprocal for the four
//               denominators of a token pair (both gates), gelu as z / (1 + 2^w) with one reciprocal
//               per token pair; every rounding of the reference, so that the outputs agree with
//               the reference's bfloat16 arithmetic on all but a fraction of a percent of the elements.
//   kMathFast   the input gate as 0.5 + 0.5 tanh(z / 2) and the gelu as 0.5 z (1 + tanh u) in
//               packed bfloat16 (tanh.approx.bf16x2): 5.5 instead of 6 special-function operations
//               and about 15 fewer instructions per element; a third to a half of the outputs then
//               differ from the reference's by one bfloat16 step.  The recurrence gate keeps the
//               exact form: where a = exp(log_a) sits near 1 a one-step change of that gate flips
//               the rounding of a, and the state of such a slow channel drifts from the reference's.
enum { kMathExact = 0, kMathFast = 1 };

// conv1d.cu
cudaError_t launch_conv1d_prefill(const void* x, const void* pos, int pos64, const void* w,
                                  const void* b, int64_t B, int64_t T, int64_t E, int dtype,
                                  void* out, void* cache_out, cudaStream_t s,
                                  const ChanPrep& prep = ChanPrep());
// the cache a prefill returns, alone (the fused RG-LRU kernel computes the convolution itself)
cudaError_t launch_conv1d_cache(const void* x, const void* pos, int pos64, int64_t B, int64_t T,
                                int64_t E, int dtype, void* cache_out, cudaStream_t s);
cudaError_t launch_conv1d_decode(const void* x, const void* cache_in, const void* w, const void* b,
                                 int64_t B, int64_t E, int dtype, void* out, void* cache_out,
                                 cudaStream_t s);

// blockdiag_simt.cu
cudaError_t launch_blockdiag_linear_simt(const void* x, const void* w, const void* b, int64_t M,
                                         int H, int bw, int dtype, void* out, cudaStream_t s);
// Gate projections + gate arithmetic: writes a (reset-masked) and the normalised input.
cudaError_t launch_gates_simt(const void* c, const void* pos, int pos64, const void* a_param,
                              const void* wx, const void* bx, const void* wa, const void* ba,
                              int64_t M, int H, int bw, int dtype, void* a_out, void* xn_out,
                              cudaStream_t s);

// gates_tc.cu: the same as launch_gates_simt on tcgen05 tensor cores (bfloat16, head width 256).
// packed_w: gates_tc_packed_bytes(H) bytes of scratch for the K-major copy of the weights.
bool gates_tc_supported(int dtype, int bw, int64_t M);
size_t gates_tc_packed_bytes(int H);
cudaError_t launch_gates_tc(const void* c, const void* pos, int pos64, const void* a_param,
                            const void* wx, const void* bx, const void* wa, const void* ba,
                            int64_t M, int H, void* packed_w, int packed_ready, void* a_out,
                            void* xn_out, void* ws_header, cudaStream_t s);

// gates_tf32.cu: the same for float32 and head width 256, as three TF32 products per float32
// product (hi/lo split of both operands, float32 accumulation in tensor memory).  packed_w:
// gates_tf32_packed_bytes(H) bytes of scratch for the split K-major copies of the weights.
bool gates_tf32_supported(int dtype, int bw, int64_t M);
size_t gates_tf32_packed_bytes(int H);
cudaError_t launch_pack_gate_weights_tf32(const void* wx, const void* wa, int H, void* packed_w,
                                          cudaStream_t s);
cudaError_t launch_gates_tf32(const void* c, const void* pos, int pos64, const void* a_param,
                              const void* wx, const void* bx, const void* wa, const void* ba,
                              int64_t M, int H, void* packed_w, bool packed_valid, void* a_out, void* xn_out,
                              void* ws_header, cudaStream_t s, const ScanPrep& prep = ScanPrep());

// Packs the gate weights only (the first step of launch_gates_tc), for callers that keep the
// packed copy across calls; launch_gates_tc with packed_ready != 0 then skips its own packing.
cudaError_t launch_pack_gate_weights(const void* wx, const void* wa, int H, void* packed_w,
                                     cudaStream_t s);

// decode_tc.cu: one decode step of the whole sub-path (conv step, gates on tcgen05, state update,
// join) in a single kernel; bfloat16, head width 256.  packed_w as produced by
// launch_pack_gate_weights.  cache_out must not alias cache_in.
cudaError_t launch_path_decode_tc(const void* xb, const void* yb, const void* pos, int pos64,
                                  const void* conv_w, const void* conv_b, const void* a_param,
                                  const void* bx, const void* ba, const void* packed_w,
                                  const float* h_in, const void* cache_in, int64_t B, int H,
                                  void* out, float* h_out, void* cache_out, void* ws_header,
                                  cudaStream_t s, int math);

// rglru_chan_tc.cu: gate projections + gate arithmetic + scan (+ join) in one kernel with
// channel-major accumulators (TMEM lane = channel), so that gate arithmetic, recurrence and join
// run in registers in time order; bfloat16, head width 256, any T.  math: one of the kMath*
// variants of tc_common.cuh (how the sigmoids and the gelu are evaluated).
// ws: rglru_chan_workspace_bytes(B, T, E) bytes whose first word is the caller's status word.
bool rglru_chan_supported(int dtype, int bw, int64_t B, int64_t T);
size_t rglru_chan_workspace_bytes(int64_t B, int64_t T, int64_t E);
// what the launch below does first unless `prepared`
ChanPrep rglru_chan_prep(void* ws, const void* a_param, int64_t B, int64_t T, int H);
cudaError_t launch_rglru_chan(const void* c, const void* pos, int pos64, const void* a_param,
                              const void* bx, const void* ba, const void* packed_w, const float* h0,
                              const void* yb, int y_activated, int64_t B, int64_t T, int H,
                              void* out, float* h_last, void* ws, int math, cudaStream_t s,
                              const void* conv_w = nullptr, const void* conv_b = nullptr,
                              bool prepared = false);

// rglru_f32_tc.cu: the same in float32 (gates on three float16 products per float32 product).  Supported where
// the tiles of 128 tokens a sequence is cut into are not mostly empty.  out must not overlap c; the join is the gelu one.
// zx, za: float32 [B, T, E] of scratch for the gates' arguments of tokens that are not left to the halves.
// ws: rglru_f32_workspace_bytes(B, T, E) bytes whose first word is the caller's status word.
bool rglru_f32_supported(int dtype, int bw, int64_t B, int64_t T, int H);
size_t rglru_f32_workspace_bytes(int64_t B, int64_t T, int64_t E);
size_t rglru_f32_packed_bytes(int H);
cudaError_t launch_pack_gate_weights_f16(const void* wx, const void* wa, int H, void* packed_w, cudaStream_t s);
// what the launch below does first unless `prepared`
ChanPrep rglru_f32_prep(void* ws, int64_t B, int64_t T, int H);
cudaError_t launch_rglru_f32(const void* c, const void* pos, int pos64, const void* a_param, const void* wx,
                             const void* bx, const void* wa, const void* ba, const void* packed_w, const float* h0,
                             const void* yb, int64_t B, int64_t T, int H, float* zx, float* za, void* out,
                             float* h_last, void* ws, cudaStream_t s, bool prepared);

// gemm_rows.cu: up to three projections (matrices) of the same M <= 8 rows in one launch, with
// RMSNorm of the rows in front (norm_scale, or NULL) and act 0 / 1 / 2 or cap as below behind (act 1 on the
// first matrix only); one
// residual for a single matrix.  early: no kernel in front of this one on the stream that could still be
// running writes weights (it is one of the library's own, launched by the same call), so they may
// be fetched before it ends.
struct RowsMatrix {
  const void* w;
  const void* bias;
  void* out;
  int n;
};
// whether that kernel is the one for M <= 8 rows without a norm
bool rows_gemm_suits(int64_t M, int64_t K);
bool rows_gemm_supported(int dtype, int64_t M, int64_t K, int64_t N, bool norm);
cudaError_t launch_rows_gemm(const void* x, const void* norm_scale, float eps, const RowsMatrix* mats,
                             int n_mats, const void* residual, int64_t M, int K, int act, float cap,
                             bool early, cudaStream_t s);
// gemm_small_tc.cu: the same projections (no norm) for up to some hundreds of rows, weights split over
// all SMs (the K slices of a feature tile are a thread-block cluster and add up in distributed
// shared memory).  act 0: bias; 1: gelu_tanh of the first matrix's rounded result; 2: GeGLU over the packed
// up-projection of the MLP (w as pack_mlp_up_kernel writes it, n = 2 X rows, out [M, X]).  status:
// optional device int raised on a bounded-wait timeout.  early as for launch_rows_gemm; wide: CTAs
// that never share an SM with another of the same launch (kernels in a chain alternate).
bool dense_small_supported(int dtype, int64_t M, int64_t K, int64_t N);
cudaError_t launch_dense_small(const void* x, const RowsMatrix* mats, int n_mats, const void* residual,
                               int64_t M, int K, int act, float cap, int* status, bool early, bool wide,
                               cudaStream_t s);
// decode_rows.cu: launch_path_decode_tc for small batches; early as for launch_rows_gemm.
cudaError_t launch_path_decode_rows(const void* xb, const void* yb, const void* pos, int pos64,
                                    const void* conv_w, const void* conv_b, const void* a_param,
                                    const void* bx, const void* ba, const void* packed_w,
                                    const float* h_in, const void* cache_in, int64_t B, int H,
                                    void* out, float* h_out, void* cache_out, cudaStream_t s,
                                    int math, bool early);

// gemm_tc.cu: out [M,N] = x [M,K] W[N,K]^T + bias (bfloat16, float32 accumulation) on tcgen05;
// act == 1 applies gelu_tanh to the rounded result; act == 2 is the GeGLU epilogue of the MLP
// block (W and bias packed by launch_pack_mlp_up, N = 2 X, out [M, X]); residual != null adds a
// [M,N] tensor to the rounded result and rounds again (not together with gelu).  cap != 0 (no bias,
// gelu or residual) is the logits soft cap: tanh(acc / cap) * cap with every rounding of the
// reference.  status: optional device int raised on a bounded-wait timeout.
// Any number of rows, up to three matrices of the same K in one launch; act 1 applies to the first
// matrix, act 2, cap and a residual take a single one.
bool dense_tc_supported(int dtype, int64_t M, int64_t K, int64_t N);
cudaError_t launch_dense_tc(const void* x, const RowsMatrix* mats, int n_mats, const void* residual, int64_t M,
                            int K, int act, int* status, cudaStream_t s, float cap = 0.0f);

// attention_decode.cu: one new token per sequence against the ring cache keys / values [B,W,256]
// (num_tokens [B] int32 tokens seen so far): q [B,N,256], k_new [B,256], v_new [B,256]
// -> out [B,N*256]; update != 0 then stores k_new / v_new in ring slot num_tokens % W and adds one
// to num_tokens.
// float32, q and k_new rotated: the ring is updated in place.  ws: attention_decode_workspace_bytes.
bool attention_decode_supported(int hd, int N, int W);
size_t attention_decode_workspace_bytes(int64_t B, int N, int W);
cudaError_t launch_attention_decode(const void* q, const void* k_new, const void* v_new, void* keys,
                                    void* values, int* num_tokens, int64_t B, int N, int W,
                                    int update, void* out, void* ws, cudaStream_t s);
// bfloat16; q and k_new are rotated by the positions pos [B], unless it is NULL.  The updated ring goes to
// keys, values, seen, which may be the tensors it is read from; status: raised if a bounded wait gives up.
cudaError_t launch_attention_decode_ring(const void* q, const void* k_new, const void* v_new, const void* pos,
                                         int pos64, const void* keys_in, const void* values_in,
                                         const int* seen_in, void* keys, void* values, int* seen, int64_t B,
                                         int N, int W, int update, void* out, int* status, cudaStream_t s);

// embed.cu: rows of the embedding table scaled by a constant (Embedder.encode), and the index of
// the first maximum of every row of a [M, V] matrix (greedy sampling).
cudaError_t launch_embed(const void* tokens, int tokens64, const void* table, int64_t M, int64_t V,
                         int64_t D, float scale, int dtype, void* out, cudaStream_t s);
cudaError_t launch_argmax(const void* x, int64_t M, int64_t V, int dtype, int* out, cudaStream_t s);
// up [2,M,X], bias [2,X] -> out [M,X] = gelu_tanh(up[0] + bias[0]) * (up[1] + bias[1]), four roundings.
cudaError_t launch_geglu_bias(const void* up, const void* bias, int64_t M, int64_t X, int dtype,
                              void* out, cudaStream_t s);

// ffw_up.w [2, D, X], ffw_up.b [2, X] -> packed_w [2X, D], packed_b [2X] (gemm_tc.cu, mode 3).
cudaError_t launch_pack_mlp_up(const void* w, const void* b, int D, int X, void* packed_w,
                               void* packed_b, cudaStream_t s);

// attention.cu: rotary embedding in place (x [rows, heads, hd], the first half of each head), and
// the local multi-query attention of the attention blocks in prefill form: q [B,T,N,256] and
// k [B,T,256] (rotated in place first if `rotate`), v [B,T,256], bfloat16 -> out [B,T,N*256], which may
// be q.  cache_k, cache_v [B,window,256] and num_tokens [B]: the ring cache a prompt leaves behind, or
// NULL.  ws: attention_workspace_bytes.
cudaError_t launch_rope(void* x, const void* pos, int pos64, int64_t rows, int heads, int hd,
                        int dtype, cudaStream_t s);
bool attention_supported(int dtype, int hd, int64_t B, int64_t T, int N);
size_t attention_workspace_bytes(int64_t B, int64_t T);
cudaError_t launch_attention_prefill(void* q, void* k, const void* v, const void* pos, int pos64, int64_t B,
                                     int64_t T, int N, int window, bool rotate, void* cache_k,
                                     void* cache_v, int* num_tokens, void* out, void* ws, cudaStream_t s);

// rmsnorm.cu: out [M,D] = x * rsqrt(mean(x^2) + eps) * (scale + 1) with the reference's roundings
// (torch/layers.py:65-73); one warp per row held in registers.
bool rmsnorm_supported(int dtype, int64_t D);
cudaError_t launch_rmsnorm(const void* x, const void* scale, int64_t M, int64_t D, float eps,
                           int dtype, void* out, cudaStream_t s, const void* addend = nullptr,
                           void* sum_out = nullptr);
// The same for few bfloat16 rows: a block per row, launched as a programmatic dependent; early as for
// launch_rows_gemm.
cudaError_t launch_rmsnorm_rows(const void* x, const void* scale, int64_t M, int64_t D, float eps, bool early,
                                void* out, cudaStream_t s);

// scan.cu
size_t scan_workspace_bytes(int64_t B, int64_t T, int64_t E, int dtype);
// y_mul (optional): the join y * gelu_tanh(y_mul), or y * y_mul when y_activated != 0 (the factor
// was already passed through gelu by whoever produced it).  skip_time_tiles / spin_limit: only for
// the wait-expiry self-test (rgk_selftest_wait_expiry); 0 = the whole problem, the default limit.
// what the launch below clears first unless `prepared`
ScanPrep scan_prep(void* ws, int64_t B, int64_t T, int64_t E, int dtype);
cudaError_t launch_scan(const void* x, const void* a, const uint8_t* reset, const void* pos,
                        int pos64, const float* h0, const void* y_mul, int y_activated, int64_t B,
                        int64_t T, int64_t E, int dtype, void* y, float* h_last, void* ws,
                        cudaStream_t s, int skip_time_tiles = 0, unsigned spin_limit = 0,
                        bool prepared = false);

// The scan's built-in scratch (a __device__ array inside scan.cu): its size, and its address on the
// current device (looked up with cudaGetSymbolAddress on first use per device).
size_t scan_static_scratch_bytes();
cudaError_t scan_static_scratch(void** ptr_out);

// decode.cu
// One recurrence step from precomputed a / normalised x: h_out = a h_in + xn (float32, unrounded),
// out = round(h_out) [* gelu_tanh(yb)].
cudaError_t launch_decode_update(const void* a, const void* xn, const float* h_in, const void* yb,
                                 int64_t B, int64_t E, int dtype, void* out, float* h_out,
                                 cudaStream_t s);

}  // namespace rgk
