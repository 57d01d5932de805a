// extern "C" surface of librgk (include/rgk.h): argument validation, error text, workspace carving
// and the composition of the kernels into the calls the reference's Python methods map to.
#include <cstdarg>
#include <cstdio>
#include <atomic>
#include <cstring>

#include "../../include/rgk.h"
#include "rgk_common.cuh"
#include "rgk_internal.h"

namespace {

thread_local char g_err[512] = "";

int fail(int code, const char* fmt, ...) {
  va_list ap;
  va_start(ap, fmt);
  vsnprintf(g_err, sizeof(g_err), fmt, ap);
  va_end(ap);
  return code;
}

int cuda_fail(cudaError_t e, const char* what) {
  return fail(RGK_ECUDA, "%s: %s", what, cudaGetErrorString(e));
}

bool aligned16(const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15u) == 0; }

size_t up256(size_t v) { return (v + 255) & ~static_cast<size_t>(255); }

int elem_size(int dtype) { return dtype == RGK_BF16 ? 2 : 4; }

// Compute capability of each device, looked up once (immutable afterwards).
int device_ok() {
  static int cached[64];  // 0 unknown, 1 ok, -1 wrong arch
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return cuda_fail(e, "cudaGetDevice");
  if (dev >= 0 && dev < 64 && cached[dev] == 1) return RGK_OK;
  int major = 0;
  e = cudaDeviceGetAttribute(&major, cudaDevAttrComputeCapabilityMajor, dev);
  if (e != cudaSuccess) return cuda_fail(e, "cudaDeviceGetAttribute");
  if (major != 10) {
    return fail(RGK_EARCH, "device %d has compute capability %d.x; librgk is built for sm_100a only",
                dev, major);
  }
  if (dev >= 0 && dev < 64) cached[dev] = 1;
  return RGK_OK;
}

#define RGK_REQUIRE(cond, code, ...) \
  do {                               \
    if (!(cond)) return fail(code, __VA_ARGS__); \
  } while (0)

#define RGK_CHECK_DEVICE()          \
  do {                              \
    int rc_ = device_ok();          \
    if (rc_ != RGK_OK) return rc_;  \
  } while (0)

#define RGK_CUDA(expr, what)                              \
  do {                                                    \
    cudaError_t e_ = (expr);                              \
    if (e_ != cudaSuccess) return cuda_fail(e_, what);    \
  } while (0)

int check_common(int64_t B, int64_t T, int64_t E, int dtype) {
  RGK_REQUIRE(dtype == RGK_F32 || dtype == RGK_BF16, RGK_EINVAL, "unknown dtype %d", dtype);
  RGK_REQUIRE(B >= 0 && T >= 0 && E >= 0, RGK_EINVAL, "negative size (B=%lld T=%lld E=%lld)",
              (long long)B, (long long)T, (long long)E);
  const int pack = dtype == RGK_BF16 ? 8 : 4;
  RGK_REQUIRE(E % pack == 0, RGK_ESHAPE, "width %lld is not a multiple of %d (16-byte channel packs)",
              (long long)E, pack);
  RGK_REQUIRE(B <= 65535, RGK_ESHAPE, "batch %lld exceeds 65535", (long long)B);
  RGK_REQUIRE(T <= (1 << 21), RGK_ESHAPE, "sequence length %lld exceeds 2^21", (long long)T);
  RGK_REQUIRE(E <= (1 << 20), RGK_ESHAPE, "width %lld exceeds 2^20", (long long)E);
  return RGK_OK;
}

int check_heads(int64_t E, int H) {
  RGK_REQUIRE(H >= 1 && E % H == 0, RGK_ESHAPE, "width %lld is not divisible by %d heads",
              (long long)E, H);
  RGK_REQUIRE((E / H) % 16 == 0, RGK_ESHAPE, "head width %lld is not a multiple of 16",
              (long long)(E / H));
  return RGK_OK;
}

int check_params(const rgk_params* p, bool need_conv) {
  RGK_REQUIRE(p != nullptr, RGK_EINVAL, "params is NULL");
  RGK_REQUIRE(p->a_param && p->gate_x_w && p->gate_x_b && p->gate_a_w && p->gate_a_b, RGK_EINVAL,
              "a gate parameter pointer is NULL");
  RGK_REQUIRE(!need_conv || (p->conv_w && p->conv_b), RGK_EINVAL, "conv parameter pointer is NULL");
  RGK_REQUIRE(aligned16(p->a_param) && aligned16(p->gate_x_w) && aligned16(p->gate_x_b) &&
                  aligned16(p->gate_a_w) && aligned16(p->gate_a_b) &&
                  (!need_conv || (aligned16(p->conv_w) && aligned16(p->conv_b))),
              RGK_EALIGN, "parameter pointers must be 16-byte aligned");
  return RGK_OK;
}

// Gate projections + gate arithmetic with the kernel `gates_impl` selects.
int run_gates(const void* c, const void* pos, int pos64, const rgk_params* p, int64_t M, int H,
              int bw, int dtype, int gates_impl, void* wpack, void* a, void* xn, void* ws_header,
              cudaStream_t s, const rgk::ScanPrep& prep = rgk::ScanPrep()) {
  const bool tc_ok = rgk::gates_tc_supported(dtype, bw, M);
  const bool tf32_ok = rgk::gates_tf32_supported(dtype, bw, M);
  if (gates_impl == RGK_GATES_TCGEN05 && !tc_ok && !tf32_ok)
    return fail(RGK_ESHAPE, "the tcgen05 gate kernels cover head width 256 only "
                            "(dtype %d, head width %d)", dtype, bw);
  if (tf32_ok && gates_impl != RGK_GATES_SIMT) {
    cudaError_t e = rgk::launch_gates_tf32(c, pos, pos64, p->a_param, p->gate_x_w, p->gate_x_b,
                                           p->gate_a_w, p->gate_a_b, M, H,
                                           p->gates_packed ? const_cast<void*>(p->gates_packed) : wpack,
                                           p->gates_packed != nullptr, a, xn, ws_header, s, prep);
    if (e != cudaSuccess) return cuda_fail(e, "tcgen05 TF32 gates launch");
    return RGK_OK;
  }
  if (tc_ok && gates_impl != RGK_GATES_SIMT) {
    cudaError_t e = rgk::launch_gates_tc(
        c, pos, pos64, p->a_param, p->gate_x_w, p->gate_x_b, p->gate_a_w, p->gate_a_b, M, H,
        p->gates_packed ? const_cast<void*>(p->gates_packed) : wpack, p->gates_packed != nullptr, a,
        xn, ws_header, s);
    if (e != cudaSuccess) return cuda_fail(e, "tcgen05 gates launch");
    return RGK_OK;
  }
  cudaError_t e = rgk::launch_gates_simt(c, pos, pos64, p->a_param, p->gate_x_w, p->gate_x_b,
                                         p->gate_a_w, p->gate_a_b, M, H, bw, dtype, a, xn, s);
  if (e != cudaSuccess) return cuda_fail(e, "gates launch");
  return RGK_OK;
}

// Whether the prefill path convolves inside the fused RG-LRU kernel (rgk_set_conv_fusion).  Off by
// default: on a B200 the two conv warps a CTA can afford cannot keep up with its sixteen epilogue
// warps (the same bits, at about half the speed of the separate conv kernel).
static std::atomic<int> g_conv_fusion{0};
static bool conv_fusion_enabled() { return g_conv_fusion.load(std::memory_order_relaxed) != 0; }

// RG-LRU on a conv output c: fused kernel when asked for / possible, else gates then scan.
// With xb != nullptr the Conv1D is this function's job as well: `c` is then only a buffer for the
// conv output, which the fused kernel does not need (it convolves xb itself, unless out aliases
// xb: the units read each other's input rows) and the other routes fill with conv1d_prefill.
int run_rglru(const void* c, const void* pos, int pos64, const rgk_params* p, const float* h0,
              const void* yb, int y_activated, int64_t B, int64_t T, int64_t E, int H, int dtype,
              int gates_impl, void* wpack, void* a_buf, void* xn_buf, void* scan_ws, void* out,
              float* h_last, cudaStream_t s, const void* xb = nullptr, void* conv_cache_out = nullptr) {
  const int bw = (int)(E / H);
  const bool chan_route = rgk::rglru_chan_supported(dtype, bw, B, T) &&
                          (gates_impl == RGK_GATES_AUTO || gates_impl >= RGK_GATES_FUSED);
  const bool fuse_conv = xb != nullptr && chan_route && out != xb && conv_fusion_enabled();
  // float32 in one kernel: a unit reads the head's other channels of its tokens while they are being written
  // elsewhere, so not where the output lies over the input
  const size_t act = static_cast<size_t>(B) * T * E * elem_size(dtype);
  const uintptr_t c0 = reinterpret_cast<uintptr_t>(c), out0 = reinterpret_cast<uintptr_t>(out);
  const bool f32_route = gates_impl == RGK_GATES_AUTO && rgk::rglru_f32_supported(dtype, bw, B, T, H) &&
                         !y_activated && (c0 + act <= out0 || out0 + act <= c0);
  if (xb != nullptr) {
    cudaError_t e = fuse_conv
        ? rgk::launch_conv1d_cache(xb, pos, pos64, B, T, E, dtype, conv_cache_out, s)
        : rgk::launch_conv1d_prefill(xb, pos, pos64, p->conv_w, p->conv_b, B, T, E, dtype,
                                     const_cast<void*>(c), conv_cache_out, s,
                                    chan_route ? rgk::rglru_chan_prep(scan_ws, p->a_param, B, T, H)
                                    : f32_route ? rgk::rglru_f32_prep(scan_ws, B, T, H) : rgk::ChanPrep());
    if (e != cudaSuccess) return cuda_fail(e, "conv1d launch");
  }
  if (f32_route) {
    const void* packed = wpack;
    if (p->gates_packed != nullptr) {                  // behind the TF32 copy
      packed = static_cast<const char*>(p->gates_packed) + rgk::gates_tf32_packed_bytes(H);
    } else {
      cudaError_t e = rgk::launch_pack_gate_weights_f16(p->gate_x_w, p->gate_a_w, H, wpack, s);
      if (e != cudaSuccess) return cuda_fail(e, "pack_gate_weights launch");
    }
    cudaError_t e = rgk::launch_rglru_f32(c, pos, pos64, p->a_param, p->gate_x_w, p->gate_x_b, p->gate_a_w,
                                          p->gate_a_b, packed, h0, yb, B, T, H, static_cast<float*>(a_buf),
                                          static_cast<float*>(xn_buf), out, h_last, scan_ws, s, xb != nullptr);
    if (e != cudaSuccess) return cuda_fail(e, "float32 RG-LRU launch");
    return RGK_OK;
  }
  const bool fused_ok = rgk::rglru_chan_supported(dtype, bw, B, T);
  const bool want_fused = gates_impl >= RGK_GATES_FUSED;
  if (want_fused && !fused_ok)
    return fail(RGK_ESHAPE, "the fused RG-LRU kernel covers bfloat16 and head width 256 "
                            "(dtype %d, head width %d, T %lld)", dtype, bw, (long long)T);
  if (fused_ok && (gates_impl == RGK_GATES_AUTO || want_fused)) {
    const int math = gates_impl == RGK_GATES_FUSED_EXACT ? rgk::kMathExact : rgk::kMathFast;
    const void* packed = p->gates_packed;
    if (packed == nullptr) {
      cudaError_t e = rgk::launch_pack_gate_weights(p->gate_x_w, p->gate_a_w, H, wpack, s);
      if (e != cudaSuccess) return cuda_fail(e, "pack_gate_weights launch");
      packed = wpack;
    }
    cudaError_t e = rgk::launch_rglru_chan(fuse_conv ? xb : c, pos, pos64, p->a_param, p->gate_x_b,
                                           p->gate_a_b, packed, h0, yb, y_activated, B, T, H, out,
                                           h_last, scan_ws, math, s, fuse_conv ? p->conv_w : nullptr,
                                           fuse_conv ? p->conv_b : nullptr, xb != nullptr && !fuse_conv);
    if (e != cudaSuccess) return cuda_fail(e, "fused RG-LRU launch");
    return RGK_OK;
  }
  // the float32 gate kernel clears what the scan wants cleared
  const int impl = want_fused ? RGK_GATES_AUTO : gates_impl;
  const bool prepared = rgk::gates_tf32_supported(dtype, bw, B * T) && impl != RGK_GATES_SIMT;
  int rc = run_gates(c, pos, pos64, p, B * T, H, bw, dtype, impl, wpack, a_buf, xn_buf, scan_ws, s,
                     prepared ? rgk::scan_prep(scan_ws, B, T, E, dtype) : rgk::ScanPrep());
  if (rc) return rc;
  cudaError_t e = rgk::launch_scan(xn_buf, a_buf, nullptr, nullptr, 0, h0, yb, y_activated, B, T, E,
                                   dtype, out, h_last, scan_ws, s, 0, 0, prepared);
  if (e != cudaSuccess) return cuda_fail(e, "scan launch");
  return RGK_OK;
}

// Carves the workspace of the composed calls: [scan scratch | c | a | xn | packed gate weights].
struct PathWs {
  void* scan;
  void* c;
  void* a;
  void* xn;
  void* wpack;
  size_t total;
};

PathWs carve(void* ws, int64_t B, int64_t T, int64_t E, int dtype) {
  PathWs w;
  size_t scan_bytes = rgk::scan_workspace_bytes(B, T, E, dtype);
  const size_t fused_bytes = dtype == RGK_BF16 ? rgk::rglru_chan_workspace_bytes(B, T, E)
                                               : rgk::rglru_f32_workspace_bytes(B, T, E);
  if (fused_bytes > scan_bytes) scan_bytes = fused_bytes;
  const size_t act = up256(static_cast<size_t>(B) * T * E * elem_size(dtype));
  char* base = static_cast<char*>(ws);
  w.scan = base;
  w.c = base ? base + scan_bytes : nullptr;
  w.a = base ? base + scan_bytes + act : nullptr;
  w.xn = base ? base + scan_bytes + 2 * act : nullptr;
  w.wpack = base ? base + scan_bytes + 3 * act : nullptr;
  // K-major copy of both gate weights for the tensor-core kernels: 2 * E * 256 bfloat16, or for
  // float32 the same split into a high and a low part (2 * 2 * E * 256 float32).
  w.total = scan_bytes + 3 * act + up256(static_cast<size_t>(E) * (dtype == RGK_BF16 ? 1024 : 4096));
  return w;
}

}  // namespace

extern "C" {

int rgk_abi_version(void) { return RGK_ABI_VERSION; }

const char* rgk_last_error(void) { return g_err; }

int rgk_device_check(void) { return device_ok(); }

size_t rgk_workspace_bytes(int64_t B, int64_t T, int64_t E, int dtype) {
  if (B < 0 || T < 0 || E < 0 || (dtype != RGK_F32 && dtype != RGK_BF16)) return 0;
  if (T < 1) T = 1;
  return carve(nullptr, B, T, E, dtype).total;
}

int rgk_workspace_status(void* workspace, void* stream) {
  RGK_REQUIRE(workspace != nullptr, RGK_EINVAL, "workspace is NULL");
  int status = 0;
  RGK_CUDA(cudaStreamSynchronize(static_cast<cudaStream_t>(stream)), "cudaStreamSynchronize");
  RGK_CUDA(cudaMemcpy(&status, workspace, sizeof(int), cudaMemcpyDeviceToHost), "cudaMemcpy");
  if (status == rgk::kStatusBounds) {
    RGK_CUDA(cudaMemset(workspace, 0, sizeof(int)), "cudaMemset");
    return fail(RGK_EBOUNDS, "a range-checked index fell outside its array (checks build); the "
                             "access was skipped and the results are invalid");
  }
  if (status == rgk::kStatusTimeout) {
    // reported once: the word is cleared so that later calls are judged on their own
    RGK_CUDA(cudaMemset(workspace, 0, sizeof(int)), "cudaMemset");
    return fail(RGK_ETIMEOUT, "a bounded device-side wait expired since the status word was last "
                              "cleared; results of the calls on this workspace since then are invalid");
  }
  return RGK_OK;
}

int rgk_set_conv_fusion(int enabled) {
  return g_conv_fusion.exchange(enabled != 0 ? 1 : 0, std::memory_order_relaxed);
}

int rgk_conv1d_prefill(const void* x, const void* segment_pos, int pos_dtype, const void* w,
                       const void* b, int64_t B, int64_t T, int64_t E, int W, int dtype, void* out,
                       void* cache_out, void* stream) {
  int rc = check_common(B, T, E, dtype);
  if (rc) return rc;
  RGK_REQUIRE(W == 4, RGK_ESHAPE, "temporal width %d is not supported (only 4)", W);
  RGK_REQUIRE(pos_dtype == RGK_I32 || pos_dtype == RGK_I64, RGK_EINVAL, "unknown index dtype");
  RGK_REQUIRE(x && segment_pos && w && b && out, RGK_EINVAL, "NULL pointer argument");
  RGK_REQUIRE(aligned16(x) && aligned16(w) && aligned16(b) && aligned16(out) && aligned16(cache_out),
              RGK_EALIGN, "pointers must be 16-byte aligned");
  RGK_CHECK_DEVICE();
  RGK_CUDA(rgk::launch_conv1d_prefill(x, segment_pos, pos_dtype, w, b, B, T, E, dtype, out,
                                      cache_out, static_cast<cudaStream_t>(stream)),
           "conv1d_prefill launch");
  if (T == 0 && cache_out && B * E > 0)
    RGK_CUDA(cudaMemsetAsync(cache_out, 0, (size_t)B * 3 * E * elem_size(dtype),
                             static_cast<cudaStream_t>(stream)), "cudaMemsetAsync");
  return RGK_OK;
}

int rgk_conv1d_decode(const void* x, const void* cache_in, const void* w, const void* b, int64_t B,
                      int64_t E, int W, int dtype, void* out, void* cache_out, void* stream) {
  int rc = check_common(B, 1, E, dtype);
  if (rc) return rc;
  RGK_REQUIRE(W == 4, RGK_ESHAPE, "temporal width %d is not supported (only 4)", W);
  RGK_REQUIRE(x && cache_in && w && b && out, RGK_EINVAL, "NULL pointer argument");
  RGK_REQUIRE(aligned16(x) && aligned16(cache_in) && aligned16(w) && aligned16(b) &&
                  aligned16(out) && aligned16(cache_out),
              RGK_EALIGN, "pointers must be 16-byte aligned");
  RGK_CHECK_DEVICE();
  RGK_CUDA(rgk::launch_conv1d_decode(x, cache_in, w, b, B, E, dtype, out, cache_out,
                                     static_cast<cudaStream_t>(stream)),
           "conv1d_decode launch");
  return RGK_OK;
}

int rgk_blockdiag_linear(const void* x, const void* w, const void* b, int64_t M, int H, int bw,
                         int dtype, void* out, void* stream) {
  RGK_REQUIRE(dtype == RGK_F32 || dtype == RGK_BF16, RGK_EINVAL, "unknown dtype %d", dtype);
  RGK_REQUIRE(M >= 0 && H >= 1 && bw >= 1, RGK_EINVAL, "bad size (M=%lld H=%d bw=%d)", (long long)M,
              H, bw);
  RGK_REQUIRE(bw % 16 == 0, RGK_ESHAPE, "head width %d is not a multiple of 16", bw);
  RGK_REQUIRE(M <= (int64_t)0x7fffffff * 64, RGK_ESHAPE, "too many rows");
  RGK_REQUIRE(x && w && b && out, RGK_EINVAL, "NULL pointer argument");
  RGK_CHECK_DEVICE();
  RGK_CUDA(rgk::launch_blockdiag_linear_simt(x, w, b, M, H, bw, dtype, out,
                                             static_cast<cudaStream_t>(stream)),
           "blockdiag_linear launch");
  return RGK_OK;
}

int rgk_linear_scan(const void* x, const void* a, const uint8_t* reset, const float* h0,
                    const void* y_mul, int64_t B, int64_t T, int64_t E, int dtype, void* y,
                    float* h_last, void* workspace, size_t workspace_bytes, void* stream) {
  int rc = check_common(B, T, E, dtype);
  if (rc) return rc;
  RGK_REQUIRE(x && a && y, RGK_EINVAL, "NULL pointer argument");
  RGK_REQUIRE(aligned16(x) && aligned16(a) && aligned16(y) && aligned16(y_mul) && aligned16(h0) &&
                  aligned16(h_last),
              RGK_EALIGN, "pointers must be 16-byte aligned");
  if (B * T * E == 0) return RGK_OK;
  const size_t need = rgk::scan_workspace_bytes(B, T, E, dtype);
  RGK_REQUIRE(workspace != nullptr && workspace_bytes >= need, RGK_EWORKSPACE,
              "workspace of %zu bytes needed, %zu given", need, workspace_bytes);
  RGK_REQUIRE((reinterpret_cast<uintptr_t>(workspace) & 255u) == 0, RGK_EALIGN,
              "workspace must be 256-byte aligned");
  RGK_CHECK_DEVICE();
  RGK_CUDA(rgk::launch_scan(x, a, reset, nullptr, 0, h0, y_mul, 0, B, T, E, dtype, y, h_last,
                            workspace, static_cast<cudaStream_t>(stream)),
           "scan launch");
  return RGK_OK;
}

size_t rgk_gate_pack_bytes(int H) { return H > 0 ? rgk::gates_tc_packed_bytes(H) : 0; }

size_t rgk_gate_pack_bytes_for(int H, int dtype) {
  if (H <= 0) return 0;
  if (dtype == RGK_BF16) return rgk::gates_tc_packed_bytes(H);
  if (dtype == RGK_F32) return rgk::gates_tf32_packed_bytes(H) + rgk::rglru_f32_packed_bytes(H);
  return 0;
}

int rgk_pack_gate_weights(const rgk_params* p, int H, int bw, int dtype, void* packed_out,
                          void* stream) {
  int rc = check_params(p, false);
  if (rc) return rc;
  RGK_REQUIRE(H >= 1 && packed_out != nullptr && aligned16(packed_out), RGK_EINVAL,
              "bad H or packed_out");
  RGK_REQUIRE(rgk::gates_tc_supported(dtype, bw, 1) || rgk::gates_tf32_supported(dtype, bw, 1),
              RGK_ESHAPE, "packed gate weights exist for head width 256 only");
  RGK_CHECK_DEVICE();
  if (dtype == RGK_F32) {
    RGK_CUDA(rgk::launch_pack_gate_weights_tf32(p->gate_x_w, p->gate_a_w, H, packed_out,
                                                static_cast<cudaStream_t>(stream)),
             "pack_gate_weights (TF32 split) launch");
    RGK_CUDA(rgk::launch_pack_gate_weights_f16(p->gate_x_w, p->gate_a_w, H,
                                               static_cast<char*>(packed_out) + rgk::gates_tf32_packed_bytes(H),
                                               static_cast<cudaStream_t>(stream)),
             "pack_gate_weights (float16 split) launch");
    return RGK_OK;
  }
  RGK_CUDA(rgk::launch_pack_gate_weights(p->gate_x_w, p->gate_a_w, H, packed_out,
                                         static_cast<cudaStream_t>(stream)),
           "pack_gate_weights launch");
  return RGK_OK;
}

int rgk_linear_scan_static(const void* x, const void* a, const uint8_t* reset, const float* h0,
                           const void* y_mul, int64_t B, int64_t T, int64_t E, int dtype, void* y,
                           float* h_last, int* status_out, void* stream) {
  int rc = check_common(B, T, E, dtype);
  if (rc) return rc;
  RGK_REQUIRE(x && a && y, RGK_EINVAL, "NULL pointer argument");
  RGK_REQUIRE(aligned16(x) && aligned16(a) && aligned16(y) && aligned16(y_mul) && aligned16(h0) &&
                  aligned16(h_last),
              RGK_EALIGN, "pointers must be 16-byte aligned");
  if (B * T * E == 0) return RGK_OK;
  const size_t need = rgk::scan_workspace_bytes(B, T, E, dtype);
  const size_t have = rgk::scan_static_scratch_bytes();
  RGK_REQUIRE(need <= have, RGK_ESHAPE,
              "problem needs %zu bytes of scan scratch but the built-in scratch holds %zu; use "
              "rgk_linear_scan with a caller workspace for sizes this large", need, have);
  RGK_CHECK_DEVICE();
  void* scratch = nullptr;
  RGK_CUDA(rgk::scan_static_scratch(&scratch), "cudaGetSymbolAddress(built-in scan scratch)");
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  // The array keeps whatever the previous call left: the status word is cleared here, the ticket
  // and the look-back flags by the launch below; records are rewritten before they are read.
  RGK_CUDA(cudaMemsetAsync(scratch, 0, sizeof(int), s), "cudaMemsetAsync");
  RGK_CUDA(rgk::launch_scan(x, a, reset, nullptr, 0, h0, y_mul, 0, B, T, E, dtype, y, h_last, scratch,
                            s),
           "scan launch");
  if (status_out != nullptr)
    RGK_CUDA(cudaMemcpyAsync(status_out, scratch, sizeof(int), cudaMemcpyDeviceToDevice, s),
             "cudaMemcpyAsync");
  return RGK_OK;
}

int rgk_selftest_wait_expiry(void* workspace, size_t workspace_bytes, void* stream) {
  // A scan over 2 sequences x 3 time tiles x 64 channels whose first time tile is never launched:
  // the tiles of the second time tile look back for records nobody publishes, give up after 200
  // polls (tens of microseconds), raise the status word, take a zero carry and finish.
  const int64_t B = 2, T = 3 * 128, E = 64;
  const size_t act = static_cast<size_t>(B * T * E) * 2;
  const size_t need = up256(rgk::scan_workspace_bytes(B, T, E, RGK_BF16)) + 3 * up256(act);
  RGK_REQUIRE(workspace != nullptr && workspace_bytes >= need, RGK_EWORKSPACE,
              "workspace of %zu bytes needed, %zu given", need, workspace_bytes);
  RGK_REQUIRE((reinterpret_cast<uintptr_t>(workspace) & 255u) == 0, RGK_EALIGN,
              "workspace must be 256-byte aligned");
  RGK_CHECK_DEVICE();
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  char* base = static_cast<char*>(workspace);
  char* x = base + up256(rgk::scan_workspace_bytes(B, T, E, RGK_BF16));
  char* a = x + up256(act);
  char* y = a + up256(act);
  RGK_CUDA(cudaMemsetAsync(x, 0, 3 * up256(act), s), "cudaMemsetAsync");
  RGK_CUDA(rgk::launch_scan(x, a, nullptr, nullptr, 0, nullptr, nullptr, 0, B, T, E, RGK_BF16, y,
                            nullptr, workspace, s, /*skip_time_tiles=*/1, /*spin_limit=*/200),
           "scan launch");
  return RGK_OK;
}

int rgk_rglru_forward(const void* x, const void* segment_pos, int pos_dtype, const rgk_params* p,
                      const float* h0, int64_t B, int64_t T, int64_t E, int H, int dtype,
                      int gates_impl, void* y, float* h_last, void* workspace,
                      size_t workspace_bytes, void* stream) {
  int rc = check_common(B, T, E, dtype);
  if (rc) return rc;
  if ((rc = check_heads(E, H))) return rc;
  if ((rc = check_params(p, false))) return rc;
  RGK_REQUIRE(pos_dtype == RGK_I32 || pos_dtype == RGK_I64, RGK_EINVAL, "unknown index dtype");
  RGK_REQUIRE(gates_impl >= RGK_GATES_AUTO && gates_impl <= RGK_GATES_FUSED_EXACT, RGK_EINVAL,
              "unknown gates_impl %d", gates_impl);
  RGK_REQUIRE(x && segment_pos && y, RGK_EINVAL, "NULL pointer argument");
  RGK_REQUIRE(aligned16(x) && aligned16(y) && aligned16(h0) && aligned16(h_last), RGK_EALIGN,
              "pointers must be 16-byte aligned");
  if (B * T * E == 0) return RGK_OK;
  const PathWs w = carve(workspace, B, T, E, dtype);
  RGK_REQUIRE(workspace != nullptr && workspace_bytes >= w.total, RGK_EWORKSPACE,
              "workspace of %zu bytes needed, %zu given", w.total, workspace_bytes);
  RGK_REQUIRE((reinterpret_cast<uintptr_t>(workspace) & 255u) == 0, RGK_EALIGN,
              "workspace must be 256-byte aligned");
  RGK_CHECK_DEVICE();
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  const int bw = (int)(E / H);
  (void)bw;
  return run_rglru(x, segment_pos, pos_dtype, p, h0, nullptr, 0, B, T, E, H, dtype, gates_impl,
                   w.wpack, w.a, w.xn, w.scan, y, h_last, s);
}

int rgk_recurrent_path_prefill(const void* xb, const void* yb, const void* segment_pos,
                               int pos_dtype, const rgk_params* p, const float* h0, int64_t B,
                               int64_t T, int64_t E, int H, int W, int dtype, int gates_impl,
                               void* out, float* h_last, void* conv_cache_out, void* workspace,
                               size_t workspace_bytes, void* stream) {
  int rc = check_common(B, T, E, dtype);
  if (rc) return rc;
  if ((rc = check_heads(E, H))) return rc;
  if ((rc = check_params(p, true))) return rc;
  RGK_REQUIRE(W == 4, RGK_ESHAPE, "temporal width %d is not supported (only 4)", W);
  RGK_REQUIRE(pos_dtype == RGK_I32 || pos_dtype == RGK_I64, RGK_EINVAL, "unknown index dtype");
  RGK_REQUIRE(gates_impl >= RGK_GATES_AUTO && gates_impl <= RGK_GATES_FUSED_EXACT, RGK_EINVAL,
              "unknown gates_impl %d", gates_impl);
  RGK_REQUIRE(xb && segment_pos && out, RGK_EINVAL, "NULL pointer argument");
  RGK_REQUIRE(aligned16(xb) && aligned16(yb) && aligned16(out) && aligned16(h0) &&
                  aligned16(h_last) && aligned16(conv_cache_out),
              RGK_EALIGN, "pointers must be 16-byte aligned");
  RGK_REQUIRE(T >= 1 || B * E == 0, RGK_ESHAPE, "prefill needs at least one token");
  if (B * T * E == 0) return RGK_OK;
  const PathWs w = carve(workspace, B, T, E, dtype);
  RGK_REQUIRE(workspace != nullptr && workspace_bytes >= w.total, RGK_EWORKSPACE,
              "workspace of %zu bytes needed, %zu given", w.total, workspace_bytes);
  RGK_REQUIRE((reinterpret_cast<uintptr_t>(workspace) & 255u) == 0, RGK_EALIGN,
              "workspace must be 256-byte aligned");
  RGK_CHECK_DEVICE();
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  const int bw = (int)(E / H);
  (void)bw;
  return run_rglru(w.c, segment_pos, pos_dtype, p, h0, yb, 0, B, T, E, H, dtype, gates_impl,
                   w.wpack, w.a, w.xn, w.scan, out, h_last, s, xb, conv_cache_out);
}

int rgk_dense_linear(const void* x, const void* weight, const void* bias, int64_t M, int64_t K,
                     int64_t N, int dtype, int act, void* out, int* status, void* stream) {
  RGK_REQUIRE(dtype == RGK_F32 || dtype == RGK_BF16, RGK_EINVAL, "unknown dtype %d", dtype);
  RGK_REQUIRE(act == RGK_ACT_NONE || act == RGK_ACT_GELU_TANH, RGK_EINVAL, "unknown act %d", act);
  RGK_REQUIRE(M >= 0 && K >= 1 && N >= 1, RGK_EINVAL, "bad size (M=%lld K=%lld N=%lld)",
              (long long)M, (long long)K, (long long)N);
  RGK_REQUIRE(x && weight && out, RGK_EINVAL, "NULL pointer argument");
  RGK_REQUIRE(aligned16(x) && aligned16(weight) && aligned16(out) && aligned16(bias), RGK_EALIGN,
              "pointers must be 16-byte aligned");
  RGK_REQUIRE(rgk::dense_tc_supported(dtype, M > 0 ? M : 1, K, N), RGK_ESHAPE,
              "the tensor-core linear covers bfloat16 with K and N multiples of 8 "
              "(dtype %d, K=%lld, N=%lld)", dtype, (long long)K, (long long)N);
  if (M == 0) return RGK_OK;
  RGK_CHECK_DEVICE();
  const rgk::RowsMatrix mat = {weight, bias, out, (int)N};
  RGK_CUDA(rgk::launch_dense_tc(x, &mat, 1, nullptr, M, (int)K, act == RGK_ACT_GELU_TANH, status,
                                static_cast<cudaStream_t>(stream)),
           "dense linear launch");
  return RGK_OK;
}

static constexpr int kRowsGemm = 8;                // rows that the kernel that streams weights into registers takes

// Up to how many rows the few-row kernels take a projection.  Every SM has weights to stream there, where
// a pair of CTAs of the GEMM walks all of K for its tile: at 128 rows 9.2 us against 11.2 for 2560 x
// 2560 and 14.9 against 24.1 for 7680 -> 2560, at 199 12.8 / 11.4 and 17.9 / 25.4, at 300 21.3 / 27.0 for
// the latter; wide outputs fill the chip sooner (2560 -> 15360: 16.6 / 19.0 at 48 rows, 21.7 / 20.3 at 128).
// From two tiles of 128 features an SM on (logits) the persistent form of the GEMM has its epilogues under the
// loads of the next tile and the few-row kernel has not: 2560 -> 256000 at 9, 33 and 64 rows 307 / 226,
// 421 / 229 and 360 / 226, 2560 -> 64000 86 / 76, 111 / 77 and 106 / 74; plain: nothing but the cap follows.
static bool few_rows(int64_t M, int64_t K, int64_t N, bool plain = false) {
  if (plain && N >= 2 * 128 * 148) return false;
  return M <= (N >= 4 * K ? 96 : (K >= 2 * N ? 352 : 160));
}

// Projections of few rows on the kernel for their number: up to kRowsGemm rows the one that streams
// weights into registers, above that the one with 128-feature tensor-core tiles, and the GEMM of many rows
// where that is faster (its epilogues have gelu or a residual, not both).
static cudaError_t few_rows_linear(const void* x, const rgk::RowsMatrix* mats, int n_mats,
                                   const void* residual, int64_t M, int K, int act, float cap, int* status,
                                   bool early, bool wide, cudaStream_t s) {
  if (M <= kRowsGemm && rgk::rows_gemm_suits(M, K))
    return rgk::launch_rows_gemm(x, nullptr, 0.0f, mats, n_mats, residual, M, K, act, cap, early, s);
  const bool plain = n_mats == 1 && act == 0 && residual == nullptr;
  if (!few_rows(M, K, mats[0].n, plain) && (act == 0 || residual == nullptr))
    return rgk::launch_dense_tc(x, mats, n_mats, residual, M, K, act, status, s, cap);
  return rgk::launch_dense_small(x, mats, n_mats, residual, M, K, act, cap, status, early, wide, s);
}

// The same with RMSNorm of the rows in front: inside the kernel, or as one of its own into xn.
static cudaError_t few_rows_norm_linear(const void* x, const void* scale, float eps, void* xn,
                                        const rgk::RowsMatrix* mats, int n_mats, int64_t M, int K, int act,
                                        int* status, bool early, cudaStream_t s) {
  if (M <= kRowsGemm && rgk::rows_gemm_supported(RGK_BF16, M, K, 8, true))
    return rgk::launch_rows_gemm(x, scale, eps, mats, n_mats, nullptr, M, K, act, 0.0f, early, s);
  cudaError_t e = rgk::launch_rmsnorm_rows(x, scale, M, K, eps, early, xn, s);
  if (e != cudaSuccess) return e;
  return few_rows_linear(xn, mats, n_mats, nullptr, M, K, act, 0.0f, status, true, true, s);
}

// Projections of a prompt's rows.
static cudaError_t prompt_linear(const void* x, const rgk::RowsMatrix* mats, int n_mats, const void* residual,
                                 int64_t M, int K, int act, int* status, cudaStream_t s) {
  if (few_rows(M, K, mats[0].n))
    return few_rows_linear(x, mats, n_mats, residual, M, K, act, 0.0f, status, false, true, s);
  return rgk::launch_dense_tc(x, mats, n_mats, residual, M, K, act, status, s);
}
// RMSNorm of a prompt's rows: a block per row while the warps of the other kernel would not fill the chip.
static cudaError_t prompt_norm(const void* x, const void* scale, int64_t M, int64_t D, float eps, void* out,
                               cudaStream_t s) {
  return M <= 512 ? rgk::launch_rmsnorm_rows(x, scale, M, D, eps, false, out, s)
                  : rgk::launch_rmsnorm(x, scale, M, D, eps, RGK_BF16, out, s);
}

int rgk_dense_linear_small(const void* x, const void* weight, const void* bias, const void* residual,
                           int64_t M, int64_t K, int64_t N, int dtype, int act, void* out,
                           int* status, void* stream) {
  RGK_REQUIRE(dtype == RGK_F32 || dtype == RGK_BF16, RGK_EINVAL, "unknown dtype %d", dtype);
  RGK_REQUIRE(act == RGK_ACT_NONE || act == RGK_ACT_GELU_TANH || act == RGK_ACT_GEGLU, RGK_EINVAL,
              "unknown act %d", act);
  RGK_REQUIRE(M >= 0 && K >= 1 && N >= 1, RGK_EINVAL, "bad size (M=%lld K=%lld N=%lld)",
              (long long)M, (long long)K, (long long)N);
  RGK_REQUIRE(x && weight && out, RGK_EINVAL, "NULL pointer argument");
  RGK_REQUIRE(act != RGK_ACT_GEGLU || (residual == nullptr && bias != nullptr && N % 128 == 0),
              RGK_ESHAPE, "GeGLU takes the packed up-projection with its bias (N = 2 X with X a "
              "multiple of 64, N=%lld) and no residual", (long long)N);
  RGK_REQUIRE(aligned16(x) && aligned16(weight) && aligned16(out) && aligned16(bias) &&
              aligned16(residual), RGK_EALIGN, "pointers must be 16-byte aligned");
  RGK_REQUIRE(M <= 256 && rgk::dense_small_supported(dtype, M > 0 ? M : 1, K, N), RGK_ESHAPE,
              "the few-row linear covers bfloat16 with M <= 256 and K and N multiples of 8 "
              "(dtype %d, M=%lld, K=%lld, N=%lld)", dtype, (long long)M, (long long)K, (long long)N);
  if (M == 0) return RGK_OK;
  RGK_CHECK_DEVICE();
  const rgk::RowsMatrix mat = {weight, bias, out, (int)N};
  RGK_CUDA(few_rows_linear(x, &mat, 1, residual, M, (int)K, act, 0.0f, status, false, true,
                           static_cast<cudaStream_t>(stream)),
           "few-row dense linear launch");
  return RGK_OK;
}

int rgk_dense_linear_small_pair(const void* x, const void* weight_a, const void* bias_a,
                                const void* weight_b, const void* bias_b, int64_t M, int64_t K,
                                int64_t N_a, int64_t N_b, int dtype, void* out_a, void* out_b,
                                int* status, void* stream) {
  RGK_REQUIRE(dtype == RGK_F32 || dtype == RGK_BF16, RGK_EINVAL, "unknown dtype %d", dtype);
  RGK_REQUIRE(M >= 0 && K >= 1 && N_a >= 1 && N_b >= 1, RGK_EINVAL,
              "bad size (M=%lld K=%lld N_a=%lld N_b=%lld)", (long long)M, (long long)K,
              (long long)N_a, (long long)N_b);
  RGK_REQUIRE(x && weight_a && weight_b && out_a && out_b, RGK_EINVAL, "NULL pointer argument");
  RGK_REQUIRE(aligned16(x) && aligned16(weight_a) && aligned16(weight_b) && aligned16(out_a) &&
              aligned16(out_b) && aligned16(bias_a) && aligned16(bias_b), RGK_EALIGN,
              "pointers must be 16-byte aligned");
  RGK_REQUIRE(M <= 256 && rgk::dense_small_supported(dtype, M > 0 ? M : 1, K, N_a + N_b) && N_a % 128 == 0 &&
              N_b % 8 == 0, RGK_ESHAPE,
              "the paired few-row linear covers bfloat16 with M <= 256, K and N_b multiples of 8 and "
              "N_a a multiple of 128 (dtype %d, M=%lld, K=%lld, N_a=%lld, N_b=%lld)", dtype,
              (long long)M, (long long)K, (long long)N_a, (long long)N_b);
  if (M == 0) return RGK_OK;
  RGK_CHECK_DEVICE();
  const rgk::RowsMatrix mats[2] = {{weight_a, bias_a, out_a, (int)N_a}, {weight_b, bias_b, out_b, (int)N_b}};
  RGK_CUDA(few_rows_linear(x, mats, 2, nullptr, M, (int)K, 0, 0.0f, status, false, true,
                           static_cast<cudaStream_t>(stream)),
           "paired few-row dense linear launch");
  return RGK_OK;
}

int rgk_embed(const void* tokens, int token_dtype, const void* table, int64_t M, int64_t V,
              int64_t D, float scale, int dtype, void* out, void* stream) {
  RGK_REQUIRE(dtype == RGK_F32 || dtype == RGK_BF16, RGK_EINVAL, "unknown dtype %d", dtype);
  RGK_REQUIRE(token_dtype == RGK_I32 || token_dtype == RGK_I64, RGK_EINVAL,
              "unknown token dtype %d", token_dtype);
  RGK_REQUIRE(M >= 0 && V >= 1 && D >= 1, RGK_EINVAL, "bad size (M=%lld V=%lld D=%lld)",
              (long long)M, (long long)V, (long long)D);
  RGK_REQUIRE(tokens && table && out, RGK_EINVAL, "NULL pointer argument");
  RGK_REQUIRE(aligned16(table) && aligned16(out), RGK_EALIGN, "pointers must be 16-byte aligned");
  RGK_REQUIRE((D * (int64_t)elem_size(dtype)) % 16 == 0, RGK_ESHAPE,
              "the embedding width must be a multiple of a 16-byte pack (D=%lld)", (long long)D);
  if (M == 0) return RGK_OK;
  RGK_CHECK_DEVICE();
  RGK_CUDA(rgk::launch_embed(tokens, token_dtype == RGK_I64, table, M, V, D, scale, dtype, out,
                             static_cast<cudaStream_t>(stream)),
           "embed launch");
  return RGK_OK;
}

int rgk_logits(const void* x, const void* table, int64_t M, int64_t D, int64_t V, float cap,
               int dtype, void* out, int* status, void* stream) {
  RGK_REQUIRE(dtype == RGK_F32 || dtype == RGK_BF16, RGK_EINVAL, "unknown dtype %d", dtype);
  RGK_REQUIRE(M >= 0 && D >= 1 && V >= 1, RGK_EINVAL, "bad size (M=%lld D=%lld V=%lld)",
              (long long)M, (long long)D, (long long)V);
  RGK_REQUIRE(cap >= 0.0f, RGK_EINVAL, "the soft cap must not be negative");
  RGK_REQUIRE(x && table && out, RGK_EINVAL, "NULL pointer argument");
  RGK_REQUIRE(aligned16(x) && aligned16(table) && aligned16(out), RGK_EALIGN,
              "pointers must be 16-byte aligned");
  RGK_REQUIRE(rgk::dense_tc_supported(dtype, M > 0 ? M : 1, D, V), RGK_ESHAPE,
              "the tensor-core logits cover bfloat16 with D and V multiples of 8 "
              "(dtype %d, D=%lld, V=%lld)", dtype, (long long)D, (long long)V);
  if (M == 0) return RGK_OK;
  RGK_CHECK_DEVICE();
  if (M <= 256) {
    const rgk::RowsMatrix mat = {table, nullptr, out, (int)V};
    RGK_CUDA(few_rows_linear(x, &mat, 1, nullptr, M, (int)D, 0, cap, status, false, true,
                             static_cast<cudaStream_t>(stream)),
             "logits launch");
    return RGK_OK;
  }
  const rgk::RowsMatrix mat = {table, nullptr, out, (int)V};
  RGK_CUDA(rgk::launch_dense_tc(x, &mat, 1, nullptr, M, (int)D, 0, status, static_cast<cudaStream_t>(stream),
                                cap),
           "logits launch");
  return RGK_OK;
}

int rgk_argmax(const void* x, int64_t M, int64_t V, int dtype, int* out, void* stream) {
  RGK_REQUIRE(dtype == RGK_F32 || dtype == RGK_BF16, RGK_EINVAL, "unknown dtype %d", dtype);
  RGK_REQUIRE(M >= 0 && V >= 1 && V < ((int64_t)1 << 31), RGK_EINVAL, "bad size (M=%lld V=%lld)",
              (long long)M, (long long)V);
  RGK_REQUIRE(x && out, RGK_EINVAL, "NULL pointer argument");
  RGK_REQUIRE(aligned16(x), RGK_EALIGN, "pointers must be 16-byte aligned");
  if (M == 0) return RGK_OK;
  RGK_CHECK_DEVICE();
  RGK_CUDA(rgk::launch_argmax(x, M, V, dtype, out, static_cast<cudaStream_t>(stream)),
           "argmax launch");
  return RGK_OK;
}

int rgk_geglu_bias(const void* up, const void* bias, int64_t M, int64_t X, int dtype, void* out,
                   void* stream) {
  RGK_REQUIRE(dtype == RGK_F32 || dtype == RGK_BF16, RGK_EINVAL, "unknown dtype %d", dtype);
  RGK_REQUIRE(M >= 0 && X >= 1, RGK_EINVAL, "bad size (M=%lld X=%lld)", (long long)M, (long long)X);
  RGK_REQUIRE(up && bias && out, RGK_EINVAL, "NULL pointer argument");
  RGK_REQUIRE(aligned16(up) && aligned16(bias) && aligned16(out), RGK_EALIGN,
              "pointers must be 16-byte aligned");
  RGK_REQUIRE((X * (int64_t)elem_size(dtype)) % 16 == 0, RGK_ESHAPE,
              "the expanded width must be a multiple of a 16-byte pack (X=%lld)", (long long)X);
  if (M == 0) return RGK_OK;
  RGK_CHECK_DEVICE();
  RGK_CUDA(rgk::launch_geglu_bias(up, bias, M, X, dtype, out, static_cast<cudaStream_t>(stream)),
           "geglu launch");
  return RGK_OK;
}

size_t rgk_block_workspace_bytes(int64_t B, int64_t T, int64_t D, int64_t E, int dtype) {
  if (B < 0 || T < 0 || D < 0 || E < 0 || (dtype != RGK_F32 && dtype != RGK_BF16)) return 0;
  if (T < 1) T = 1;
  const size_t act = up256(static_cast<size_t>(B) * T * E * elem_size(dtype));
  return carve(nullptr, B, T, E, dtype).total + 2 * act;
}

// Validation and launches shared by the block entry points.  x_in is what linear_x / linear_y read
// (the block input, or its RMSNorm), residual (may be NULL) is added to linear_out's result, `ws` is
// a block workspace.
static int block_prefill_impl(const void* x_in, const void* residual, const void* segment_pos,
                              int pos_dtype, const rgk_block_params* p, int64_t B, int64_t T,
                              int64_t D, int64_t E, int H, int dtype, void* out, float* h_last,
                              void* conv_cache_out, void* workspace, cudaStream_t s) {
  const PathWs w = carve(workspace, B, T, E, dtype);
  const size_t act = up256(static_cast<size_t>(B) * T * E * elem_size(dtype));
  char* xb = static_cast<char*>(workspace) + w.total;   // later reused for the joined output
  char* yb = xb + act;
  int* status = static_cast<int*>(workspace);
  const int64_t M = B * T;
  int rc;
  // both input projections in one launch; the y branch's gelu in its epilogue, in float32 (the join of the
  // RG-LRU kernel would evaluate it with the packed bfloat16 tanh)
  const rgk::RowsMatrix in[2] = {{p->linear_y_w, p->linear_y_b, yb, (int)E},
                                 {p->linear_x_w, p->linear_x_b, xb, (int)E}};
  RGK_CUDA(prompt_linear(x_in, in, 2, nullptr, M, (int)D, 1, status, s),
           "linear_y, linear_x launch");
  // Conv1D inside the RG-LRU kernel where that kernel applies (the joined output y * gelu(yb) then
  // goes to the conv-output buffer, which the fused form does not use), else as its own kernel
  // (a warp reads its tile of yb before it writes the same tile of the output); with a separate
  // conv kernel xb has been consumed by then and receives the output
  const bool fused = rgk::rglru_chan_supported(dtype, (int)(E / H), B, T) && conv_fusion_enabled();
  char* joined = fused ? yb : xb;
  if ((rc = run_rglru(w.c, segment_pos, pos_dtype, &p->path, nullptr, yb, 1, B, T, E, H,
                      dtype, RGK_GATES_AUTO, w.wpack, w.a, w.xn, w.scan, joined, h_last, s, xb,
                      conv_cache_out)))
    return rc;
  const rgk::RowsMatrix last = {p->linear_out_w, p->linear_out_b, out, (int)D};
  RGK_CUDA(prompt_linear(joined, &last, 1, residual, M, (int)E, 0, status, s),
           "linear_out launch");
  return RGK_OK;
}

static int check_block_args(const void* x, const void* segment_pos, int pos_dtype,
                            const rgk_block_params* p, int64_t B, int64_t T, int64_t D, int64_t E,
                            int H, int W, int dtype, const void* out, const float* h_last,
                            const void* conv_cache_out) {
  int rc = check_common(B, T, E, dtype);
  if (rc) return rc;
  if ((rc = check_heads(E, H))) return rc;
  RGK_REQUIRE(p != nullptr, RGK_EINVAL, "params is NULL");
  if ((rc = check_params(&p->path, true))) return rc;
  RGK_REQUIRE(p->linear_y_w && p->linear_x_w && p->linear_out_w, RGK_EINVAL,
              "a linear weight pointer is NULL");
  RGK_REQUIRE(aligned16(p->linear_y_w) && aligned16(p->linear_x_w) && aligned16(p->linear_out_w) &&
                  aligned16(p->linear_y_b) && aligned16(p->linear_x_b) && aligned16(p->linear_out_b),
              RGK_EALIGN, "parameter pointers must be 16-byte aligned");
  RGK_REQUIRE(W == 4, RGK_ESHAPE, "temporal width %d is not supported (only 4)", W);
  RGK_REQUIRE(pos_dtype == RGK_I32 || pos_dtype == RGK_I64, RGK_EINVAL, "unknown index dtype");
  RGK_REQUIRE(x && segment_pos && out, RGK_EINVAL, "NULL pointer argument");
  RGK_REQUIRE(aligned16(x) && aligned16(out) && aligned16(h_last) && aligned16(conv_cache_out),
              RGK_EALIGN, "pointers must be 16-byte aligned");
  RGK_REQUIRE(D >= 8 && D % 8 == 0, RGK_ESHAPE, "block width %lld is not a multiple of 8",
              (long long)D);
  const int bw = (int)(E / H);
  RGK_REQUIRE(rgk::gates_tc_supported(dtype, bw, B * T > 0 ? B * T : 1), RGK_ESHAPE,
              "the fused block covers bfloat16 with head width 256 only (dtype %d, head width %d)",
              dtype, bw);
  return RGK_OK;
}

int rgk_recurrent_block_prefill(const void* x, const void* segment_pos, int pos_dtype,
                                const rgk_block_params* p, int64_t B, int64_t T, int64_t D,
                                int64_t E, int H, int W, int dtype, void* out, float* h_last,
                                void* conv_cache_out, void* workspace, size_t workspace_bytes,
                                void* stream) {
  int rc = check_block_args(x, segment_pos, pos_dtype, p, B, T, D, E, H, W, dtype, out, h_last,
                            conv_cache_out);
  if (rc) return rc;
  if (B * T * E == 0) return RGK_OK;
  const size_t need = rgk_block_workspace_bytes(B, T, D, E, dtype);
  RGK_REQUIRE(workspace != nullptr && workspace_bytes >= need, RGK_EWORKSPACE,
              "workspace of %zu bytes needed, %zu given", need, workspace_bytes);
  RGK_REQUIRE((reinterpret_cast<uintptr_t>(workspace) & 255u) == 0, RGK_EALIGN,
              "workspace must be 256-byte aligned");
  RGK_CHECK_DEVICE();
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  return block_prefill_impl(x, nullptr, segment_pos, pos_dtype, p, B, T, D, E, H, dtype, out, h_last,
                            conv_cache_out, workspace, s);
}

int rgk_rmsnorm(const void* x, const void* scale, int64_t M, int64_t D, float eps, int dtype,
                void* out, void* stream) {
  RGK_REQUIRE(dtype == RGK_F32 || dtype == RGK_BF16, RGK_EINVAL, "unknown dtype %d", dtype);
  RGK_REQUIRE(M >= 0 && D >= 1, RGK_EINVAL, "bad size (M=%lld D=%lld)", (long long)M, (long long)D);
  RGK_REQUIRE(x && scale && out, RGK_EINVAL, "NULL pointer argument");
  RGK_REQUIRE(aligned16(x) && aligned16(scale) && aligned16(out), RGK_EALIGN,
              "pointers must be 16-byte aligned");
  RGK_REQUIRE(rgk::rmsnorm_supported(dtype, D), RGK_ESHAPE,
              "RMSNorm covers widths that are multiples of a 16-byte pack, up to 1024 packs "
              "(dtype %d, D=%lld)", dtype, (long long)D);
  if (M == 0) return RGK_OK;
  RGK_CHECK_DEVICE();
  RGK_CUDA(rgk::launch_rmsnorm(x, scale, M, D, eps, dtype, out, static_cast<cudaStream_t>(stream)),
           "rmsnorm launch");
  return RGK_OK;
}

int rgk_add_rmsnorm(const void* a, const void* b, const void* scale, int64_t M, int64_t D, float eps,
                    int dtype, void* sum_out, void* out, void* stream) {
  RGK_REQUIRE(dtype == RGK_F32 || dtype == RGK_BF16, RGK_EINVAL, "unknown dtype %d", dtype);
  RGK_REQUIRE(M >= 0 && D >= 1, RGK_EINVAL, "bad size (M=%lld D=%lld)", (long long)M, (long long)D);
  RGK_REQUIRE(a && b && scale && sum_out && out, RGK_EINVAL, "NULL pointer argument");
  RGK_REQUIRE(aligned16(a) && aligned16(b) && aligned16(scale) && aligned16(sum_out) && aligned16(out),
              RGK_EALIGN, "pointers must be 16-byte aligned");
  RGK_REQUIRE(rgk::rmsnorm_supported(dtype, D), RGK_ESHAPE,
              "RMSNorm covers widths that are multiples of a 16-byte pack, up to 1024 packs "
              "(dtype %d, D=%lld)", dtype, (long long)D);
  if (M == 0) return RGK_OK;
  RGK_CHECK_DEVICE();
  RGK_CUDA(rgk::launch_rmsnorm(a, scale, M, D, eps, dtype, out, static_cast<cudaStream_t>(stream), b,
                               sum_out),
           "add + rmsnorm launch");
  return RGK_OK;
}

size_t rgk_residual_workspace_bytes(int64_t B, int64_t T, int64_t D, int64_t E, int dtype) {
  const size_t block = rgk_block_workspace_bytes(B, T, D, E, dtype);
  if (block == 0) return 0;
  if (T < 1) T = 1;
  return block + up256(static_cast<size_t>(B) * T * D * elem_size(dtype));
}

int rgk_residual_block_prefill(const void* x, const void* segment_pos, int pos_dtype,
                               const rgk_block_params* p, const void* norm_scale, float eps,
                               int64_t B, int64_t T, int64_t D, int64_t E, int H, int W, int dtype,
                               void* out, float* h_last, void* conv_cache_out, void* workspace,
                               size_t workspace_bytes, void* stream) {
  int rc = check_block_args(x, segment_pos, pos_dtype, p, B, T, D, E, H, W, dtype, out, h_last,
                            conv_cache_out);
  if (rc) return rc;
  RGK_REQUIRE(norm_scale != nullptr, RGK_EINVAL, "norm_scale is NULL");
  RGK_REQUIRE(aligned16(norm_scale), RGK_EALIGN, "norm_scale must be 16-byte aligned");
  RGK_REQUIRE(rgk::rmsnorm_supported(dtype, D), RGK_ESHAPE, "block width %lld is not covered by the "
              "RMSNorm kernel", (long long)D);
  if (B * T * E == 0) return RGK_OK;
  const size_t block = rgk_block_workspace_bytes(B, T, D, E, dtype);
  const size_t need = rgk_residual_workspace_bytes(B, T, D, E, dtype);
  RGK_REQUIRE(workspace != nullptr && workspace_bytes >= need, RGK_EWORKSPACE,
              "workspace of %zu bytes needed, %zu given", need, workspace_bytes);
  RGK_REQUIRE((reinterpret_cast<uintptr_t>(workspace) & 255u) == 0, RGK_EALIGN,
              "workspace must be 256-byte aligned");
  RGK_CHECK_DEVICE();
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  void* xn = static_cast<char*>(workspace) + block;      // temporal_pre_norm(x)
  RGK_CUDA(prompt_norm(x, norm_scale, B * T, D, eps, xn, s), "rmsnorm launch");
  return block_prefill_impl(xn, x, segment_pos, pos_dtype, p, B, T, D, E, H, dtype, out, h_last,
                            conv_cache_out, workspace, s);
}

// ---- MLP block and the channel half of the residual block --------------------------------------

static size_t mlp_pack_w_bytes(int64_t D, int64_t X) { return up256(static_cast<size_t>(2 * X) * D * 2); }

size_t rgk_mlp_pack_bytes(int64_t D, int64_t X) {
  if (D < 8 || X < 64 || D % 8 != 0 || X % 64 != 0) return 0;
  return mlp_pack_w_bytes(D, X) + up256(static_cast<size_t>(2 * X) * 2);
}

int rgk_pack_mlp_up(const void* w, const void* b, int64_t D, int64_t X, int dtype, void* packed_out,
                    void* stream) {
  RGK_REQUIRE(dtype == RGK_BF16, RGK_ESHAPE, "the packed MLP weights are bfloat16 only (dtype %d)",
              dtype);
  RGK_REQUIRE(w && b && packed_out, RGK_EINVAL, "NULL pointer argument");
  RGK_REQUIRE(D >= 8 && D % 8 == 0 && X >= 64 && X % 64 == 0 && D < (1 << 24) && X < (1 << 23),
              RGK_ESHAPE, "the MLP kernels cover widths that are multiples of 8 and expanded widths "
              "that are multiples of 64 (D=%lld, X=%lld)", (long long)D, (long long)X);
  RGK_REQUIRE(aligned16(w) && aligned16(b) && aligned16(packed_out), RGK_EALIGN,
              "pointers must be 16-byte aligned");
  RGK_CHECK_DEVICE();
  char* out = static_cast<char*>(packed_out);
  RGK_CUDA(rgk::launch_pack_mlp_up(w, b, (int)D, (int)X, out, out + mlp_pack_w_bytes(D, X),
                                   static_cast<cudaStream_t>(stream)),
           "pack_mlp_up launch");
  return RGK_OK;
}

size_t rgk_mlp_workspace_bytes(int64_t M, int64_t D, int64_t X, int dtype) {
  if (M < 0 || D < 1 || X < 1 || dtype != RGK_BF16) return 0;
  if (M < 1) M = 1;
  return 256 + up256(static_cast<size_t>(M) * X * 2) + up256(static_cast<size_t>(M) * D * 2);
}

// out = ffw_down(gelu(up_0) * up_1) [+ residual]; x_in is the MLP's input.
static int mlp_impl(const void* x_in, const void* packed_up, const void* down_w, const void* down_b,
                    const void* residual, int64_t M, int64_t D, int64_t X, void* out,
                    void* workspace, cudaStream_t s) {
  int* status = static_cast<int*>(workspace);
  char* act = static_cast<char*>(workspace) + 256;
  const char* pw = static_cast<const char*>(packed_up);
  const rgk::RowsMatrix up = {pw, pw + mlp_pack_w_bytes(D, X), act, (int)(2 * X)};
  RGK_CUDA(prompt_linear(x_in, &up, 1, nullptr, M, (int)D, 2, status, s), "ffw_up launch");
  const rgk::RowsMatrix down = {down_w, down_b, out, (int)D};
  RGK_CUDA(prompt_linear(act, &down, 1, residual, M, (int)X, 0, status, s), "ffw_down launch");
  return RGK_OK;
}

static int check_mlp_args(const void* x, const void* packed_up, const void* down_w,
                          const void* down_b, int64_t M, int64_t D, int64_t X, int dtype,
                          const void* out, const void* workspace, size_t workspace_bytes) {
  RGK_REQUIRE(dtype == RGK_BF16, RGK_ESHAPE, "the MLP kernels are bfloat16 only (dtype %d)", dtype);
  RGK_REQUIRE(M >= 0 && M < ((int64_t)1 << 31), RGK_EINVAL, "bad row count %lld", (long long)M);
  RGK_REQUIRE(D >= 8 && D % 8 == 0 && X >= 64 && X % 64 == 0 && D < (1 << 24) && X < (1 << 23),
              RGK_ESHAPE, "the MLP kernels cover widths that are multiples of 8 and expanded widths "
              "that are multiples of 64 (D=%lld, X=%lld)", (long long)D, (long long)X);
  RGK_REQUIRE(x && packed_up && down_w && out, RGK_EINVAL, "NULL pointer argument");
  RGK_REQUIRE(aligned16(x) && aligned16(packed_up) && aligned16(down_w) && aligned16(down_b) &&
                  aligned16(out),
              RGK_EALIGN, "pointers must be 16-byte aligned");
  if (M == 0) return RGK_OK;
  const size_t need = rgk_mlp_workspace_bytes(M, D, X, dtype);
  RGK_REQUIRE(workspace != nullptr && workspace_bytes >= need, RGK_EWORKSPACE,
              "workspace of %zu bytes needed, %zu given", need, workspace_bytes);
  RGK_REQUIRE((reinterpret_cast<uintptr_t>(workspace) & 255u) == 0, RGK_EALIGN,
              "workspace must be 256-byte aligned");
  return RGK_OK;
}

int rgk_mlp_block(const void* x, const void* packed_up, const void* down_w, const void* down_b,
                  const void* residual, int64_t M, int64_t D, int64_t X, int dtype, void* out,
                  void* workspace, size_t workspace_bytes, void* stream) {
  int rc = check_mlp_args(x, packed_up, down_w, down_b, M, D, X, dtype, out, workspace,
                          workspace_bytes);
  if (rc) return rc;
  RGK_REQUIRE(aligned16(residual), RGK_EALIGN, "pointers must be 16-byte aligned");
  if (M == 0) return RGK_OK;
  RGK_CHECK_DEVICE();
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  return mlp_impl(x, packed_up, down_w, down_b, residual, M, D, X, out, workspace, s);
}

int rgk_residual_channel(const void* residual_in, const void* norm_scale, float eps,
                         const void* packed_up, const void* down_w, const void* down_b, int64_t M,
                         int64_t D, int64_t X, int dtype, void* out, void* workspace,
                         size_t workspace_bytes, void* stream) {
  int rc = check_mlp_args(residual_in, packed_up, down_w, down_b, M, D, X, dtype, out, workspace,
                          workspace_bytes);
  if (rc) return rc;
  RGK_REQUIRE(norm_scale != nullptr, RGK_EINVAL, "norm_scale is NULL");
  RGK_REQUIRE(aligned16(norm_scale), RGK_EALIGN, "norm_scale must be 16-byte aligned");
  RGK_REQUIRE(rgk::rmsnorm_supported(dtype, D), RGK_ESHAPE, "block width %lld is not covered by the "
              "RMSNorm kernel", (long long)D);
  if (M == 0) return RGK_OK;
  RGK_CHECK_DEVICE();
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  void* xn = static_cast<char*>(workspace) + 256 + up256(static_cast<size_t>(M) * X * 2);
  RGK_CUDA(prompt_norm(residual_in, norm_scale, M, D, eps, xn, s), "rmsnorm launch");
  return mlp_impl(xn, packed_up, down_w, down_b, residual_in, M, D, X, out, workspace, s);
}

// ---- local attention ----------------------------------------------------------------------------

int rgk_rope(void* x, const void* segment_pos, int pos_dtype, int64_t rows, int heads, int head_dim,
             int dtype, void* stream) {
  RGK_REQUIRE(dtype == RGK_F32 || dtype == RGK_BF16, RGK_EINVAL, "unknown dtype %d", dtype);
  RGK_REQUIRE(pos_dtype == RGK_I32 || pos_dtype == RGK_I64, RGK_EINVAL, "unknown index dtype");
  RGK_REQUIRE(rows >= 0 && heads >= 1 && head_dim >= 4 && head_dim % 4 == 0, RGK_EINVAL,
              "bad size (rows=%lld heads=%d head_dim=%d)", (long long)rows, heads, head_dim);
  RGK_REQUIRE(x && segment_pos, RGK_EINVAL, "NULL pointer argument");
  if (rows == 0) return RGK_OK;
  RGK_CHECK_DEVICE();
  RGK_CUDA(rgk::launch_rope(x, segment_pos, pos_dtype == RGK_I64, rows, heads, head_dim, dtype,
                            static_cast<cudaStream_t>(stream)),
           "rope launch");
  return RGK_OK;
}

size_t rgk_attention_workspace_bytes(int64_t B, int64_t T) {
  if (B < 0 || T < 0) return 0;
  return rgk::attention_workspace_bytes(B < 1 ? 1 : B, T < 1 ? 1 : T);
}

int rgk_local_attention_prefill(const void* q, const void* k, const void* v, const void* segment_pos,
                                int pos_dtype, int64_t B, int64_t T, int N, int head_dim, int window,
                                int dtype, void* out, void* workspace, size_t workspace_bytes,
                                void* stream) {
  RGK_REQUIRE(pos_dtype == RGK_I32 || pos_dtype == RGK_I64, RGK_EINVAL, "unknown index dtype");
  RGK_REQUIRE(B >= 0 && T >= 0 && N >= 1 && window >= 1, RGK_EINVAL, "bad size");
  RGK_REQUIRE(q && k && v && segment_pos && out, RGK_EINVAL, "NULL pointer argument");
  RGK_REQUIRE(aligned16(q) && aligned16(k) && aligned16(v) && aligned16(out), RGK_EALIGN,
              "pointers must be 16-byte aligned");
  RGK_REQUIRE(rgk::attention_supported(dtype, head_dim, B > 0 ? B : 1, T > 0 ? T : 1, N), RGK_ESHAPE,
              "the attention kernel covers bfloat16 with head dimension 256 (dtype %d, head_dim %d)",
              dtype, head_dim);
  if (B * T == 0) return RGK_OK;
  const size_t need = rgk_attention_workspace_bytes(B, T);
  RGK_REQUIRE(workspace != nullptr && workspace_bytes >= need, RGK_EWORKSPACE,
              "workspace of %zu bytes needed, %zu given", need, workspace_bytes);
  RGK_REQUIRE((reinterpret_cast<uintptr_t>(workspace) & 255u) == 0, RGK_EALIGN,
              "workspace must be 256-byte aligned");
  RGK_CHECK_DEVICE();
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  RGK_CUDA(rgk::launch_attention_prefill(const_cast<void*>(q), const_cast<void*>(k), v, segment_pos,
                                         pos_dtype == RGK_I64, B, T, N, window, false, nullptr, nullptr,
                                         nullptr, out, workspace, s),
           "attention launch");
  return RGK_OK;
}

// [attention workspace | q, later the encoded heads | k | v | the normalised input]
size_t rgk_attention_block_workspace_bytes(int64_t B, int64_t T, int64_t D) {
  if (B < 0 || T < 0 || D < 256) return 0;
  const size_t m = static_cast<size_t>(B < 1 ? 1 : B) * (T < 1 ? 1 : T);
  return up256(rgk_attention_workspace_bytes(B, T)) + 2 * up256(m * D * 2) + 2 * up256(m * 512);
}

int rgk_attention_block_prefill(const void* x, const void* segment_pos, int pos_dtype,
                                const rgk_attention_params* p, const void* norm_scale, float eps, int64_t B,
                                int64_t T, int64_t D, int N, int head_dim, int window, int dtype, void* out,
                                void* keys, void* values, int* num_tokens, void* workspace,
                                size_t workspace_bytes, void* stream) {
  RGK_REQUIRE(pos_dtype == RGK_I32 || pos_dtype == RGK_I64, RGK_EINVAL, "unknown index dtype");
  RGK_REQUIRE(B >= 0 && T >= 0 && N >= 1 && window >= 1, RGK_EINVAL, "bad size");
  RGK_REQUIRE(x && segment_pos && out && p && p->q_w && p->k_w && p->v_w && p->final_w, RGK_EINVAL,
              "NULL pointer argument");
  RGK_REQUIRE((keys == nullptr) == (values == nullptr) && (keys == nullptr) == (num_tokens == nullptr),
              RGK_EINVAL, "the cache tensors go together");
  RGK_REQUIRE(aligned16(x) && aligned16(out) && aligned16(norm_scale) && aligned16(keys) && aligned16(values) &&
                  aligned16(p->q_w) && aligned16(p->k_w) && aligned16(p->v_w) && aligned16(p->final_w) &&
                  aligned16(p->final_b),
              RGK_EALIGN, "pointers must be 16-byte aligned");
  RGK_REQUIRE(rgk::attention_supported(dtype, head_dim, B > 0 ? B : 1, T > 0 ? T : 1, N) &&
                  D == (int64_t)N * head_dim,
              RGK_ESHAPE, "the attention block covers bfloat16 with head dimension 256 and as many heads as "
              "the width holds (dtype %d, head_dim %d, width %lld)", dtype, head_dim, (long long)D);
  RGK_REQUIRE(norm_scale == nullptr || rgk::rmsnorm_supported(dtype, D), RGK_ESHAPE,
              "block width %lld is not covered by the RMSNorm kernel", (long long)D);
  if (B * T == 0) return RGK_OK;
  const size_t need = rgk_attention_block_workspace_bytes(B, T, D);
  RGK_REQUIRE(workspace != nullptr && workspace_bytes >= need, RGK_EWORKSPACE,
              "workspace of %zu bytes needed, %zu given", need, workspace_bytes);
  RGK_REQUIRE((reinterpret_cast<uintptr_t>(workspace) & 255u) == 0, RGK_EALIGN,
              "workspace must be 256-byte aligned");
  RGK_CHECK_DEVICE();
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  const int64_t M = B * T;
  int* status = static_cast<int*>(workspace);
  char* q = static_cast<char*>(workspace) + up256(rgk_attention_workspace_bytes(B, T));
  char* k = q + up256((size_t)M * D * 2);
  char* v = k + up256((size_t)M * 512);
  char* xn = v + up256((size_t)M * 512);
  const void* in = x;
  if (norm_scale != nullptr) {
    RGK_CUDA(prompt_norm(x, norm_scale, M, D, eps, xn, s), "rmsnorm launch");
    in = xn;
  }
  const rgk::RowsMatrix qkv[3] = {{p->q_w, nullptr, q, (int)D}, {p->k_w, nullptr, k, head_dim},
                                  {p->v_w, nullptr, v, head_dim}};
  RGK_CUDA(prompt_linear(in, qkv, 3, nullptr, M, (int)D, 0, status, s), "proj_q, proj_k, proj_v launch");
  RGK_CUDA(rgk::launch_attention_prefill(q, k, v, segment_pos, pos_dtype == RGK_I64, B, T, N, window, true,
                                         keys, values, num_tokens, q, workspace, s),
           "attention launch");
  const rgk::RowsMatrix last = {p->final_w, p->final_b, out, (int)D};
  RGK_CUDA(prompt_linear(q, &last, 1, norm_scale != nullptr ? x : nullptr, M, (int)D, 0, status, s),
           "proj_final launch");
  return RGK_OK;
}

size_t rgk_attention_decode_workspace_bytes(int64_t B, int N, int window) {
  if (B < 0 || N < 1 || window < 1) return 0;
  return rgk::attention_decode_workspace_bytes(B < 1 ? 1 : B, N, window);
}

int rgk_local_attention_decode(const void* q, const void* k_new, const void* v_new, void* keys,
                               void* values, int* num_tokens, int64_t B, int N, int head_dim,
                               int window, int dtype, int update, void* out, void* workspace,
                               size_t workspace_bytes, void* stream) {
  RGK_REQUIRE(dtype == RGK_F32 || dtype == RGK_BF16, RGK_EINVAL, "unknown dtype %d", dtype);
  RGK_REQUIRE(B >= 0 && N >= 1 && window >= 1, RGK_EINVAL, "bad size");
  RGK_REQUIRE(q && k_new && v_new && keys && values && num_tokens && out, RGK_EINVAL,
              "NULL pointer argument");
  RGK_REQUIRE(aligned16(q) && aligned16(k_new) && aligned16(v_new) && aligned16(keys) &&
                  aligned16(values) && aligned16(out), RGK_EALIGN,
              "pointers must be 16-byte aligned");
  RGK_REQUIRE(rgk::attention_decode_supported(head_dim, N, window), RGK_ESHAPE,
              "the decode attention kernel covers head dimension 256 and 1/2/4/8/10 query heads "
              "(head_dim %d, heads %d, window %d)",
              head_dim, N, window);
  if (B == 0) return RGK_OK;
  const size_t need = rgk_attention_decode_workspace_bytes(B, N, window);
  RGK_REQUIRE(workspace != nullptr && workspace_bytes >= need, RGK_EWORKSPACE,
              "workspace of %zu bytes needed, %zu given", need, workspace_bytes);
  RGK_REQUIRE((reinterpret_cast<uintptr_t>(workspace) & 255u) == 0, RGK_EALIGN,
              "workspace must be 256-byte aligned");
  RGK_CHECK_DEVICE();
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  RGK_CUDA(dtype == RGK_BF16
               ? rgk::launch_attention_decode_ring(q, k_new, v_new, nullptr, 0, keys, values, num_tokens, keys,
                                                   values, num_tokens, B, N, window, update, out,
                                                   static_cast<int*>(workspace), s)
               : rgk::launch_attention_decode(q, k_new, v_new, keys, values, num_tokens, B, N, window, update,
                                              out, workspace, s),
           "decode attention launch");
  return RGK_OK;
}

// One decode step of the sub-path on the kernel for its batch: up to kDecodeRows rows the one whose
// CTAs serve 16 rows, above that the one with 128-row tensor-core tiles.
static constexpr int kDecodeRows = 96;
static cudaError_t path_decode_bf16(const void* xb, const void* yb, const void* pos, int pos64,
                                    const rgk_params* p, const void* packed, const float* h_in,
                                    const void* conv_in, int64_t B, int H, int gates_impl, void* out,
                                    float* h_out, void* conv_out, void* ws_header, cudaStream_t s,
                                    bool early) {
  const int math = gates_impl == RGK_GATES_FUSED_EXACT || gates_impl == RGK_GATES_TCGEN05
                       ? rgk::kMathExact : rgk::kMathFast;
  if (B <= kDecodeRows)
    return rgk::launch_path_decode_rows(xb, yb, pos, pos64, p->conv_w, p->conv_b, p->a_param, p->gate_x_b,
                                        p->gate_a_b, packed, h_in, conv_in, B, H, out, h_out, conv_out,
                                        s, math, early);
  return rgk::launch_path_decode_tc(xb, yb, pos, pos64, p->conv_w, p->conv_b, p->a_param, p->gate_x_b,
                                    p->gate_a_b, packed, h_in, conv_in, B, H, out, h_out, conv_out,
                                    ws_header, s, math);
}

int rgk_recurrent_path_decode(const void* xb, const void* yb, const void* segment_pos,
                              int pos_dtype, const rgk_params* p, const float* h_in,
                              const void* conv_cache_in, int64_t B, int64_t E, int H, int W,
                              int dtype, int gates_impl, void* out, float* h_out,
                              void* conv_cache_out, void* workspace, size_t workspace_bytes,
                              void* stream) {
  int rc = check_common(B, 1, E, dtype);
  if (rc) return rc;
  if ((rc = check_heads(E, H))) return rc;
  if ((rc = check_params(p, true))) return rc;
  RGK_REQUIRE(W == 4, RGK_ESHAPE, "temporal width %d is not supported (only 4)", W);
  RGK_REQUIRE(pos_dtype == RGK_I32 || pos_dtype == RGK_I64, RGK_EINVAL, "unknown index dtype");
  RGK_REQUIRE(gates_impl >= RGK_GATES_AUTO && gates_impl <= RGK_GATES_FUSED_EXACT, RGK_EINVAL,
              "unknown gates_impl %d", gates_impl);
  RGK_REQUIRE(xb && segment_pos && h_in && conv_cache_in && out && h_out, RGK_EINVAL,
              "NULL pointer argument");
  RGK_REQUIRE(aligned16(xb) && aligned16(yb) && aligned16(out) && aligned16(h_in) &&
                  aligned16(h_out) && aligned16(conv_cache_in) && aligned16(conv_cache_out),
              RGK_EALIGN, "pointers must be 16-byte aligned");
  if (B * E == 0) return RGK_OK;
  const PathWs w = carve(workspace, B, 1, E, dtype);
  RGK_REQUIRE(workspace != nullptr && workspace_bytes >= w.total, RGK_EWORKSPACE,
              "workspace of %zu bytes needed, %zu given", w.total, workspace_bytes);
  RGK_REQUIRE((reinterpret_cast<uintptr_t>(workspace) & 255u) == 0, RGK_EALIGN,
              "workspace must be 256-byte aligned");
  RGK_CHECK_DEVICE();
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  const int bw = (int)(E / H);
  if (gates_impl != RGK_GATES_SIMT && rgk::gates_tc_supported(dtype, bw, B)) {
    // The whole step in one kernel, and nothing else on the stream: a decode loop is one launch
    // per layer.  The states may be updated in place: every element of h and of the conv cache is read and
    // then written by one and the same thread.
    const void* packed = p->gates_packed;
    if (packed == nullptr) {
      RGK_CUDA(rgk::launch_pack_gate_weights(p->gate_x_w, p->gate_a_w, H, w.wpack, s),
               "pack_gate_weights launch");
      packed = w.wpack;
    }
    RGK_CUDA(path_decode_bf16(xb, yb, segment_pos, pos_dtype, p, packed, h_in, conv_cache_in, B, H,
                              gates_impl, out, h_out, conv_cache_out, workspace, s, false),
             "fused decode launch");
    return RGK_OK;
  }
  RGK_CUDA(rgk::launch_conv1d_decode(xb, conv_cache_in, p->conv_w, p->conv_b, B, E, dtype, w.c,
                                     conv_cache_out, s),
           "conv1d_decode launch");
  if ((rc = run_gates(w.c, segment_pos, pos_dtype, p, B, H, bw, dtype, gates_impl, w.wpack, w.a,
                      w.xn, workspace, s)))
    return rc;
  RGK_CUDA(rgk::launch_decode_update(w.a, w.xn, h_in, yb, B, E, dtype, out, h_out, s),
           "decode_update launch");
  return RGK_OK;
}

// ---- one token through a whole residual block ---------------------------------------------------------

int rgk_residual_decode_rows(void) { return 256; }

// [header | four tensors [B, E] | two [B, D] | the hidden activations [B, X]]
size_t rgk_residual_decode_workspace_bytes(int64_t B, int64_t D, int64_t E, int64_t X, int N, int window) {
  if (B < 0 || D < 1 || E < 1 || X < 1 || N < 0 || window < 0) return 0;
  if (B < 1) B = 1;
  return 256 + 4 * up256((size_t)B * E * 2) + 2 * up256((size_t)B * D * 2) + up256((size_t)B * X * 2);
}

static int check_residual_decode(const void* x, const void* segment_pos, int pos_dtype,
                                 const void* norm_scale, const rgk_channel_params* c, int64_t B,
                                 int64_t D, int64_t E, int64_t X, int N, int window, int dtype,
                                 const void* out, void* workspace, size_t workspace_bytes) {
  RGK_REQUIRE(dtype == RGK_BF16, RGK_ESHAPE, "the residual decode step is bfloat16 only (dtype %d)", dtype);
  RGK_REQUIRE(pos_dtype == RGK_I32 || pos_dtype == RGK_I64, RGK_EINVAL, "unknown index dtype");
  RGK_REQUIRE(B >= 0, RGK_EINVAL, "negative batch");
  RGK_REQUIRE(B <= rgk_residual_decode_rows(), RGK_ESHAPE, "the residual decode step covers up to %d "
              "sequences (B=%lld)", rgk_residual_decode_rows(), (long long)B);
  RGK_REQUIRE(x && segment_pos && norm_scale && out && c && c->norm_scale && c->packed_up && c->down_w,
              RGK_EINVAL, "NULL pointer argument");
  RGK_REQUIRE(aligned16(x) && aligned16(norm_scale) && aligned16(out) && aligned16(c->norm_scale) &&
                  aligned16(c->packed_up) && aligned16(c->down_w) && aligned16(c->down_b),
              RGK_EALIGN, "pointers must be 16-byte aligned");
  RGK_REQUIRE(D >= 8 && D % 8 == 0 && X >= 64 && X % 64 == 0 && D < (1 << 24) && X < (1 << 23) &&
                  rgk::rmsnorm_supported(dtype, D),
              RGK_ESHAPE, "widths the residual decode step does not cover (D=%lld, X=%lld)", (long long)D,
              (long long)X);
  const size_t need = rgk_residual_decode_workspace_bytes(B, D, E, X, N, window);
  RGK_REQUIRE(workspace != nullptr && workspace_bytes >= need, RGK_EWORKSPACE,
              "workspace of %zu bytes needed, %zu given", need, workspace_bytes);
  RGK_REQUIRE((reinterpret_cast<uintptr_t>(workspace) & 255u) == 0, RGK_EALIGN,
              "workspace must be 256-byte aligned");
  return RGK_OK;
}

// The channel half, r -> out, with `hidden` [B, X] as scratch; always behind kernels of this call.
static int channel_decode(const void* r, const rgk_channel_params* c, int64_t B, int64_t D, int64_t X,
                          void* xn, void* hidden, void* out, int* status, cudaStream_t s) {
  const char* pw = static_cast<const char*>(c->packed_up);
  const rgk::RowsMatrix up = {pw, pw + mlp_pack_w_bytes(D, X), hidden, (int)(2 * X)};
  RGK_CUDA(few_rows_norm_linear(r, c->norm_scale, c->eps, xn, &up, 1, B, (int)D, 2, status, true, s),
           "ffw_up launch");
  const rgk::RowsMatrix down = {c->down_w, c->down_b, out, (int)D};
  RGK_CUDA(few_rows_linear(hidden, &down, 1, r, B, (int)X, 0, 0.0f, status, true, false, s),
           "ffw_down launch");
  return RGK_OK;
}

int rgk_recurrent_residual_decode(const void* x, const void* segment_pos, int pos_dtype,
                                  const rgk_block_params* p, const void* norm_scale, float eps,
                                  const rgk_channel_params* channel, const float* h_in,
                                  const void* conv_cache_in, int64_t B, int64_t D, int64_t E, int64_t X,
                                  int H, int W, int dtype, int gates_impl, void* out, float* h_out,
                                  void* conv_cache_out, int chained, void* workspace,
                                  size_t workspace_bytes, void* stream) {
  int rc = check_block_args(x, segment_pos, pos_dtype, p, B, 1, D, E, H, W, dtype, out, h_out,
                            conv_cache_out);
  if (rc) return rc;
  if ((rc = check_residual_decode(x, segment_pos, pos_dtype, norm_scale, channel, B, D, E, X, 0, 0, dtype,
                                  out, workspace, workspace_bytes)))
    return rc;
  RGK_REQUIRE(gates_impl >= RGK_GATES_AUTO && gates_impl <= RGK_GATES_FUSED_EXACT &&
                  gates_impl != RGK_GATES_SIMT, RGK_EINVAL, "unknown gates_impl %d", gates_impl);
  RGK_REQUIRE(h_in && conv_cache_in && h_out && conv_cache_out && p->path.gates_packed, RGK_EINVAL,
              "NULL pointer argument");
  RGK_REQUIRE(aligned16(h_in) && aligned16(conv_cache_in), RGK_EALIGN, "pointers must be 16-byte aligned");
  if (B == 0) return RGK_OK;
  RGK_CHECK_DEVICE();
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  char* yb = static_cast<char*>(workspace) + 256;
  const size_t act = up256((size_t)B * E * 2), wide = up256((size_t)B * D * 2);
  char *xb = yb + act, *z = xb + act, *r = z + 2 * act, *xn = r + wide, *hidden = xn + wide;
  int* status = static_cast<int*>(workspace);
  const rgk::RowsMatrix in[2] = {{p->linear_y_w, p->linear_y_b, yb, (int)E},
                                 {p->linear_x_w, p->linear_x_b, xb, (int)E}};
  RGK_CUDA(few_rows_norm_linear(x, norm_scale, eps, xn, in, 2, B, (int)D, 0, status, chained != 0, s),
           "linear_y, linear_x launch");
  RGK_CUDA(path_decode_bf16(xb, yb, segment_pos, pos_dtype, &p->path, p->path.gates_packed, h_in,
                            conv_cache_in, B, H, gates_impl, z, h_out, conv_cache_out, workspace, s, true),
           "fused decode launch");
  const rgk::RowsMatrix last = {p->linear_out_w, p->linear_out_b, r, (int)D};
  RGK_CUDA(few_rows_linear(z, &last, 1, x, B, (int)E, 0, 0.0f, status, true, false, s),
           "linear_out launch");
  return channel_decode(r, channel, B, D, X, xn, hidden, out, status, s);
}

int rgk_attention_residual_decode(const void* x, const void* segment_pos, int pos_dtype,
                                  const rgk_attention_params* p, const void* norm_scale, float eps,
                                  const rgk_channel_params* channel, const void* keys_in,
                                  const void* values_in, const int* num_tokens_in, void* keys, void* values,
                                  int* num_tokens, int64_t B, int64_t D, int64_t X, int N, int head_dim,
                                  int window, int dtype, int update, void* out, int chained,
                                  void* workspace, size_t workspace_bytes, void* stream) {
  RGK_REQUIRE(N >= 1 && window >= 1, RGK_EINVAL, "bad size (heads=%d window=%d)", N, window);
  int rc = check_residual_decode(x, segment_pos, pos_dtype, norm_scale, channel, B, D, D, X, N, window,
                                 dtype, out, workspace, workspace_bytes);
  if (rc) return rc;
  RGK_REQUIRE(p && p->q_w && p->k_w && p->v_w && p->final_w && keys_in && values_in && num_tokens_in &&
                  keys && values && num_tokens, RGK_EINVAL, "NULL pointer argument");
  RGK_REQUIRE(aligned16(keys_in) && aligned16(values_in), RGK_EALIGN, "pointers must be 16-byte aligned");
  RGK_REQUIRE((keys_in == keys) == (values_in == values) && (keys_in == keys) == (num_tokens_in == num_tokens),
              RGK_EINVAL, "the cache tensors are updated in place together or not at all");
  RGK_REQUIRE(aligned16(p->q_w) && aligned16(p->k_w) && aligned16(p->v_w) && aligned16(p->final_w) &&
                  aligned16(p->final_b) && aligned16(keys) && aligned16(values),
              RGK_EALIGN, "pointers must be 16-byte aligned");
  RGK_REQUIRE(rgk::attention_decode_supported(head_dim, N, window) && D == (int64_t)N * head_dim, RGK_ESHAPE,
              "the decode attention kernel covers head dimension 256 and 1/2/4/8/10 query heads "
              "(head_dim %d, heads %d, window %d)", head_dim, N, window);
  if (B == 0) return RGK_OK;
  RGK_CHECK_DEVICE();
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  char* q = static_cast<char*>(workspace) + 256;
  const size_t wide = up256((size_t)B * D * 2);
  char *k = q + wide, *v = k + up256((size_t)B * head_dim * 2), *enc = q + 3 * wide, *r = enc + wide;
  char *xn = r + wide, *hidden = xn + wide;
  int* status = static_cast<int*>(workspace);
  const rgk::RowsMatrix in[3] = {{p->q_w, nullptr, q, (int)D}, {p->k_w, nullptr, k, head_dim},
                                 {p->v_w, nullptr, v, head_dim}};
  RGK_CUDA(few_rows_norm_linear(x, norm_scale, eps, xn, in, 3, B, (int)D, 0, status, chained != 0, s),
           "proj_q, proj_k, proj_v launch");
  RGK_CUDA(rgk::launch_attention_decode_ring(q, k, v, segment_pos, pos_dtype == RGK_I64, keys_in, values_in,
                                             num_tokens_in, keys, values, num_tokens, B, N, window, update,
                                             enc, status, s),
           "decode attention launch");
  const rgk::RowsMatrix last = {p->final_w, p->final_b, r, (int)D};
  RGK_CUDA(few_rows_linear(enc, &last, 1, x, B, (int)D, 0, 0.0f, status, true, false, s),
           "proj_final launch");
  return channel_decode(r, channel, B, D, X, xn, hidden, out, status, s);
}

}  // extern "C"
