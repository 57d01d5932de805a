// The host side of a call, natively: what the modules' forwards do between Python and the C ABI
// (argument checks, parameter and packed-weight lookup, output allocation, workspace, stream, the
// librgk call), as CPython functions on torch's C++ API.
//
// Why: a call of the decode path is one kernel of about 10 us, and the same steps written in Python
// with ctypes take 35 us (measured: 26 layers 0.90 ms a step on the host against 0.29 ms on the
// device), so that every small call was bound by its host code.  Here they take a few microseconds.
//
// Every function returns NotImplemented for arguments it does not handle - a CPU tensor, a dtype
// mismatch, a strided input, parameters of another size, and wherever a module's parameters stand for a
// call of the module, one of another class, with hooks or with a forward of its own (`plain`) - and the
// Python form of the same forward then runs, which also raises the errors.  Nothing is cached here:
// parameters are looked up in the modules on every call.
#include <ATen/ATen.h>
#include <ATen/cuda/EmptyTensor.h>
#include <c10/cuda/CUDAFunctions.h>
#include <c10/cuda/CUDAStream.h>
#include <dlfcn.h>
#include <torch/csrc/Exceptions.h>
#include <torch/csrc/autograd/python_variable.h>

#include "../../include/rgk.h"

namespace {

// ---- librgk ------------------------------------------------------------------------------------
struct Lib {
  decltype(&rgk_workspace_bytes) workspace_bytes;
  decltype(&rgk_recurrent_path_prefill) path_prefill;
  decltype(&rgk_recurrent_path_decode) path_decode;
  decltype(&rgk_rglru_forward) rglru_forward;
  decltype(&rgk_residual_decode_rows) residual_decode_rows;
  decltype(&rgk_residual_decode_workspace_bytes) residual_decode_workspace_bytes;
  decltype(&rgk_recurrent_residual_decode) recurrent_residual_decode;
  decltype(&rgk_attention_residual_decode) attention_residual_decode;
  decltype(&rgk_block_workspace_bytes) block_workspace_bytes;
  decltype(&rgk_residual_workspace_bytes) residual_workspace_bytes;
  decltype(&rgk_recurrent_block_prefill) recurrent_block_prefill;
  decltype(&rgk_residual_block_prefill) residual_block_prefill;
  decltype(&rgk_attention_block_workspace_bytes) attention_block_workspace_bytes;
  decltype(&rgk_attention_block_prefill) attention_block_prefill;
  decltype(&rgk_mlp_workspace_bytes) mlp_workspace_bytes;
  decltype(&rgk_residual_channel) residual_channel;
} g_lib;
bool g_ready = false;

// ---- Python objects of the package, handed over by init() ---------------------------------------
PyObject* g_workspaces = nullptr;        // _lib._workspaces: (device, stream) -> uint8 tensor
PyObject* g_make_workspace = nullptr;    // _lib.workspace(device, nbytes): grows it
PyObject* g_raise = nullptr;             // _lib.check(rc): raises RgkError with the library's text
PyObject* g_cache_cls = nullptr;         // modules.RecurrentBlockCache
PyObject* g_ring_cls = nullptr;          // modules.AttentionBlockCache
PyObject *g_norm_cls, *g_recurrent_cls, *g_attention_cls, *g_mlp_cls, *g_residual_cls;   // module classes
PyObject *g_conv_cls, *g_lru_cls, *g_einsum_cls, *g_linear_cls;
PyObject *g_hooks, *g_pre_hooks;         // torch's hooks for every module

// interned attribute names
#define NAMES(X) X(_parameters) X(_modules) X(w) X(b) X(a_param) X(input_gate) X(a_gate) X(num_heads) \
  X(gates_impl) X(temporal_width) X(width) X(_pack_key) X(_pack_buf) X(_packed_gates) \
  X(_packed_up) X(forward) X(_forward_hooks) X(_forward_pre_hooks) X(weight) X(bias) X(scale) X(eps) X(conv_1d) \
  X(rg_lru) X(linear_x) X(linear_y) X(linear_out) X(ffw_up) X(ffw_down) X(proj_q) X(proj_k) X(proj_v) \
  X(proj_final) X(window_size) X(expanded_width) X(lru_width) X(recurrent_block) \
  X(attention_block) X(conv1d_temporal_width) X(temporal_pre_norm) X(channel_pre_norm) X(mlp_block)
#define DECL(n) PyObject* s_##n = nullptr;
NAMES(DECL)
#undef DECL

struct Ref {                             // an owned reference
  PyObject* p;
  explicit Ref(PyObject* o) : p(o) {}
  ~Ref() { Py_XDECREF(p); }
  Ref(const Ref&) = delete;
  Ref& operator=(const Ref&) = delete;
};

PyObject* not_here() {
  PyErr_Clear();
  Py_RETURN_NOTIMPLEMENTED;
}

// A dense CUDA tensor argument; null if it is anything else (a tensor that has its operations in Python or
// no memory of its own - fake, batched, functional - among that).
const at::Tensor* dense(PyObject* o) {
  if (o == nullptr || !THPVariable_Check(o)) return nullptr;
  const at::Tensor& t = THPVariable_Unpack(o);
  const c10::TensorImpl* impl = t.unsafeGetTensorImpl();
  if (impl->is_python_dispatch() || !impl->has_storage() ||
      impl->key_set().has_any(c10::DispatchKeySet({c10::DispatchKey::Functionalize, c10::DispatchKey::ZeroTensor})))
    return nullptr;
  if (!t.is_cuda() || t.layout() != at::kStrided || !t.is_contiguous()) return nullptr;
  return &t;
}

// module.__dict__[name], borrowed (the module keeps it alive for the call); null if absent.  Modules hold
// all that is asked for here as instance attributes, and looking there is cheaper than PyObject_GetAttr.
PyObject* field(PyObject* module, PyObject* name) {
  PyObject* d = PyObject_GenericGetDict(module, nullptr);
  if (d == nullptr) return nullptr;
  PyObject* v = PyDict_GetItemWithError(d, name);
  Py_DECREF(d);
  return v;
}
// module.<dict>[name], borrowed; null if absent.
PyObject* entry(PyObject* module, PyObject* dict_name, PyObject* name) {
  PyObject* d = field(module, dict_name);
  return d != nullptr && PyDict_Check(d) ? PyDict_GetItemWithError(d, name) : nullptr;
}
PyObject* submodule(PyObject* module, PyObject* name) { return entry(module, s__modules, name); }

// A parameter of the activations' dtype and the given sizes on their device.
struct Params {
  at::ScalarType dtype;
  c10::Device device;
  bool ok = true;
  const at::Tensor* get(PyObject* module, PyObject* name, at::IntArrayRef sizes) {
    const at::Tensor* t = module == nullptr ? nullptr : dense(entry(module, s__parameters, name));
    if (t == nullptr || t->scalar_type() != dtype || t->device() != device || t->sizes() != sizes) {
      ok = false;
      return nullptr;
    }
    return t;
  }
  const void* ptr(PyObject* module, PyObject* name, at::IntArrayRef sizes) {
    const at::Tensor* t = get(module, name, sizes);
    return t == nullptr ? nullptr : t->const_data_ptr();
  }
};

// Whether calling `module` is running cls.forward on its parameters and nothing else.
bool plain(PyObject* module, PyObject* cls) {
  if (module == nullptr || (PyObject*)Py_TYPE(module) != cls || field(module, s_forward) != nullptr) return false;
  for (PyObject* name : {s__forward_hooks, s__forward_pre_hooks}) {
    PyObject* hooks = field(module, name);
    if (hooks == nullptr || !PyDict_Check(hooks) || PyDict_Size(hooks) != 0) return false;
  }
  return true;
}
bool no_global_hooks() { return PyDict_Size(g_hooks) == 0 && PyDict_Size(g_pre_hooks) == 0; }

bool int_attr(PyObject* o, PyObject* name, long* v) {
  PyObject* a = field(o, name);
  if (a == nullptr || !PyLong_Check(a)) return false;
  *v = PyLong_AsLong(a);
  return !(*v == -1 && PyErr_Occurred());
}

int dtype_code(at::ScalarType t) {
  return t == at::kFloat ? RGK_F32 : t == at::kBFloat16 ? RGK_BF16 : -1;
}
int pos_code(const at::Tensor& pos) {
  return pos.scalar_type() == at::kLong ? RGK_I64 : pos.scalar_type() == at::kInt ? RGK_I32 : -1;
}

// The tensor's device made current for the call.
struct Guard {
  c10::DeviceIndex before = -1;
  explicit Guard(c10::DeviceIndex d) {
    const c10::DeviceIndex cur = c10::cuda::current_device();
    if (cur != d) {
      before = cur;
      c10::cuda::set_device(d);
    }
  }
  ~Guard() {
    if (before >= 0) c10::cuda::set_device(before);
  }
};

at::Tensor empty(at::IntArrayRef sizes, at::ScalarType dtype, c10::Device dev) {
  return at::detail::empty_cuda(sizes, dtype, dev, c10::nullopt);
}
PyObject* wrap(at::Tensor t) { return THPVariable_Wrap(std::move(t)); }

// The scratch buffer of (device, stream), shared with the Python side, of at least `bytes` bytes.  (The Python
// side is asked for it under capture too: it keeps what a graph may hold the address of.)
struct Workspace {
  void* ptr = nullptr;
  size_t bytes = 0;
};
bool capturing(cudaStream_t stream) {
  cudaStreamCaptureStatus status = cudaStreamCaptureStatusNone;
  if (cudaStreamIsCapturing(stream, &status) != cudaSuccess) cudaGetLastError();
  return status != cudaStreamCaptureStatusNone;
}
bool workspace(const at::Tensor& on, cudaStream_t stream, size_t bytes, Workspace* ws) {
  Ref index(PyLong_FromLong(on.device().index())), address(PyLong_FromUnsignedLongLong((uintptr_t)stream));
  if (index.p == nullptr || address.p == nullptr) return false;
  Ref key(PyTuple_Pack(2, index.p, address.p));
  if (key.p == nullptr) return false;
  PyObject* buf = PyDict_GetItemWithError(g_workspaces, key.p);
  Ref made(nullptr);
  if (buf == nullptr || !THPVariable_Check(buf) || (size_t)THPVariable_Unpack(buf).numel() < bytes ||
      capturing(stream)) {
    if (PyErr_Occurred()) return false;
    Ref dev(THPDevice_New(on.device()));
    Ref n(PyLong_FromSize_t(bytes));
    made.p = PyObject_CallFunctionObjArgs(g_make_workspace, dev.p, n.p, nullptr);
    if (made.p == nullptr) return false;
    buf = made.p;
  }
  const at::Tensor& t = THPVariable_Unpack(buf);       // kept alive by the dictionary
  ws->ptr = t.mutable_data_ptr();
  ws->bytes = (size_t)t.numel();
  return true;
}

// Raises for a negative status; true if the call succeeded.
bool succeeded(int rc) {
  if (rc == 0) return true;
  Ref code(PyLong_FromLong(rc));
  Ref r(PyObject_CallFunctionObjArgs(g_raise, code.p, nullptr));
  if (r.p != nullptr) PyErr_SetString(PyExc_RuntimeError, "librgk call failed");
  return false;
}

// The packed copy a module keeps of two of its parameters (RGLRU._packed_gates, MLPBlock._packed_up),
// if its key still describes them, else whatever the module's own method makes of it.  The key is
// (address, version) of both and, for the gates, the dtype.  *made: a packing kernel was enqueued.  False: a Python error is set.
bool packed(PyObject* module, const at::Tensor& p0, const at::Tensor& p1, int dt, PyObject* method,
            const void** out, bool* made = nullptr) {
  PyObject* key = field(module, s__pack_key);
  const Py_ssize_t n = dt >= 0 ? 5 : 4;
  if (key != nullptr && PyTuple_Check(key) && PyTuple_GET_SIZE(key) == n) {
    const unsigned long long want[5] = {(unsigned long long)(uintptr_t)p0.const_data_ptr(),
                                        (unsigned long long)p0._version(),
                                        (unsigned long long)(uintptr_t)p1.const_data_ptr(),
                                        (unsigned long long)p1._version(), (unsigned long long)dt};
    bool same = true;
    for (Py_ssize_t i = 0; i < n && same; ++i)
      same = PyLong_AsUnsignedLongLong(PyTuple_GET_ITEM(key, i)) == want[i];
    if (PyErr_Occurred()) PyErr_Clear();
    if (same) {
      PyObject* buf = field(module, s__pack_buf);
      if (buf != nullptr && THPVariable_Check(buf)) {
        *out = THPVariable_Unpack(buf).const_data_ptr();
        return true;
      }
    }
  }
  if (made != nullptr) *made = true;
  Ref r(PyObject_CallMethodNoArgs(module, method));
  if (r.p == nullptr) return false;
  *out = r.p == Py_None ? nullptr : PyLong_AsVoidPtr(r.p);
  return !(PyErr_Occurred());
}

// The parameters of Conv1D (may be absent) + RGLRU.
enum class Found { yes, no, error };
Found path_params(PyObject* conv, PyObject* lru, Params& pr, int dt, long width, rgk_params* p,
                  long* heads, long* impl, bool* made = nullptr) {
  long lru_width = 0;
  if (!int_attr(lru, s_num_heads, heads) || !int_attr(lru, s_gates_impl, impl) ||
      !int_attr(lru, s_width, &lru_width) || lru_width != width || *heads < 1 || width % *heads != 0)
    return Found::no;
  const long bw = width / *heads;
  PyObject* gx = submodule(lru, s_input_gate);
  PyObject* ga = submodule(lru, s_a_gate);
  const at::Tensor* wx = pr.get(gx, s_w, {*heads, bw, bw});
  const at::Tensor* wa = pr.get(ga, s_w, {*heads, bw, bw});
  p->gate_x_b = pr.ptr(gx, s_b, {*heads, bw});
  p->gate_a_b = pr.ptr(ga, s_b, {*heads, bw});
  p->a_param = pr.ptr(lru, s_a_param, {width});
  if (conv != nullptr) {
    long tw = 0;
    p->conv_w = pr.ptr(conv, s_w, {4, width});
    p->conv_b = pr.ptr(conv, s_b, {width});
    if (!int_attr(conv, s_temporal_width, &tw) || tw != 4) return Found::no;
  }
  if (!pr.ok) return Found::no;
  p->gate_x_w = wx->const_data_ptr();
  p->gate_a_w = wa->const_data_ptr();
  p->gates_packed = nullptr;
  if (!packed(lru, *wx, *wa, dt, s__packed_gates, &p->gates_packed, made)) return Found::error;
  return Found::yes;
}

PyObject* make_cache(PyObject* h, PyObject* conv) {      // steals both
  Ref rh(h), rc(conv);
  if (h == nullptr || conv == nullptr) return nullptr;
  return PyObject_CallFunctionObjArgs(g_cache_cls, h, conv, nullptr);
}

// ---- recurrent_path(xb, yb, segment_pos, conv_1d, rg_lru, cache, return_cache, out, inplace) -----
PyObject* recurrent_path(PyObject* const* args, Py_ssize_t n) {
  if (!g_ready || n != 9) return not_here();
  const at::Tensor* x = dense(args[0]);
  const at::Tensor* y = args[1] == Py_None ? nullptr : dense(args[1]);
  const at::Tensor* pos = dense(args[2]);
  PyObject *conv = args[3], *lru = args[4], *cache = args[5];
  const bool want_cache = PyObject_IsTrue(args[6]) == 1, inplace = PyObject_IsTrue(args[8]) == 1;
  if (x == nullptr || pos == nullptr || (y == nullptr && args[1] != Py_None) || x->dim() != 3 ||
      pos->dim() != 2)
    return not_here();
  const int dt = dtype_code(x->scalar_type()), pc = pos_code(*pos);
  const int64_t B = x->size(0), T = x->size(1), E = x->size(2);
  if (dt < 0 || pc < 0 || pos->device() != x->device() || pos->size(0) != B || pos->size(1) != T ||
      B * T * E == 0)
    return not_here();
  if (y != nullptr && (y->scalar_type() != x->scalar_type() || y->device() != x->device() ||
                       y->sizes() != x->sizes()))
    return not_here();
  const at::Tensor* given = args[7] == Py_None ? nullptr : dense(args[7]);
  if (args[7] != Py_None && (given == nullptr || given->scalar_type() != x->scalar_type() ||
                             given->device() != x->device() || given->sizes() != x->sizes()))
    return not_here();
  const at::Tensor *h_in = nullptr, *c_in = nullptr;
  if (cache != Py_None) {
    if (!PyTuple_Check(cache) || PyTuple_GET_SIZE(cache) != 2 || T != 1) return not_here();
    h_in = dense(PyTuple_GET_ITEM(cache, 0));
    c_in = dense(PyTuple_GET_ITEM(cache, 1));
    if (h_in == nullptr || c_in == nullptr || h_in->scalar_type() != at::kFloat ||
        c_in->scalar_type() != x->scalar_type() || h_in->device() != x->device() ||
        c_in->device() != x->device() || h_in->dim() != 2 || h_in->size(0) != B ||
        h_in->size(1) != E || c_in->dim() != 3 || c_in->size(0) != B || c_in->size(1) != 3 ||
        c_in->size(2) != E)
      return not_here();
  }
  if (!plain(conv, g_conv_cls) || !plain(lru, g_lru_cls) || !no_global_hooks()) return not_here();
  Guard guard(x->device().index());
  Params pr{x->scalar_type(), x->device()};
  rgk_params p;
  long heads = 0, impl = 0;
  switch (path_params(conv, lru, pr, dt, E, &p, &heads, &impl)) {
    case Found::no: return not_here();
    case Found::error: return nullptr;
    case Found::yes: break;
  }
  const cudaStream_t s = c10::cuda::getCurrentCUDAStream(x->device().index()).stream();
  Workspace ws;
  if (!workspace(*x, s, g_lib.workspace_bytes(B, T, E, dt), &ws)) return nullptr;
  at::Tensor out = given != nullptr ? *given : empty(x->sizes(), x->scalar_type(), x->device());
  at::Tensor h, c;
  const void* yp = y == nullptr ? nullptr : y->const_data_ptr();
  if (cache == Py_None) {
    if (want_cache) {
      h = empty({B, E}, at::kFloat, x->device());
      c = empty({B, 3, E}, x->scalar_type(), x->device());
    }
    if (!succeeded(g_lib.path_prefill(
            x->const_data_ptr(), yp, pos->const_data_ptr(), pc, &p, nullptr, B, T, E, (int)heads, 4, dt,
            (int)impl, out.mutable_data_ptr(),
            want_cache ? static_cast<float*>(h.mutable_data_ptr()) : nullptr,
            want_cache ? c.mutable_data_ptr() : nullptr, ws.ptr, ws.bytes, s)))
      return nullptr;
  } else {
    h = inplace ? *h_in : empty({B, E}, at::kFloat, x->device());
    c = inplace ? *c_in : empty({B, 3, E}, x->scalar_type(), x->device());
    if (!succeeded(g_lib.path_decode(
            x->const_data_ptr(), yp, pos->const_data_ptr(), pc, &p,
            static_cast<const float*>(h_in->const_data_ptr()), c_in->const_data_ptr(), B, E, (int)heads,
            4, dt, (int)impl, out.mutable_data_ptr(), static_cast<float*>(h.mutable_data_ptr()),
            c.mutable_data_ptr(), ws.ptr, ws.bytes, s)))
      return nullptr;
  }
  Ref o(given != nullptr ? Py_NewRef(args[7]) : wrap(std::move(out)));
  if (!want_cache) return PyTuple_Pack(2, o.p, Py_None);
  Ref made(inplace && cache != Py_None
               ? make_cache(Py_NewRef(PyTuple_GET_ITEM(cache, 0)), Py_NewRef(PyTuple_GET_ITEM(cache, 1)))
               : make_cache(wrap(std::move(h)), wrap(std::move(c))));
  if (o.p == nullptr || made.p == nullptr) return nullptr;
  return PyTuple_Pack(2, o.p, made.p);
}

// ---- RGLRU.forward: rglru(module, x, segment_pos, cache, return_cache) ---------------------------
PyObject* rglru(PyObject* const* args, Py_ssize_t n) {
  if (!g_ready || n != 5) return not_here();
  PyObject* lru = args[0];
  const at::Tensor *x = dense(args[1]), *pos = dense(args[2]);
  const at::Tensor* h_in = args[3] == Py_None ? nullptr : dense(args[3]);
  const bool want = PyObject_IsTrue(args[4]) == 1;
  if (x == nullptr || pos == nullptr || (h_in == nullptr && args[3] != Py_None) || x->dim() != 3 ||
      pos->dim() != 2)
    return not_here();
  const int dt = dtype_code(x->scalar_type()), pc = pos_code(*pos);
  const int64_t B = x->size(0), T = x->size(1), E = x->size(2);
  if (dt < 0 || pc < 0 || pos->device() != x->device() || pos->size(0) != B || pos->size(1) != T ||
      B * T * E == 0)
    return not_here();
  if (h_in != nullptr && (h_in->scalar_type() != at::kFloat || h_in->device() != x->device() ||
                          h_in->dim() != 2 || h_in->size(0) != B || h_in->size(1) != E))
    return not_here();
  Guard guard(x->device().index());
  Params pr{x->scalar_type(), x->device()};
  rgk_params p = {};
  long heads = 0, impl = 0;
  switch (path_params(nullptr, lru, pr, dt, E, &p, &heads, &impl)) {
    case Found::no: return not_here();
    case Found::error: return nullptr;
    case Found::yes: break;
  }
  const cudaStream_t s = c10::cuda::getCurrentCUDAStream(x->device().index()).stream();
  Workspace ws;
  if (!workspace(*x, s, g_lib.workspace_bytes(B, T, E, dt), &ws)) return nullptr;
  at::Tensor y = empty(x->sizes(), x->scalar_type(), x->device()), h;
  if (want) h = empty({B, E}, at::kFloat, x->device());
  if (!succeeded(g_lib.rglru_forward(
          x->const_data_ptr(), pos->const_data_ptr(), pc, &p,
          h_in == nullptr ? nullptr : static_cast<const float*>(h_in->const_data_ptr()), B, T, E,
          (int)heads, dt, (int)impl, y.mutable_data_ptr(),
          want ? static_cast<float*>(h.mutable_data_ptr()) : nullptr, ws.ptr, ws.bytes, s)))
    return nullptr;
  Ref ry(wrap(std::move(y))), rh(want ? wrap(std::move(h)) : Py_NewRef(Py_None));
  if (ry.p == nullptr || rh.p == nullptr) return nullptr;
  return PyTuple_Pack(2, ry.p, rh.p);
}

// ---- the decode step of a residual block ------------------------------------------------------------
// The decode step of a few sequences through a whole residual block, one library call.

bool exactly(PyObject* module, PyObject* cls) { return (PyObject*)Py_TYPE(module) == cls; }
bool float_attr(PyObject* o, PyObject* name, float* v) {
  PyObject* a = field(o, name);
  if (a == nullptr) return false;
  *v = (float)PyFloat_AsDouble(a);
  return !PyErr_Occurred();
}
// An activation-sized tensor of one token per sequence: [B, 1, width] or the ring's tensors.
bool shaped(const at::Tensor* t, at::ScalarType dtype, c10::Device dev, at::IntArrayRef sizes) {
  return t != nullptr && t->scalar_type() == dtype && t->device() == dev && t->sizes() == sizes;
}

// The parameters of a RecurrentBlock of width D and RG-LRU width E.
Found recurrent_params(PyObject* block, Params& pr, long D, long E, rgk_block_params* p, long* heads, long* impl,
                       bool* made) {
  PyObject *ly = submodule(block, s_linear_y), *lx = submodule(block, s_linear_x),
           *lo = submodule(block, s_linear_out);
  PyObject *conv = submodule(block, s_conv_1d), *lru = submodule(block, s_rg_lru);
  if (!plain(ly, g_linear_cls) || !plain(lx, g_linear_cls) || !plain(lo, g_linear_cls) ||
      !plain(conv, g_conv_cls) || !plain(lru, g_lru_cls))
    return Found::no;
  p->linear_y_w = pr.ptr(ly, s_weight, {E, D}); p->linear_y_b = pr.ptr(ly, s_bias, {E});
  p->linear_x_w = pr.ptr(lx, s_weight, {E, D}); p->linear_x_b = pr.ptr(lx, s_bias, {E});
  p->linear_out_w = pr.ptr(lo, s_weight, {D, E}); p->linear_out_b = pr.ptr(lo, s_bias, {D});
  if (!pr.ok) return Found::no;
  return path_params(conv, lru, pr, RGK_BF16, E, &p->path, heads, impl, made);
}
// The parameters of a LocalAttentionBlock of width D and one key/value head of 256; pr.ok says whether they
// are all there.
rgk_attention_params attention_params(PyObject* block, Params& pr, long D) {
  rgk_attention_params p = {};
  PyObject *q = submodule(block, s_proj_q), *k = submodule(block, s_proj_k), *v = submodule(block, s_proj_v),
           *f = submodule(block, s_proj_final);
  for (PyObject* m : {q, k, v, f}) pr.ok = pr.ok && plain(m, g_linear_cls);
  if (!pr.ok) return p;
  p.q_w = pr.ptr(q, s_weight, {D, D});
  p.k_w = pr.ptr(k, s_weight, {256, D});
  p.v_w = pr.ptr(v, s_weight, {256, D});
  p.final_w = pr.ptr(f, s_weight, {D, D});
  p.final_b = pr.ptr(f, s_bias, {D});
  return p;
}

// The channel half of a residual block of width D: its norm and its MLP.
struct Channel {
  long X = 0;
  float eps = 0.0f;
  const void *scale = nullptr, *down_w = nullptr, *down_b = nullptr;
  const at::Tensor *up_w = nullptr, *up_b = nullptr;       // ffw_up, which the kernels read packed
};
bool channel_params(PyObject* norm, PyObject* mlp, Params& pr, long D, Channel* c) {
  long w = 0, wn = 0;
  if (!plain(norm, g_norm_cls) || !plain(mlp, g_mlp_cls) || !int_attr(mlp, s_expanded_width, &c->X) ||
      !int_attr(mlp, s_width, &w) || !int_attr(norm, s_width, &wn) || w != D || wn != D || c->X % 64 != 0 ||
      D % 8 != 0 || !float_attr(norm, s_eps, &c->eps))
    return false;
  PyObject *up = submodule(mlp, s_ffw_up), *down = submodule(mlp, s_ffw_down);
  if (!plain(up, g_einsum_cls) || !plain(down, g_linear_cls)) return false;
  c->up_w = pr.get(up, s_w, {2, D, c->X});
  c->up_b = pr.get(up, s_b, {2, 1, 1, c->X});
  c->scale = pr.ptr(norm, s_scale, {D});
  c->down_w = pr.ptr(down, s_weight, {D, c->X});
  c->down_b = pr.ptr(down, s_bias, {D});
  return pr.ok;
}

PyObject* step(PyObject* x_arg, PyObject* pos_arg, PyObject* norm1, PyObject* block, PyObject* norm2,
               PyObject* mlp, PyObject* cache, bool want, bool inplace, bool chained) {
  const at::Tensor *x = dense(x_arg), *pos = dense(pos_arg);
  const bool recurrent = exactly(block, g_recurrent_cls);
  if (x == nullptr || pos == nullptr || !PyTuple_Check(cache) || x->scalar_type() != at::kBFloat16 ||
      x->dim() != 3 || x->size(1) != 1 || pos->dim() != 2 || pos_code(*pos) < 0 ||
      pos->device() != x->device() || pos->size(0) != x->size(0) || pos->size(1) != 1)
    return not_here();
  const int64_t B = x->size(0), D = x->size(2);
  const c10::Device dev = x->device();
  if (B == 0 || B > g_lib.residual_decode_rows() || D == 0) return not_here();
  if (!plain(block, recurrent ? g_recurrent_cls : g_attention_cls) || !plain(norm1, g_norm_cls) ||
      !no_global_hooks())
    return not_here();
  Guard guard(dev.index());
  Params pr{at::kBFloat16, dev};
  Channel ch;
  long w1 = 0;
  float eps1 = 0.0f;
  if (!channel_params(norm2, mlp, pr, D, &ch) || !int_attr(norm1, s_width, &w1) || w1 != D ||
      !float_attr(norm1, s_eps, &eps1))
    return not_here();
  const long X = ch.X;
  rgk_channel_params c = {};
  c.norm_scale = ch.scale;
  c.down_w = ch.down_w;
  c.down_b = ch.down_b;
  c.eps = ch.eps;
  const void* scale1 = pr.ptr(norm1, s_scale, {D});
  if (!pr.ok) return not_here();
  const cudaStream_t s = c10::cuda::getCurrentCUDAStream(dev.index()).stream();
  const int pc = pos_code(*pos);
  Workspace ws;
  bool made = false;                               // a packing kernel was enqueued by this call
  if (recurrent) {
    if (PyTuple_GET_SIZE(cache) != 2) return not_here();
    const at::Tensor *h_in = dense(PyTuple_GET_ITEM(cache, 0)), *c_in = dense(PyTuple_GET_ITEM(cache, 1));
    long E = 0, heads = 0, impl = 0, width = 0;
    if (!int_attr(block, s_lru_width, &E) || !int_attr(block, s_width, &width) || width != D ||
        !shaped(h_in, at::kFloat, dev, {B, E}) || !shaped(c_in, at::kBFloat16, dev, {B, 3, E}))
      return not_here();
    rgk_block_params p = {};
    switch (recurrent_params(block, pr, D, E, &p, &heads, &impl, &made)) {
      case Found::no: return not_here();
      case Found::error: return nullptr;
      case Found::yes: break;
    }
    if (E != heads * 256 || impl == RGK_GATES_SIMT || p.path.gates_packed == nullptr) return not_here();
    if (!packed(mlp, *ch.up_w, *ch.up_b, -1, s__packed_up, &c.packed_up, &made)) return nullptr;
    if (!workspace(*x, s, g_lib.residual_decode_workspace_bytes(B, D, E, X, 0, 0), &ws)) return nullptr;
    at::Tensor out = empty(x->sizes(), at::kBFloat16, dev);
    at::Tensor h = inplace ? *h_in : empty({B, E}, at::kFloat, dev);
    at::Tensor cc = inplace ? *c_in : empty({B, 3, E}, at::kBFloat16, dev);
    if (!succeeded(g_lib.recurrent_residual_decode(
            x->const_data_ptr(), pos->const_data_ptr(), pc, &p, scale1, eps1, &c,
            static_cast<const float*>(h_in->const_data_ptr()), c_in->const_data_ptr(), B, D, E, X,
            (int)heads, 4, RGK_BF16, (int)impl, out.mutable_data_ptr(),
            static_cast<float*>(h.mutable_data_ptr()), cc.mutable_data_ptr(), chained && !made ? 1 : 0,
            ws.ptr, ws.bytes, s)))
      return nullptr;
    Ref o(wrap(std::move(out)));
    if (!want) return PyTuple_Pack(2, o.p, Py_None);
    Ref state(inplace ? make_cache(Py_NewRef(PyTuple_GET_ITEM(cache, 0)), Py_NewRef(PyTuple_GET_ITEM(cache, 1)))
                      : make_cache(wrap(std::move(h)), wrap(std::move(cc))));
    if (o.p == nullptr || state.p == nullptr) return nullptr;
    return PyTuple_Pack(2, o.p, state.p);
  }
  if (PyTuple_GET_SIZE(cache) != 3) return not_here();
  const at::Tensor *keys = dense(PyTuple_GET_ITEM(cache, 0)), *values = dense(PyTuple_GET_ITEM(cache, 1)),
                   *seen = dense(PyTuple_GET_ITEM(cache, 2));
  long heads = 0, window = 0, width = 0;
  if (!int_attr(block, s_num_heads, &heads) || !int_attr(block, s_window_size, &window) ||
      !int_attr(block, s_width, &width) || width != D || heads * 256 != D ||
      !(heads == 1 || heads == 2 || heads == 4 || heads == 8 || heads == 10) ||
      !shaped(keys, at::kBFloat16, dev, {B, window, 1, 256}) ||
      !shaped(values, at::kBFloat16, dev, {B, window, 1, 256}) || !shaped(seen, at::kInt, dev, {B}))
    return not_here();
  const rgk_attention_params p = attention_params(block, pr, D);
  if (!pr.ok) return not_here();
  if (!packed(mlp, *ch.up_w, *ch.up_b, -1, s__packed_up, &c.packed_up, &made)) return nullptr;
  if (!workspace(*x, s, g_lib.residual_decode_workspace_bytes(B, D, D, X, (int)heads, (int)window), &ws))
    return nullptr;
  at::Tensor out = empty(x->sizes(), at::kBFloat16, dev);
  const bool fresh = want && !inplace;             // a new ring, written as the old one is read
  at::Tensor k = fresh ? empty(keys->sizes(), at::kBFloat16, dev) : *keys,
             v = fresh ? empty(values->sizes(), at::kBFloat16, dev) : *values,
             seen_out = fresh ? empty(seen->sizes(), at::kInt, dev) : *seen;
  if (!succeeded(g_lib.attention_residual_decode(
          x->const_data_ptr(), pos->const_data_ptr(), pc, &p, scale1, eps1, &c, keys->const_data_ptr(),
          values->const_data_ptr(), static_cast<const int*>(seen->const_data_ptr()), k.mutable_data_ptr(),
          v.mutable_data_ptr(), static_cast<int*>(seen_out.mutable_data_ptr()), B, D, X, (int)heads, 256,
          (int)window, RGK_BF16, want ? 1 : 0, out.mutable_data_ptr(), chained && !made ? 1 : 0, ws.ptr,
          ws.bytes, s)))
    return nullptr;
  Ref o(wrap(std::move(out)));
  if (o.p == nullptr) return nullptr;
  if (!want) return PyTuple_Pack(2, o.p, Py_None);
  if (!fresh) return PyTuple_Pack(2, o.p, cache);
  Ref rk(wrap(std::move(k))), rv(wrap(std::move(v))), rs(wrap(std::move(seen_out)));
  if (rk.p == nullptr || rv.p == nullptr || rs.p == nullptr) return nullptr;
  Ref ring(PyObject_CallFunctionObjArgs(g_ring_cls, rk.p, rv.p, rs.p, nullptr));
  if (ring.p == nullptr) return nullptr;
  return PyTuple_Pack(2, o.p, ring.p);
}

// ---- prefill of a temporal block, alone or inside its residual block -------------------------------

// x, segment_pos -> [norm ->] temporal block [-> + x], with the cache of the prompt.  Yes: *out and, if
// wanted, *cache are set.
Found temporal_prefill(const at::Tensor& x, const at::Tensor& pos, PyObject* norm, PyObject* block, bool want,
                       at::Tensor* out, PyObject** cache) {
  const bool recurrent = exactly(block, g_recurrent_cls);
  if (!(recurrent || exactly(block, g_attention_cls)) || !no_global_hooks()) return Found::no;
  const int64_t B = x.size(0), T = x.size(1), D = x.size(2);
  const c10::Device dev = x.device();
  Params pr{at::kBFloat16, dev};
  const void* scale = nullptr;
  float eps = 0.0f;
  long w1 = 0, width = 0;
  if (norm != nullptr) {
    if (!plain(norm, g_norm_cls) || !plain(block, recurrent ? g_recurrent_cls : g_attention_cls)) return Found::no;
    scale = pr.ptr(norm, s_scale, {D});
    if (!pr.ok || !int_attr(norm, s_width, &w1) || w1 != D || !float_attr(norm, s_eps, &eps)) return Found::no;
  }
  if (!int_attr(block, s_width, &width) || width != D || D % 8 != 0) return Found::no;
  const cudaStream_t s = c10::cuda::getCurrentCUDAStream(dev.index()).stream();
  const int pc = pos_code(pos);
  Workspace ws;
  if (recurrent) {
    long E = 0, heads = 0, impl = 0, tw = 0;
    rgk_block_params p = {};
    if (!int_attr(block, s_lru_width, &E) || !int_attr(block, s_conv1d_temporal_width, &tw) || tw != 4)
      return Found::no;
    const Found f = recurrent_params(block, pr, D, E, &p, &heads, &impl, nullptr);
    if (f != Found::yes) return f;
    if (E != heads * 256 || impl == RGK_GATES_SIMT) return Found::no;
    if (!workspace(x, s, norm != nullptr ? g_lib.residual_workspace_bytes(B, T, D, E, RGK_BF16)
                                         : g_lib.block_workspace_bytes(B, T, D, E, RGK_BF16), &ws))
      return Found::error;
    *out = empty(x.sizes(), at::kBFloat16, dev);
    at::Tensor h, c;
    if (want) {
      h = empty({B, E}, at::kFloat, dev);
      c = empty({B, 3, E}, at::kBFloat16, dev);
    }
    float* hp = want ? static_cast<float*>(h.mutable_data_ptr()) : nullptr;
    void* cp = want ? c.mutable_data_ptr() : nullptr;
    const int rc = norm != nullptr
        ? g_lib.residual_block_prefill(x.const_data_ptr(), pos.const_data_ptr(), pc, &p, scale, eps, B, T, D, E,
                                       (int)heads, 4, RGK_BF16, out->mutable_data_ptr(), hp, cp, ws.ptr,
                                       ws.bytes, s)
        : g_lib.recurrent_block_prefill(x.const_data_ptr(), pos.const_data_ptr(), pc, &p, B, T, D, E,
                                        (int)heads, 4, RGK_BF16, out->mutable_data_ptr(), hp, cp, ws.ptr,
                                        ws.bytes, s);
    if (!succeeded(rc)) return Found::error;
    if (want) *cache = make_cache(wrap(std::move(h)), wrap(std::move(c)));
  } else {
    long heads = 0, window = 0;
    const rgk_attention_params p = attention_params(block, pr, D);
    if (!pr.ok || !int_attr(block, s_num_heads, &heads) || !int_attr(block, s_window_size, &window) ||
        heads * 256 != D || window < 1)
      return Found::no;
    if (!workspace(x, s, g_lib.attention_block_workspace_bytes(B, T, D), &ws)) return Found::error;
    *out = empty(x.sizes(), at::kBFloat16, dev);
    at::Tensor k, v, seen;
    if (want) {
      k = empty({B, window, 1, 256}, at::kBFloat16, dev);
      v = empty({B, window, 1, 256}, at::kBFloat16, dev);
      seen = empty({B}, at::kInt, dev);
    }
    if (!succeeded(g_lib.attention_block_prefill(
            x.const_data_ptr(), pos.const_data_ptr(), pc, &p, scale, eps, B, T, D, (int)heads, 256, (int)window,
            RGK_BF16, out->mutable_data_ptr(), want ? k.mutable_data_ptr() : nullptr,
            want ? v.mutable_data_ptr() : nullptr,
            want ? static_cast<int*>(seen.mutable_data_ptr()) : nullptr, ws.ptr, ws.bytes, s)))
      return Found::error;
    if (want) {
      Ref rk(wrap(std::move(k))), rv(wrap(std::move(v))), rs(wrap(std::move(seen)));
      if (rk.p == nullptr || rv.p == nullptr || rs.p == nullptr) return Found::error;
      *cache = PyObject_CallFunctionObjArgs(g_ring_cls, rk.p, rv.p, rs.p, nullptr);
    }
  }
  return want && *cache == nullptr ? Found::error : Found::yes;
}

// The arguments of a prefill call: dense bfloat16 [B, T, D] and positions [B, T] on the same device.
bool prompt_args(const at::Tensor* x, const at::Tensor* pos) {
  return x != nullptr && pos != nullptr && x->scalar_type() == at::kBFloat16 && x->dim() == 3 &&
         pos->dim() == 2 && pos_code(*pos) >= 0 && pos->device() == x->device() &&
         pos->size(0) == x->size(0) && pos->size(1) == x->size(1) && x->numel() > 0;
}

// prefill(temporal block, x, segment_pos, return_cache): its forward without a cache
PyObject* prefill(PyObject* const* args, Py_ssize_t n) {
  if (!g_ready || n != 4) return not_here();
  const at::Tensor *x = dense(args[1]), *pos = dense(args[2]);
  if (!prompt_args(x, pos)) return not_here();
  Guard guard(x->device().index());
  at::Tensor out;
  PyObject* cache = nullptr;
  switch (temporal_prefill(*x, *pos, nullptr, args[0], PyObject_IsTrue(args[3]) == 1, &out, &cache)) {
    case Found::no: return not_here();
    case Found::error: return nullptr;
    case Found::yes: break;
  }
  Ref o(wrap(std::move(out))), c(cache != nullptr ? cache : Py_NewRef(Py_None));
  return o.p == nullptr ? nullptr : PyTuple_Pack(2, o.p, c.p);
}

// residual_prefill(x, segment_pos, norm, temporal block, norm, mlp, return_cache)
PyObject* residual_prefill(PyObject* const* args, Py_ssize_t n) {
  if (!g_ready || n != 7) return not_here();
  const at::Tensor *x = dense(args[0]), *pos = dense(args[1]);
  PyObject *norm2 = args[4], *mlp = args[5];
  if (!prompt_args(x, pos)) return not_here();
  const int64_t M = x->size(0) * x->size(1), D = x->size(2);
  const c10::Device dev = x->device();
  Guard guard(dev.index());
  Params pr{at::kBFloat16, dev};
  Channel ch;
  if (!channel_params(norm2, mlp, pr, D, &ch)) return not_here();
  const long X = ch.X;
  const void* packed_up = nullptr;
  if (!packed(mlp, *ch.up_w, *ch.up_b, -1, s__packed_up, &packed_up)) return nullptr;
  at::Tensor r;
  PyObject* cache = nullptr;
  switch (temporal_prefill(*x, *pos, args[2], args[3], PyObject_IsTrue(args[6]) == 1, &r, &cache)) {
    case Found::no: return not_here();
    case Found::error: return nullptr;
    case Found::yes: break;
  }
  Ref c(cache != nullptr ? cache : Py_NewRef(Py_None));
  const cudaStream_t s = c10::cuda::getCurrentCUDAStream(dev.index()).stream();
  Workspace ws;
  if (!workspace(*x, s, g_lib.mlp_workspace_bytes(M, D, X, RGK_BF16), &ws)) return nullptr;
  at::Tensor out = empty(x->sizes(), at::kBFloat16, dev);
  if (!succeeded(g_lib.residual_channel(r.const_data_ptr(), ch.scale, ch.eps, packed_up, ch.down_w, ch.down_b, M, D, X,
                                        RGK_BF16, out.mutable_data_ptr(), ws.ptr, ws.bytes, s)))
    return nullptr;
  Ref o(wrap(std::move(out)));
  return o.p == nullptr ? nullptr : PyTuple_Pack(2, o.p, c.p);
}

// residual_step(x, segment_pos, norm, temporal block, norm, mlp, cache, return_cache, inplace)
PyObject* residual_step(PyObject* const* args, Py_ssize_t n) {
  if (!g_ready || n != 9) return not_here();
  return step(args[0], args[1], args[2], args[3], args[4], args[5], args[6], PyObject_IsTrue(args[7]) == 1,
              PyObject_IsTrue(args[8]) == 1, false);
}

// block_step(ResidualBlock, x, segment_pos, cache, return_cache, inplace, chained): the same for a
// module; chained: the last work on the stream is another block's step (see rgk.h).
PyObject* block_step(PyObject* const* args, Py_ssize_t n) {
  if (!g_ready || n != 7) return not_here();
  PyObject* m = args[0];
  if (!plain(m, g_residual_cls)) return not_here();
  PyObject* temporal = submodule(m, s_recurrent_block);
  if (temporal == nullptr) temporal = submodule(m, s_attention_block);
  PyObject *norm1 = submodule(m, s_temporal_pre_norm), *norm2 = submodule(m, s_channel_pre_norm),
           *mlp = submodule(m, s_mlp_block);
  if (temporal == nullptr || norm1 == nullptr || norm2 == nullptr || mlp == nullptr) return not_here();
  return step(args[1], args[2], norm1, temporal, norm2, mlp, args[3], PyObject_IsTrue(args[4]) == 1,
              PyObject_IsTrue(args[5]) == 1, PyObject_IsTrue(args[6]) == 1);
}

// as_built(module, class): `plain`, for the Python forms, which also take a subclass that keeps the forward.
PyObject* as_built(PyObject* const* args, Py_ssize_t n) {
  if (n != 2) {
    PyErr_SetString(PyExc_TypeError, "as_built(module, class)");
    return nullptr;
  }
  if (g_hooks == nullptr || !no_global_hooks()) Py_RETURN_FALSE;
  PyObject *module = args[0], *cls = args[1], *type = (PyObject*)Py_TYPE(module);
  if (type != cls) {
    Ref own(PyObject_GetAttr(type, s_forward)), theirs(PyObject_GetAttr(cls, s_forward));
    if (own.p == nullptr || theirs.p == nullptr) PyErr_Clear();
    if (own.p != theirs.p || own.p == nullptr) Py_RETURN_FALSE;
  }
  return PyBool_FromLong(plain(module, type));
}

// ---- set-up --------------------------------------------------------------------------------------
// init(librgk path, _workspaces, workspace, check, (RecurrentBlockCache, AttentionBlockCache, RMSNorm,
// RecurrentBlock, LocalAttentionBlock, MLPBlock, ResidualBlock, Conv1D, RGLRU, Einsum, nn.Linear), torch's
// global forward hooks and pre-hooks)
PyObject* init(PyObject*, PyObject* args) {
  const char* path = nullptr;
  PyObject *spaces, *make, *raise, *cls[11], *hooks, *pre_hooks;
  if (!PyArg_ParseTuple(args, "sO!OO(OOOOOOOOOOO)O!O!", &path, &PyDict_Type, &spaces, &make, &raise, &cls[0],
                        &cls[1], &cls[2], &cls[3], &cls[4], &cls[5], &cls[6], &cls[7], &cls[8], &cls[9], &cls[10],
                        &PyDict_Type, &hooks, &PyDict_Type, &pre_hooks))
    return nullptr;
  void* so = dlopen(path, RTLD_NOW | RTLD_LOCAL);        // already loaded by ctypes: the same handle
  if (so == nullptr) {
    PyErr_Format(PyExc_RuntimeError, "dlopen(%s): %s", path, dlerror());
    return nullptr;
  }
  auto find = [&](auto* fn, const char* name) {
    *fn = reinterpret_cast<std::remove_reference_t<decltype(*fn)>>(dlsym(so, name));
    if (*fn == nullptr && !PyErr_Occurred())
      PyErr_Format(PyExc_RuntimeError, "%s does not export %s", path, name);
  };
  find(&g_lib.workspace_bytes, "rgk_workspace_bytes");
  find(&g_lib.path_prefill, "rgk_recurrent_path_prefill");
  find(&g_lib.path_decode, "rgk_recurrent_path_decode");
  find(&g_lib.rglru_forward, "rgk_rglru_forward");
  find(&g_lib.residual_decode_rows, "rgk_residual_decode_rows");
  find(&g_lib.residual_decode_workspace_bytes, "rgk_residual_decode_workspace_bytes");
  find(&g_lib.recurrent_residual_decode, "rgk_recurrent_residual_decode");
  find(&g_lib.attention_residual_decode, "rgk_attention_residual_decode");
  find(&g_lib.block_workspace_bytes, "rgk_block_workspace_bytes");
  find(&g_lib.residual_workspace_bytes, "rgk_residual_workspace_bytes");
  find(&g_lib.recurrent_block_prefill, "rgk_recurrent_block_prefill");
  find(&g_lib.residual_block_prefill, "rgk_residual_block_prefill");
  find(&g_lib.attention_block_workspace_bytes, "rgk_attention_block_workspace_bytes");
  find(&g_lib.attention_block_prefill, "rgk_attention_block_prefill");
  find(&g_lib.mlp_workspace_bytes, "rgk_mlp_workspace_bytes");
  find(&g_lib.residual_channel, "rgk_residual_channel");
  if (PyErr_Occurred()) return nullptr;
#define INTERN(n) if (s_##n == nullptr) s_##n = PyUnicode_InternFromString(#n);
  NAMES(INTERN)
#undef INTERN
  g_workspaces = Py_NewRef(spaces);
  g_make_workspace = Py_NewRef(make);
  g_raise = Py_NewRef(raise);
  PyObject** to[11] = {&g_cache_cls, &g_ring_cls, &g_norm_cls, &g_recurrent_cls, &g_attention_cls, &g_mlp_cls,
                       &g_residual_cls, &g_conv_cls, &g_lru_cls, &g_einsum_cls, &g_linear_cls};
  for (int i = 0; i < 11; ++i) *to[i] = Py_NewRef(cls[i]);
  g_hooks = Py_NewRef(hooks);
  g_pre_hooks = Py_NewRef(pre_hooks);
  g_ready = true;
  Py_RETURN_NONE;
}

// What CPython calls: torch's C++ exceptions (out of memory, no CUDA driver, the version of an inference
// tensor) leave as the Python errors they are.
template <PyObject* (*fn)(PyObject* const*, Py_ssize_t)>
PyObject* entry_point(PyObject*, PyObject* const* args, Py_ssize_t n) {
  try {
    return fn(args, n);
  } catch (...) {
    torch::translate_exception_to_python(std::current_exception());
    return nullptr;
  }
}
#define FAST(fn) \
  {#fn, reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(entry_point<fn>)), METH_FASTCALL, nullptr}
PyMethodDef methods[] = {
    {"init", init, METH_VARARGS, nullptr},
    FAST(recurrent_path),
    FAST(rglru),
    FAST(residual_step),
    FAST(block_step),
    FAST(prefill),
    FAST(residual_prefill),
    FAST(as_built),
    {nullptr, nullptr, 0, nullptr}};
PyModuleDef module_def = {PyModuleDef_HEAD_INIT, "_host", nullptr, -1, methods, nullptr, nullptr, nullptr,
                          nullptr};

}  // namespace

PyMODINIT_FUNC PyInit__host() { return PyModule_Create(&module_def); }
