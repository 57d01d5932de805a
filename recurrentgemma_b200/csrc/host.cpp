// The host side of a call, natively: what the modules' forwards do between Python and the C ABI
// (argument checks, parameter and packed-weight lookup, output allocation, workspace, stream, the
// librgk call), as CPython functions on torch's C++ API.
//
// Why: a call of the decode path is one kernel of about 10 us, and the same steps written in Python
// with ctypes take 35 us (measured: 26 layers 0.90 ms a step on the host against 0.29 ms on the
// device), so that every small call was bound by its host code.  Here they take a few microseconds.
//
// Every function returns NotImplemented for arguments it does not handle - a CPU tensor, a dtype
// mismatch, a strided input, a subclass or a module with hooks where modules are fused - and the
// Python form of the same forward then runs, which also raises the errors.  Nothing is cached here:
// parameters are looked up in the modules on every call.
#include <ATen/ATen.h>
#include <ATen/cuda/EmptyTensor.h>
#include <c10/cuda/CUDAFunctions.h>
#include <c10/cuda/CUDAStream.h>
#include <dlfcn.h>
#include <torch/csrc/autograd/python_variable.h>

#include "../../include/rgk.h"

namespace {

// ---- librgk ------------------------------------------------------------------------------------
struct Lib {
  decltype(&rgk_workspace_bytes) workspace_bytes;
  decltype(&rgk_recurrent_path_prefill) path_prefill;
  decltype(&rgk_recurrent_path_decode) path_decode;
  decltype(&rgk_rglru_forward) rglru_forward;
  decltype(&rgk_conv1d_prefill) conv1d_prefill;
  decltype(&rgk_conv1d_decode) conv1d_decode;
} g_lib;
bool g_ready = false;

// ---- Python objects of the package, handed over by init() ---------------------------------------
PyObject* g_workspaces = nullptr;        // _lib._workspaces: (device, stream) -> uint8 tensor
PyObject* g_make_workspace = nullptr;    // _lib.workspace(device, nbytes): grows it
PyObject* g_raise = nullptr;             // _lib.check(rc): raises RgkError with the library's text
PyObject* g_cache_cls = nullptr;         // modules.RecurrentBlockCache

// interned attribute names
#define NAMES(X) X(_parameters) X(_modules) X(w) X(b) X(a_param) X(input_gate) X(a_gate) X(num_heads) \
  X(gates_impl) X(temporal_width) X(width) X(_pack_key) X(_pack_buf) X(_packed_gates)
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

// A dense CUDA tensor argument; null if it is anything else.
const at::Tensor* dense(PyObject* o) {
  if (o == nullptr || !THPVariable_Check(o)) return nullptr;
  const at::Tensor& t = THPVariable_Unpack(o);
  if (!t.is_cuda() || t.layout() != at::kStrided || !t.is_contiguous()) return nullptr;
  return &t;
}

// module.<dict>[name], borrowed (the module keeps it alive for the call); null if absent.
PyObject* entry(PyObject* module, PyObject* dict_name, PyObject* name) {
  PyObject* d = PyObject_GetAttr(module, dict_name);
  if (d == nullptr) return nullptr;
  PyObject* v = PyDict_Check(d) ? PyDict_GetItemWithError(d, name) : nullptr;
  Py_DECREF(d);
  return v;
}
PyObject* submodule(PyObject* module, PyObject* name) { return entry(module, s__modules, name); }

// A parameter of the activations' dtype on their device.
struct Params {
  at::ScalarType dtype;
  c10::Device device;
  bool ok = true;
  const at::Tensor* get(PyObject* module, PyObject* name) {
    const at::Tensor* t = module == nullptr ? nullptr : dense(entry(module, s__parameters, name));
    if (t == nullptr || t->scalar_type() != dtype || t->device() != device) {
      ok = false;
      return nullptr;
    }
    return t;
  }
  const void* ptr(PyObject* module, PyObject* name) {
    const at::Tensor* t = get(module, name);
    return t == nullptr ? nullptr : t->const_data_ptr();
  }
};

bool int_attr(PyObject* o, PyObject* name, long* v) {
  Ref a(PyObject_GetAttr(o, name));
  if (a.p == nullptr || !PyLong_Check(a.p)) return false;
  *v = PyLong_AsLong(a.p);
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

// The scratch buffer of (device, stream), shared with the Python side, of at least `bytes` bytes.
struct Workspace {
  void* ptr = nullptr;
  size_t bytes = 0;
};
bool workspace(const at::Tensor& on, cudaStream_t stream, size_t bytes, Workspace* ws) {
  Ref key(Py_BuildValue("(iK)", (int)on.device().index(), (unsigned long long)(uintptr_t)stream));
  if (key.p == nullptr) return false;
  PyObject* buf = PyDict_GetItemWithError(g_workspaces, key.p);
  Ref made(nullptr);
  if (buf == nullptr || !THPVariable_Check(buf) ||
      (size_t)THPVariable_Unpack(buf).numel() < bytes) {
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

// RGLRU._packed_gates: the packed copy if its key still describes the weights, else whatever the
// module's own method makes of it.  False: a Python error is set.
bool packed_gates(PyObject* lru, const at::Tensor& wx, const at::Tensor& wa, int dt, const void** out) {
  Ref key(PyObject_GetAttr(lru, s__pack_key));
  if (key.p == nullptr) PyErr_Clear();
  if (key.p != nullptr && PyTuple_Check(key.p) && PyTuple_GET_SIZE(key.p) == 5) {
    const unsigned long long want[5] = {(unsigned long long)(uintptr_t)wx.const_data_ptr(), (unsigned long long)wx._version(),
                                        (unsigned long long)(uintptr_t)wa.const_data_ptr(), (unsigned long long)wa._version(),
                                        (unsigned long long)dt};
    bool same = true;
    for (int i = 0; i < 5 && same; ++i)
      same = PyLong_AsUnsignedLongLong(PyTuple_GET_ITEM(key.p, i)) == want[i];
    if (PyErr_Occurred()) PyErr_Clear();
    if (same) {
      Ref buf(PyObject_GetAttr(lru, s__pack_buf));
      if (buf.p != nullptr && THPVariable_Check(buf.p)) {
        *out = THPVariable_Unpack(buf.p).const_data_ptr();
        return true;
      }
      PyErr_Clear();
    }
  }
  Ref r(PyObject_CallMethodNoArgs(lru, s__packed_gates));
  if (r.p == nullptr) return false;
  *out = r.p == Py_None ? nullptr : PyLong_AsVoidPtr(r.p);
  return !(PyErr_Occurred());
}

// The parameters of Conv1D (may be absent) + RGLRU.
enum class Found { yes, no, error };
Found path_params(PyObject* conv, PyObject* lru, Params& pr, int dt, long width, rgk_params* p,
                  long* heads, long* impl) {
  PyObject* gx = submodule(lru, s_input_gate);
  PyObject* ga = submodule(lru, s_a_gate);
  const at::Tensor* wx = pr.get(gx, s_w);
  const at::Tensor* wa = pr.get(ga, s_w);
  p->gate_x_b = pr.ptr(gx, s_b);
  p->gate_a_b = pr.ptr(ga, s_b);
  p->a_param = pr.ptr(lru, s_a_param);
  if (conv != nullptr) {
    long tw = 0;
    p->conv_w = pr.ptr(conv, s_w);
    p->conv_b = pr.ptr(conv, s_b);
    if (!int_attr(conv, s_temporal_width, &tw) || tw != 4) return Found::no;
  }
  long lru_width = 0;
  if (!pr.ok || !int_attr(lru, s_num_heads, heads) || !int_attr(lru, s_gates_impl, impl) ||
      !int_attr(lru, s_width, &lru_width) || lru_width != width || *heads < 1)
    return Found::no;
  p->gate_x_w = wx->const_data_ptr();
  p->gate_a_w = wa->const_data_ptr();
  p->gates_packed = nullptr;
  if (!packed_gates(lru, *wx, *wa, dt, &p->gates_packed)) return Found::error;
  return Found::yes;
}

PyObject* make_cache(PyObject* h, PyObject* conv) {      // steals both
  Ref rh(h), rc(conv);
  if (h == nullptr || conv == nullptr) return nullptr;
  return PyObject_CallFunctionObjArgs(g_cache_cls, h, conv, nullptr);
}

// ---- recurrent_path(xb, yb, segment_pos, conv_1d, rg_lru, cache, return_cache, out, inplace) -----
PyObject* recurrent_path(PyObject*, PyObject* const* args, Py_ssize_t n) {
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
PyObject* rglru(PyObject*, PyObject* const* args, Py_ssize_t n) {
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

// ---- set-up --------------------------------------------------------------------------------------
// init(librgk path, _workspaces, workspace, check, RecurrentBlockCache)
PyObject* init(PyObject*, PyObject* args) {
  const char* path = nullptr;
  PyObject *spaces, *make, *raise, *cache_cls;
  if (!PyArg_ParseTuple(args, "sO!OOO", &path, &PyDict_Type, &spaces, &make, &raise, &cache_cls))
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
  find(&g_lib.conv1d_prefill, "rgk_conv1d_prefill");
  find(&g_lib.conv1d_decode, "rgk_conv1d_decode");
  if (PyErr_Occurred()) return nullptr;
#define INTERN(n) if (s_##n == nullptr) s_##n = PyUnicode_InternFromString(#n);
  NAMES(INTERN)
#undef INTERN
  g_workspaces = Py_NewRef(spaces);
  g_make_workspace = Py_NewRef(make);
  g_raise = Py_NewRef(raise);
  g_cache_cls = Py_NewRef(cache_cls);
  g_ready = true;
  Py_RETURN_NONE;
}

#define FAST(fn) {#fn, reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(fn)), METH_FASTCALL, nullptr}
PyMethodDef methods[] = {
    {"init", init, METH_VARARGS, nullptr},
    FAST(recurrent_path),
    FAST(rglru),
    {nullptr, nullptr, 0, nullptr}};
PyModuleDef module_def = {PyModuleDef_HEAD_INIT, "_host", nullptr, -1, methods, nullptr, nullptr, nullptr,
                          nullptr};

}  // namespace

PyMODINIT_FUNC PyInit__host() { return PyModule_Create(&module_def); }
