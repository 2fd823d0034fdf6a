// Host-side helpers of the Python layer, as a CPython extension (moe_routers_b200._host).
//
// A small call (a decode step, a route of a few tokens) takes the GPU 10..30 us, and the Python that prepared it
// took longer: allocations, tensor attributes, a ctypes call of twenty arguments, once per launch.  Here a whole
// operator is one call: its inputs are looked over, its outputs allocated and the entry points of libmoe_b200.so
// called through their addresses.  What is not plain (another device, a copy to be made first, an option, a
// wrong argument) returns None, and the Python function behind takes it with its own checks and messages.
// Calls one behind the other, Python before -> now: route of 16 x 4096: 19.4 -> 13.0 us; MoELayer, 8 experts, 16 tokens,
// 1088 -> 1408: 70 -> 41; grouped_ffn_forward on 64 pairs, 25 rows: 277 -> 44 (8 pairs: 87 -> 30).
// Nothing is kept between calls here.
//
//   bind({entry point: address}, workspaces, new_workspace, check)   once, at import
//   route(dev, stream, x, w, top_k, skew_experts, skew_bias, with_logits)      -> dict
//   fused_select(dev, stream, logits, x, experts, top_k)                       -> 7 tensors
//   sinkhorn(dev, stream, router_types, logits, top_k, iters, eps, temperature)-> (idx, gates)
//   expert_ffn(dev, stream, rows, w1, w2, offsets, activation, gates, route_row, top_k) -> output
//   grouped_lists(dev, stream, inputs, weights)                                -> list of outputs
//   empties(device_index, ((dtype, size, ..), ..))   -> tuple of uninitialised CUDA tensors
//   weight_state({name: expert module}, (name, ..))  -> bytes: address and version counter of
//       expert.<name>.weight for every expert and name, or None where one is not a plain parameter
#include "../../include/moe_b200.h"

#include <torch/csrc/Dtype.h>
#include <torch/csrc/Exceptions.h>
#include <torch/csrc/autograd/python_variable.h>
#include <torch/csrc/utils/object_ptr.h>

#include <ATen/ATen.h>

#include <algorithm>
#include <cstdint>
#include <cstring>
#include <initializer_list>
#include <vector>

namespace {

// The GIL is given up for as long as one of these lives: an allocation may have to wait for the device, whose
// work may in turn need a launch by another Python thread.
struct WithoutGil {
  PyThreadState* state = PyEval_SaveThread();
  ~WithoutGil() { PyEval_RestoreThread(state); }
};

struct TensorSpec {
  at::ScalarType type;
  int64_t sizes[3];
  int dims;
};

PyObject* empties(PyObject*, PyObject* const* args, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  TORCH_CHECK(n == 2 && PyTuple_Check(args[1]), "empties(device_index, ((dtype, size, ..), ..))");
  const long dev = PyLong_AsLong(args[0]);
  if (dev == -1 && PyErr_Occurred()) return nullptr;
  const at::TensorOptions on_gpu = at::TensorOptions().device(at::Device(at::kCUDA, (c10::DeviceIndex)dev));
  const Py_ssize_t count = PyTuple_GET_SIZE(args[1]);
  c10::SmallVector<TensorSpec, 8> specs(count);
  for (Py_ssize_t i = 0; i < count; ++i) {
    PyObject* spec = PyTuple_GET_ITEM(args[1], i);
    TORCH_CHECK(PyTuple_Check(spec) && PyTuple_GET_SIZE(spec) >= 1 && PyTuple_GET_SIZE(spec) <= 4 &&
                    THPDtype_Check(PyTuple_GET_ITEM(spec, 0)),
                "empties: (dtype, up to three sizes) expected");
    specs[i].type = reinterpret_cast<THPDtype*>(PyTuple_GET_ITEM(spec, 0))->scalar_type;
    specs[i].dims = (int)PyTuple_GET_SIZE(spec) - 1;
    for (int d = 0; d < specs[i].dims; ++d) {
      specs[i].sizes[d] = PyLong_AsLongLong(PyTuple_GET_ITEM(spec, d + 1));
      if (specs[i].sizes[d] == -1 && PyErr_Occurred()) return nullptr;
    }
  }
  c10::SmallVector<at::Tensor, 8> tensors(count);
  {
    WithoutGil released;
    for (Py_ssize_t i = 0; i < count; ++i)
      tensors[i] = at::empty(at::IntArrayRef(specs[i].sizes, specs[i].dims), on_gpu.dtype(specs[i].type));
  }
  THPObjectPtr out(PyTuple_New(count));
  if (!out) return nullptr;
  for (Py_ssize_t i = 0; i < count; ++i) {
    PyObject* t = THPVariable_Wrap(std::move(tensors[i]));
    if (t == nullptr) return nullptr;
    PyTuple_SET_ITEM(out.get(), i, t);
  }
  return out.release();
  END_HANDLE_TH_ERRORS
}

// obj.<name>'s entry `key` where obj.<name> is a dict that has one (a module's own tables), else null; borrowed
// from the dict, which its owner keeps alive while nothing else runs.
PyObject* table_entry(PyObject* obj, PyObject* table, PyObject* key) {
  PyObject* dict = PyObject_GetAttr(obj, table);
  if (dict == nullptr) throw python_error();
  PyObject* found = PyDict_Check(dict) ? PyDict_GetItemWithError(dict, key) : nullptr;
  Py_DECREF(dict);
  if (found == nullptr && PyErr_Occurred()) throw python_error();
  return found;
}

PyObject* weight_state(PyObject*, PyObject* const* args, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  TORCH_CHECK(n == 2 && PyDict_Check(args[0]) && PyTuple_Check(args[1]), "weight_state({name: module}, (name, ..))");
  static PyObject* const modules = PyUnicode_InternFromString("_modules");
  static PyObject* const parameters = PyUnicode_InternFromString("_parameters");
  static PyObject* const weight = PyUnicode_InternFromString("weight");
  const Py_ssize_t names = PyTuple_GET_SIZE(args[1]);
  PyObject* out = PyBytes_FromStringAndSize(nullptr, PyDict_GET_SIZE(args[0]) * names * 16);
  if (out == nullptr) return nullptr;
  char* dst = PyBytes_AS_STRING(out);
  try {
    PyObject *key, *expert;
    Py_ssize_t pos = 0;
    while (PyDict_Next(args[0], &pos, &key, &expert)) {
      for (Py_ssize_t i = 0; i < names; ++i) {
        PyObject* sub = table_entry(expert, modules, PyTuple_GET_ITEM(args[1], i));
        PyObject* p = sub != nullptr ? table_entry(sub, parameters, weight) : nullptr;
        // a weight that is no plain parameter (a parametrisation, an assigned tensor): the caller looks it up
        if (p == nullptr || !THPVariable_Check(p)) {
          Py_DECREF(out);
          Py_RETURN_NONE;
        }
        const at::Tensor& t = THPVariable_Unpack(p);
        const uint64_t pair[2] = {reinterpret_cast<uint64_t>(t.data_ptr()),
                                  static_cast<uint64_t>(t.unsafeGetTensorImpl()->version_counter().current_version())};
        memcpy(dst, pair, 16);
        dst += 16;
      }
    }
  } catch (...) {
    Py_DECREF(out);
    throw;
  }
  return out;
  END_HANDLE_TH_ERRORS
}

// ---- operators in one call ---------------------------------------------------------------------------
struct Api {
  decltype(&moe_workspace_bytes) workspace_bytes;
  decltype(&moe_route_fused) route_fused;
  decltype(&moe_fused_select) fused_select;
  decltype(&moe_sinkhorn) sinkhorn;
  decltype(&moe_sinkhorn_router) sinkhorn_router;
  decltype(&moe_grouped_gemm) grouped_gemm;
  decltype(&moe_expert_ffn) expert_ffn;
  decltype(&moe_store_offsets) store_offsets;
};
Api api;
PyObject* workspaces;     // {(device, stream): tensor}
PyObject* new_workspace;  // (device, tokens, experts, top_k) -> tensor, for what the table does not hold
PyObject* check_status;   // raises the library's error

PyObject* bind(PyObject*, PyObject* const* args, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  TORCH_CHECK(n == 4 && PyDict_Check(args[0]) && PyDict_Check(args[1]), "bind({name: address}, workspaces, new_workspace, check)");
  const struct { const char* name; void** to; } entries[] = {
      {"moe_workspace_bytes", reinterpret_cast<void**>(&api.workspace_bytes)},
      {"moe_route_fused", reinterpret_cast<void**>(&api.route_fused)},
      {"moe_fused_select", reinterpret_cast<void**>(&api.fused_select)},
      {"moe_sinkhorn", reinterpret_cast<void**>(&api.sinkhorn)},
      {"moe_sinkhorn_router", reinterpret_cast<void**>(&api.sinkhorn_router)},
      {"moe_grouped_gemm", reinterpret_cast<void**>(&api.grouped_gemm)},
      {"moe_expert_ffn", reinterpret_cast<void**>(&api.expert_ffn)},
      {"moe_store_offsets", reinterpret_cast<void**>(&api.store_offsets)},
  };
  for (const auto& e : entries) {
    PyObject* address = PyDict_GetItemString(args[0], e.name);
    TORCH_CHECK(address != nullptr, "bind: no address of ", e.name);
    *e.to = PyLong_AsVoidPtr(address);
    if (PyErr_Occurred()) return nullptr;
  }
  PyObject** const kept[] = {&workspaces, &new_workspace, &check_status};
  for (int i = 0; i < 3; ++i) {
    Py_INCREF(args[1 + i]);
    Py_XSETREF(*kept[i], args[1 + i]);
  }
  Py_RETURN_NONE;
  END_HANDLE_TH_ERRORS
}

// An argument that a kernel can read as it is: a plain contiguous tensor of the current device, of `dims`
// dimensions; null otherwise.
const at::Tensor* plain(PyObject* o, long dev, int dims) {
  if (!THPVariable_CheckExact(o)) return nullptr;
  const at::Tensor& t = THPVariable_Unpack(o);
  if (!t.is_cuda() || t.layout() != at::kStrided || t.dim() != dims || t.get_device() != dev || !t.is_contiguous()) return nullptr;
  return &t;
}
bool half_type(const at::Tensor& t) { return t.scalar_type() == at::kHalf || t.scalar_type() == at::kBFloat16; }
int type_code(const at::Tensor& t) {
  return t.scalar_type() == at::kHalf ? MOE_F16 : t.scalar_type() == at::kBFloat16 ? MOE_BF16 : t.scalar_type() == at::kFloat ? MOE_F32 : -1;
}
bool small_int(PyObject* o, int lo, int hi, int& v) {
  if (!PyLong_CheckExact(o)) return false;
  int over = 0;
  const long l = PyLong_AsLongAndOverflow(o, &over);
  if (over != 0 || l < lo || l > hi) return false;
  v = (int)l;
  return true;
}
bool number(PyObject* o, float& v) {
  if (!PyFloat_CheckExact(o) && !PyLong_CheckExact(o)) return false;
  const double d = PyFloat_AsDouble(o);
  if (d == -1.0 && PyErr_Occurred()) { PyErr_Clear(); return false; }
  v = (float)d;
  return true;
}
constexpr int kMaxInt = 0x7fffffff;
bool fits(const at::Tensor& t) {
  for (const int64_t n : t.sizes())
    if (n > kMaxInt) return false;
  return true;
}

// Device and stream of the call, and the calling stream's scratch buffer.
struct Call {
  long dev;
  void* stream;
  PyObject* key_stream;
  THPObjectPtr ws_ref;
  void* ws = nullptr;
  size_t ws_bytes = 0;

  Call(PyObject* device, PyObject* stream_) : dev(PyLong_AsLong(device)), stream(PyLong_AsVoidPtr(stream_)), key_stream(stream_) {
    if (PyErr_Occurred()) throw python_error();
  }
  void workspace(PyObject* device, int tokens, int experts, int top_k) {
    const size_t need = std::max<size_t>(api.workspace_bytes(tokens, experts, top_k), 1 << 16);
    THPObjectPtr key(PyTuple_Pack(2, device, key_stream));
    if (!key) throw python_error();
    PyObject* found = PyDict_GetItemWithError(workspaces, key.get());
    if (found == nullptr && PyErr_Occurred()) throw python_error();
    if (found != nullptr && THPVariable_Check(found) && (size_t)THPVariable_Unpack(found).numel() >= need) {
      Py_INCREF(found);
      ws_ref = found;
    } else {
      ws_ref = PyObject_CallFunction(new_workspace, "Oiii", device, tokens, experts, top_k);
      if (!ws_ref) throw python_error();
    }
    const at::Tensor& t = THPVariable_Unpack(ws_ref.get());
    ws = t.data_ptr();
    ws_bytes = (size_t)t.numel();
  }
  at::TensorOptions on_gpu() const { return at::TensorOptions().device(at::Device(at::kCUDA, (c10::DeviceIndex)dev)); }
  at::Tensor make(at::IntArrayRef sizes, at::ScalarType type) const { return at::empty(sizes, on_gpu().dtype(type)); }
};
// Raises the error of an entry point that did not return MOE_OK.
void checked(int rc) {
  if (rc == MOE_OK) return;
  THPObjectPtr r(PyObject_CallFunction(check_status, "i", rc));
  throw python_error();
}
template <typename T>
T* data(const at::Tensor& t) { return static_cast<T*>(t.data_ptr()); }

struct Routing {
  at::Tensor idx, gates, packed, counts, offsets, row_route, route_row, logits;
  void make(const Call& c, int64_t t, int64_t d, int64_t e, int64_t k, at::ScalarType type, bool with_logits) {
    idx = c.make({t, k}, at::kInt);
    gates = c.make({t, k}, at::kFloat);
    packed = c.make({t * k, d}, type);
    counts = c.make({e}, at::kInt);
    offsets = c.make({e + 1}, at::kInt);
    row_route = c.make({t * k}, at::kInt);
    route_row = c.make({t * k}, at::kInt);
    if (with_logits) logits = c.make({t, e}, at::kFloat);
  }
};

PyObject* route(PyObject*, PyObject* const* args, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  TORCH_CHECK(n == 8, "route: 8 arguments");
  Call c(args[0], args[1]);
  const at::Tensor *x = plain(args[2], c.dev, 2), *w = plain(args[3], c.dev, 2);
  int k, skew;
  float bias;
  if (!x || !w || !half_type(*x) || w->scalar_type() != x->scalar_type() || !fits(*x) || !fits(*w) ||
      !small_int(args[4], 1, 8, k) || !small_int(args[5], -kMaxInt, kMaxInt, skew) || !number(args[6], bias)) Py_RETURN_NONE;
  const bool with_logits = args[7] == Py_True;
  const int64_t t = x->size(0), d = x->size(1), e = w->size(0);
  if (e == 0 || w->size(1) != d || t * k > kMaxInt) Py_RETURN_NONE;
  c.workspace(args[0], (int)t, (int)e, k);
  Routing r;
  int rc;
  {
    WithoutGil released;
    r.make(c, t, d, e, k, x->scalar_type(), with_logits);
    rc = api.route_fused(x->data_ptr(), w->data_ptr(), type_code(*x), (int)t, (int)d, (int)e, k, skew, bias, data<int32_t>(r.idx),
                         data<float>(r.gates), data<int32_t>(r.counts), data<int32_t>(r.offsets), r.packed.data_ptr(),
                         data<int32_t>(r.row_route), data<int32_t>(r.route_row), with_logits ? data<float>(r.logits) : nullptr,
                         c.ws, c.ws_bytes, c.stream);
  }
  checked(rc);
  THPObjectPtr out(PyDict_New());
  if (!out) return nullptr;
  static PyObject* const names[] = {
      PyUnicode_InternFromString("idx"), PyUnicode_InternFromString("gates"), PyUnicode_InternFromString("counts"),
      PyUnicode_InternFromString("offsets"), PyUnicode_InternFromString("packed"), PyUnicode_InternFromString("row_route"),
      PyUnicode_InternFromString("route_row"), PyUnicode_InternFromString("logits")};
  at::Tensor* const tensors[] = {&r.idx, &r.gates, &r.counts, &r.offsets, &r.packed, &r.row_route, &r.route_row, &r.logits};
  for (int i = 0; i < (with_logits ? 8 : 7); ++i) {
    THPObjectPtr v(THPVariable_Wrap(std::move(*tensors[i])));
    if (!v || PyDict_SetItem(out.get(), names[i], v.get()) != 0) return nullptr;
  }
  static PyObject* const workspace = PyUnicode_InternFromString("workspace");
  if (PyDict_SetItem(out.get(), workspace, c.ws_ref.get()) != 0) return nullptr;
  return out.release();
  END_HANDLE_TH_ERRORS
}

PyObject* tuple_of(std::initializer_list<at::Tensor*> tensors) {
  THPObjectPtr out(PyTuple_New((Py_ssize_t)tensors.size()));
  if (!out) throw python_error();
  Py_ssize_t i = 0;
  for (at::Tensor* t : tensors) {
    PyObject* v = THPVariable_Wrap(std::move(*t));
    if (v == nullptr) throw python_error();
    PyTuple_SET_ITEM(out.get(), i++, v);
  }
  return out.release();
}

PyObject* fused_select(PyObject*, PyObject* const* args, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  TORCH_CHECK(n == 6, "fused_select: 6 arguments");
  Call c(args[0], args[1]);
  const at::Tensor *logits = plain(args[2], c.dev, 2), *x = plain(args[3], c.dev, 2);
  int e, k;
  if (!logits || !x || type_code(*logits) < 0 || !fits(*x) || x->element_size() > kMaxInt || !small_int(args[4], 1, 1024, e) ||
      !small_int(args[5], 1, 8, k)) Py_RETURN_NONE;
  const int64_t t = x->size(0), d = x->size(1);
  if (logits->size(0) < t || logits->size(1) != e || t * k > kMaxInt) Py_RETURN_NONE;
  c.workspace(args[0], (int)t, e, k);
  Routing r;
  int rc;
  {
    WithoutGil released;
    r.make(c, t, d, e, k, x->scalar_type(), false);
    rc = api.fused_select(logits->data_ptr(), type_code(*logits), x->data_ptr(), (int)x->element_size(), (int)t, (int)d, e, k,
                          data<int32_t>(r.idx), data<float>(r.gates), data<int32_t>(r.counts), data<int32_t>(r.offsets),
                          r.packed.data_ptr(), data<int32_t>(r.row_route), data<int32_t>(r.route_row), c.ws, c.ws_bytes, c.stream);
  }
  checked(rc);
  return tuple_of({&r.idx, &r.gates, &r.counts, &r.offsets, &r.packed, &r.row_route, &r.route_row});
  END_HANDLE_TH_ERRORS
}

PyObject* sinkhorn(PyObject*, PyObject* const* args, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  TORCH_CHECK(n == 8, "sinkhorn: 8 arguments");
  Call c(args[0], args[1]);
  const bool router = args[2] == Py_True;
  const at::Tensor* logits = plain(args[3], c.dev, 2);
  int k, iters;
  float eps, temperature;
  if (!logits || type_code(*logits) < 0 || !fits(*logits) || !small_int(args[4], 1, 8, k) || !small_int(args[5], -kMaxInt, kMaxInt, iters) ||
      !number(args[6], eps) || !number(args[7], temperature)) Py_RETURN_NONE;
  const int64_t t = logits->size(0), e = logits->size(1);
  if (e == 0) Py_RETURN_NONE;
  c.workspace(args[0], (int)t, (int)e, k);
  at::Tensor idx, gates;
  int rc;
  {
    WithoutGil released;
    idx = c.make({t, k}, router ? at::kLong : at::kInt);
    gates = c.make({t, k}, router ? logits->scalar_type() : at::kFloat);
    rc = router ? api.sinkhorn_router(logits->data_ptr(), type_code(*logits), (int)t, (int)e, k, iters, eps, temperature,
                                      data<int64_t>(idx), gates.data_ptr(), c.ws, c.ws_bytes, c.stream)
                : api.sinkhorn(logits->data_ptr(), type_code(*logits), (int)t, (int)e, k, iters, eps, temperature,
                               data<int32_t>(idx), data<float>(gates), c.ws, c.ws_bytes, c.stream);
  }
  checked(rc);
  return tuple_of({&idx, &gates});
  END_HANDLE_TH_ERRORS
}

PyObject* expert_ffn(PyObject*, PyObject* const* args, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  TORCH_CHECK(n == 10, "expert_ffn: 10 arguments");
  Call c(args[0], args[1]);
  const at::Tensor *a = plain(args[2], c.dev, 2), *w1 = plain(args[3], c.dev, 3), *w2 = plain(args[4], c.dev, 3);
  const at::Tensor *offsets = plain(args[5], c.dev, 1), *gates = plain(args[7], c.dev, 2), *route_row = plain(args[8], c.dev, 1);
  int act, k;
  if (!a || !w1 || !w2 || !offsets || !gates || !route_row || !small_int(args[6], 0, 3, act) || !small_int(args[9], 1, 8, k) ||
      !half_type(*a) || w1->scalar_type() != a->scalar_type() || w2->scalar_type() != a->scalar_type() ||
      offsets->scalar_type() != at::kInt || gates->scalar_type() != at::kFloat || route_row->scalar_type() != at::kInt ||
      !fits(*a) || !fits(*w1) || !fits(*w2)) Py_RETURN_NONE;
  const int64_t rows = a->size(0), d = a->size(1), e = w1->size(0);
  const int64_t h = act == MOE_ACT_SWIGLU ? w1->size(1) / 2 : w1->size(1), d2 = w2->size(1);
  const int64_t routes = rows / k * k;
  // (with an odd number of SwiGLU features an expert's weights are not 2 h rows apart, which moe_expert_ffn assumes)
  if (e == 0 || (act == MOE_ACT_SWIGLU && w1->size(1) % 2 != 0) || w1->size(2) != d || w2->size(0) != e || w2->size(2) != h || offsets->numel() <= e || gates->numel() < routes ||
      gates->size(1) != k || route_row->numel() < routes) Py_RETURN_NONE;
  c.workspace(args[0], 1, (int)e, 1);
  const int type = type_code(*a);
  at::Tensor hidden, y, out;
  int rc;
  {
    WithoutGil released;
    hidden = c.make({rows, h}, a->scalar_type());
    y = c.make({rows, d2}, a->scalar_type());
    out = c.make({rows / k, d2}, a->scalar_type());
    rc = api.expert_ffn(a->data_ptr(), w1->data_ptr(), hidden.data_ptr(), w2->data_ptr(), y.data_ptr(), data<int32_t>(*offsets), (int)e,
                        (int)rows, (int)d, (int)h, (int)d2, act, data<float>(*gates), data<int32_t>(*route_row), k, out.data_ptr(),
                        type, c.ws, c.ws_bytes, c.stream);
  }
  checked(rc);
  return THPVariable_Wrap(std::move(out));
  END_HANDLE_TH_ERRORS
}

// The tensors of a list as one buffer: all fp16, of `cols` columns (and, with `same_rows`, of one shape), each
// beginning where the one before it ends, inside one storage.  Tensors without rows lie anywhere.  `first` becomes a
// reference of its own, which holds that storage: the list is the caller's, and another thread may change it as soon as
// the GIL is given up or Python code runs.
bool one_buffer(PyObject* list, long dev, int64_t cols, bool same_rows, at::Tensor& first, int64_t& rows, int64_t* counts) {
  const Py_ssize_t n = PyList_GET_SIZE(list);
  rows = 0;
  const char* next = nullptr;
  for (Py_ssize_t i = 0; i < n; ++i) {
    const at::Tensor* t = plain(PyList_GET_ITEM(list, i), dev, 2);
    if (!t || t->scalar_type() != at::kHalf || t->size(1) != cols) return false;
    counts[i] = t->size(0);
    rows += counts[i];
    if (same_rows && counts[i] != counts[0]) return false;
    if (t->numel() == 0) continue;
    const char* at = static_cast<const char*>(t->data_ptr());
    if (!first.defined()) first = *t;
    else if (at != next) return false;
    next = at + t->numel() * 2;
  }
  if (!first.defined() || rows > kMaxInt) return false;
  const c10::Storage& storage = first.storage();
  return next <= static_cast<const char*>(storage.data()) + storage.nbytes();
}

PyObject* grouped_lists(PyObject*, PyObject* const* args, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  TORCH_CHECK(n == 4, "grouped_lists: 4 arguments");
  Call c(args[0], args[1]);
  if (!PyList_CheckExact(args[2]) || !PyList_CheckExact(args[3])) Py_RETURN_NONE;
  const Py_ssize_t e = PyList_GET_SIZE(args[2]);
  if (e == 0 || e > 1024 || PyList_GET_SIZE(args[3]) != e) Py_RETURN_NONE;
  const at::Tensor* w0 = plain(PyList_GET_ITEM(args[3], 0), c.dev, 2);
  if (!w0) Py_RETURN_NONE;
  const int64_t k = w0->size(0), cols = w0->size(1);
  at::Tensor a, w;
  int64_t rows, w_rows;
  c10::SmallVector<int64_t, 64> counts(e), w_counts(e);
  if (k > kMaxInt || cols > kMaxInt || !one_buffer(args[2], c.dev, k, false, a, rows, counts.data()) ||
      !one_buffer(args[3], c.dev, cols, true, w, w_rows, w_counts.data())) Py_RETURN_NONE;
  c.workspace(args[0], 1, (int)e, 1);
  c10::SmallVector<int32_t, 65> ends(e + 1);
  ends[0] = 0;
  for (Py_ssize_t i = 0; i < e; ++i) ends[i + 1] = ends[i] + (int32_t)counts[i];
  std::vector<at::Tensor> pieces;
  int rc;
  {
    WithoutGil released;
    const at::Tensor offsets = c.make({e + 1}, at::kInt), out = c.make({rows, cols}, at::kHalf);
    rc = api.store_offsets(ends.data(), (int)e + 1, data<int32_t>(offsets), c.stream);
    if (rc == MOE_OK)
      rc = api.grouped_gemm(a.data_ptr(), w.data_ptr(), out.data_ptr(), data<int32_t>(offsets), (int)e, (int)rows, (int)k, (int)cols,
                            MOE_W_KN, k * cols, MOE_ACT_NONE, nullptr, nullptr, MOE_F16, 0, c.ws, c.ws_bytes, c.stream);
    if (rc == MOE_OK) pieces = out.split_with_sizes(counts, 0);
  }
  checked(rc);
  THPObjectPtr list(PyList_New(e));
  if (!list) return nullptr;
  for (Py_ssize_t i = 0; i < e; ++i) {
    PyObject* v = THPVariable_Wrap(std::move(pieces[i]));
    if (v == nullptr) return nullptr;
    PyList_SET_ITEM(list.get(), i, v);
  }
  return list.release();
  END_HANDLE_TH_ERRORS
}

#define MOE_METHOD(f) {#f, reinterpret_cast<PyCFunction>(reinterpret_cast<void*>(f)), METH_FASTCALL, nullptr}
PyMethodDef methods[] = {
    MOE_METHOD(bind), MOE_METHOD(route), MOE_METHOD(fused_select), MOE_METHOD(sinkhorn), MOE_METHOD(expert_ffn),
    MOE_METHOD(grouped_lists),
    {"empties", reinterpret_cast<PyCFunction>(reinterpret_cast<void*>(empties)), METH_FASTCALL, nullptr},
    {"weight_state", reinterpret_cast<PyCFunction>(reinterpret_cast<void*>(weight_state)), METH_FASTCALL, nullptr},
    {nullptr, nullptr, 0, nullptr},
};
PyModuleDef module = {PyModuleDef_HEAD_INIT, "_host", nullptr, -1, methods, nullptr, nullptr, nullptr, nullptr};

}  // namespace

extern "C" __attribute__((visibility("default"))) PyObject* PyInit__host(void) { return PyModule_Create(&module); }
