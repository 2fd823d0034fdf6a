// Host-side helpers of the Python layer, as a CPython extension (moe_routers_b200._host).
//
// A small call (a decode step, a route of a few tokens) takes the GPU 10..30 us; seven torch.empty calls from
// Python took 17 us of host time for it, and the layer's check that its stacked weights are still those of its
// parameters 260 us at 64 experts.  Nothing is kept between calls here.
//
//   empties(device_index, ((dtype, size, ..), ..))   -> tuple of uninitialised CUDA tensors
//   weight_state({name: expert module}, (name, ..))  -> bytes: address and version counter of
//       expert.<name>.weight for every expert and name, or None where one is not a plain parameter
#include <torch/csrc/Dtype.h>
#include <torch/csrc/Exceptions.h>
#include <torch/csrc/autograd/python_variable.h>
#include <torch/csrc/utils/object_ptr.h>

#include <ATen/ATen.h>

#include <cstdint>
#include <cstring>

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

PyMethodDef methods[] = {
    {"empties", reinterpret_cast<PyCFunction>(reinterpret_cast<void*>(empties)), METH_FASTCALL, nullptr},
    {"weight_state", reinterpret_cast<PyCFunction>(reinterpret_cast<void*>(weight_state)), METH_FASTCALL, nullptr},
    {nullptr, nullptr, 0, nullptr},
};
PyModuleDef module = {PyModuleDef_HEAD_INIT, "_host", nullptr, -1, methods, nullptr, nullptr, nullptr, nullptr};

}  // namespace

extern "C" __attribute__((visibility("default"))) PyObject* PyInit__host(void) { return PyModule_Create(&module); }
