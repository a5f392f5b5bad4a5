// Entry points that take torch tensors as they are: argument checks, output allocation and the
// current stream in C++ instead of a dozen Python attribute reads per call, each 0.1-0.5 us on the
// path of a kernel that takes 3 us. Every function returns None without an effect when an argument
// is not what it handles; the Python wrapper then says what is wrong with it.
#include <Python.h>
#include <torch/csrc/autograd/python_variable.h>

#include <ATen/ops/empty.h>
#include <c10/cuda/CUDAStream.h>

#include <cstdint>

#include "../bindings/native_api.h"

namespace {

const pplx_py::NativeApi* g_api = nullptr;

// Borrowed view of a tensor argument; nullptr when `obj` is no tensor.
inline const at::Tensor* tensor(PyObject* obj) { return THPVariable_Check(obj) ? &THPVariable_Unpack(obj) : nullptr; }

inline bool is_matrix(const at::Tensor& t, int64_t rows, int64_t cols, at::ScalarType type) {
  return t.dim() == 2 && t.size(0) == rows && t.size(1) == cols && t.stride(1) == 1 && t.scalar_type() == type;
}

inline at::Tensor new_matrix(const at::Tensor& like, int64_t rows, int64_t cols, at::ScalarType type) {
  return at::empty({rows, cols}, like.options().dtype(type));
}

template <typename F>
PyObject* guarded(F&& f) {
  try {
    return f();
  } catch (const std::exception& e) {
    if (!PyErr_Occurred()) PyErr_SetString(PyExc_RuntimeError, e.what());
    return nullptr;
  }
}

// topk_route(logits, topk, bias | None, out_indices | None, out_weights | None) -> (indices, weights)
PyObject* topk_route(PyObject*, PyObject* const* args, Py_ssize_t nargs) {
  return guarded([&]() -> PyObject* {
    if (nargs != 5) Py_RETURN_NONE;
    const at::Tensor* logits = tensor(args[0]);
    const int64_t k = PyLong_AsLongLong(args[1]);
    if (k == -1 && PyErr_Occurred()) return nullptr;
    if (logits == nullptr || !logits->is_cuda() || logits->dim() != 2 || logits->stride(1) != 1) Py_RETURN_NONE;
    const at::ScalarType type = logits->scalar_type();
    if (type != at::kFloat && type != at::kBFloat16) Py_RETURN_NONE;
    const int64_t tokens = logits->size(0), experts = logits->size(1);
    const at::Tensor* bias = nullptr;
    if (args[2] != Py_None) {
      bias = tensor(args[2]);
      if (bias == nullptr || bias->dim() != 1 || bias->size(0) != experts || bias->scalar_type() != at::kFloat ||
          !bias->is_contiguous()) {
        Py_RETURN_NONE;
      }
    }
    at::Tensor out[2];
    constexpr at::ScalarType kTypes[2] = {at::kUInt32, at::kFloat};
    for (int i = 0; i < 2; ++i) {
      if (args[3 + i] == Py_None) {
        out[i] = new_matrix(*logits, tokens, k, kTypes[i]);
      } else {
        const at::Tensor* given = tensor(args[3 + i]);
        if (given == nullptr || !is_matrix(*given, tokens, k, kTypes[i])) Py_RETURN_NONE;
        out[i] = *given;
      }
    }
    pplx::ops::TopkRouteParams p;
    p.logits = logits->const_data_ptr();
    p.logits_stride = logits->stride(0);
    p.logits_bf16 = type == at::kBFloat16;
    p.bias = bias == nullptr ? nullptr : static_cast<const float*>(bias->const_data_ptr());
    p.indices = static_cast<uint32_t*>(out[0].data_ptr());
    p.indices_stride = out[0].stride(0);
    p.weights = static_cast<float*>(out[1].data_ptr());
    p.weights_stride = out[1].stride(0);
    p.tokens = static_cast<int>(tokens);
    p.num_experts = static_cast<int>(experts);
    p.k = static_cast<int>(k);
    if (!g_api->topk_route(p, c10::cuda::getCurrentCUDAStream().stream())) return nullptr;
    PyObject* result = PyTuple_New(2);
    if (result == nullptr) return nullptr;
    for (int i = 0; i < 2; ++i) {
      PyObject* item = args[3 + i];
      if (item == Py_None) {
        item = THPVariable_Wrap(std::move(out[i]));
        if (item == nullptr) {
          Py_DECREF(result);
          return nullptr;
        }
      } else {
        Py_INCREF(item);
      }
      PyTuple_SET_ITEM(result, i, item);
    }
    return result;
  });
}

PyMethodDef kMethods[] = {
    {"topk_route", reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(topk_route)), METH_FASTCALL, nullptr},
    {nullptr, nullptr, 0, nullptr},
};

PyModuleDef kModule = {PyModuleDef_HEAD_INIT, "_torch_ops", "Entry points that read torch tensors natively.", -1, kMethods};

}  // namespace

extern "C" __attribute__((visibility("default"))) PyObject* PyInit__torch_ops() {
  PyObject* native = PyImport_ImportModule("pplx_garden._native");
  if (native == nullptr) return nullptr;
  PyObject* capsule = PyObject_GetAttrString(native, "_api");
  Py_DECREF(native);   // sys.modules keeps it
  if (capsule == nullptr) return nullptr;
  g_api = static_cast<const pplx_py::NativeApi*>(PyCapsule_GetPointer(capsule, pplx_py::kNativeApiName));
  Py_DECREF(capsule);  // an attribute of the module
  if (g_api == nullptr) return nullptr;
  return PyModule_Create(&kModule);
}
