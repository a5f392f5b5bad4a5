// Entry points that take torch tensors as they are: argument checks, output allocation and the
// current stream in C++ instead of a dozen Python attribute reads per call, each 0.1-0.5 us on the
// path of a kernel that takes 3 us. Every function returns None without an effect when an argument
// is not what it handles; the Python wrapper then says what is wrong with it.
#include <Python.h>
#include <torch/csrc/Dtype.h>
#include <torch/csrc/autograd/python_variable.h>

#include <ATen/ops/empty.h>
#include <ATen/ops/zeros.h>
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

// ---------------------------------------------------------------------------
// all-to-all
// ---------------------------------------------------------------------------

// What the argument checks of one context depend on; a capsule that the Python object keeps.
struct A2APlan {
  void* context;
  int64_t topk, hidden, scales, local_experts, num_experts, world;   // scales: 0 = none
  at::ScalarType in_type, out_type;
  int quantize_mode;
};
constexpr const char* kPlanName = "pplx_garden.a2a_plan";

const A2APlan* plan_of(PyObject* capsule) {
  return static_cast<const A2APlan*>(PyCapsule_GetPointer(capsule, kPlanName));
}

// a2a_plan(handle, topk, hidden, scales, local_experts, num_experts, world, in_dtype, out_dtype, quantize_mode)
PyObject* a2a_plan(PyObject*, PyObject* const* args, Py_ssize_t nargs) {
  if (nargs != 10 || !THPDtype_Check(args[7]) || !THPDtype_Check(args[8])) {
    PyErr_SetString(PyExc_TypeError, "a2a_plan takes seven numbers, two dtypes and a number");
    return nullptr;
  }
  int64_t v[10] = {};
  for (int i = 0; i < 10; ++i) {
    if (i != 7 && i != 8) v[i] = static_cast<int64_t>(PyLong_AsUnsignedLongLong(args[i]));
  }
  if (PyErr_Occurred()) return nullptr;
  auto* plan = new A2APlan{reinterpret_cast<void*>(v[0]), v[1], v[2], v[3], v[4], v[5], v[6],
                           reinterpret_cast<THPDtype*>(args[7])->scalar_type,
                           reinterpret_cast<THPDtype*>(args[8])->scalar_type, static_cast<int>(v[9])};
  PyObject* capsule = PyCapsule_New(plan, kPlanName, [](PyObject* c) { delete plan_of(c); });
  if (capsule == nullptr) delete plan;
  return capsule;
}

template <typename T>
T* ptr(const at::Tensor& t) {
  return static_cast<T*>(const_cast<void*>(t.const_data_ptr()));
}

// The routing table and the optional token bound, as dispatch and combine take them.
bool routing_ok(const A2APlan& p, const at::Tensor* indices, const at::Tensor* weights, int64_t tokens) {
  return indices != nullptr && weights != nullptr && is_matrix(*indices, tokens, p.topk, at::kUInt32) &&
         is_matrix(*weights, tokens, p.topk, at::kFloat);
}
bool bound_ok(PyObject* obj, const int32_t** out) {
  *out = nullptr;
  if (obj == Py_None) return true;
  const at::Tensor* t = tensor(obj);
  if (t == nullptr || t->numel() != 1 || t->scalar_type() != at::kInt) return false;
  *out = ptr<const int32_t>(*t);
  return true;
}

// a2a_dispatch(plan, out_num_tokens, out_x, out_x_scale | None, x, x_scale | None, indices, weights,
//              bound_m | None, do_send, do_recv, logits | None, logits_bias | None) -> True | None
PyObject* a2a_dispatch(PyObject*, PyObject* const* args, Py_ssize_t nargs) {
  return guarded([&]() -> PyObject* {
    if (nargs != 13) Py_RETURN_NONE;
    const A2APlan* plan = plan_of(args[0]);
    if (plan == nullptr) return nullptr;
    const A2APlan& p = *plan;
    const at::Tensor *num = tensor(args[1]), *out_x = tensor(args[2]), *x = tensor(args[4]);
    const at::Tensor *indices = tensor(args[6]), *weights = tensor(args[7]);
    const bool send = PyObject_IsTrue(args[9]) == 1, recv = PyObject_IsTrue(args[10]) == 1;
    if (num == nullptr || out_x == nullptr || x == nullptr || (!send && !recv)) Py_RETURN_NONE;
    if (num->dim() != 1 || num->size(0) != p.local_experts || num->scalar_type() != at::kInt || num->stride(0) != 1) {
      Py_RETURN_NONE;
    }
    if (out_x->dim() != 2 || !is_matrix(*out_x, out_x->size(0), p.hidden, p.in_type)) Py_RETURN_NONE;
    if (x->dim() != 2 || x->size(1) != p.hidden || x->stride(1) != 1) Py_RETURN_NONE;
    const int64_t tokens = x->size(0);
    const at::Tensor *out_scale = nullptr, *x_scale = nullptr;
    for (int i : {3, 5}) {
      if (args[i] == Py_None) continue;
      const at::Tensor* t = tensor(args[i]);
      if (t == nullptr || p.scales == 0 || t->dim() != 2 || t->scalar_type() != at::kFloat) Py_RETURN_NONE;
      (i == 3 ? out_scale : x_scale) = t;
    }
    int quantize = 0;
    if (x->scalar_type() != p.in_type) {
      // fused quantisation: bf16 in, e4m3 + 1x128 fp32 scales on the wire
      if (x->scalar_type() != at::kBFloat16 || p.in_type != at::kFloat8_e4m3fn || x_scale != nullptr ||
          p.scales != p.hidden / 128 || out_scale == nullptr) {
        Py_RETURN_NONE;
      }
      quantize = p.quantize_mode;
    } else if (x_scale != nullptr ? out_scale == nullptr : p.scales != 0) {
      Py_RETURN_NONE;
    }
    if (!routing_ok(p, indices, weights, tokens)) Py_RETURN_NONE;
    const int32_t* bound;
    if (!bound_ok(args[8], &bound)) Py_RETURN_NONE;

    pplx::DispatchSendArgs s{};
    s.num_tokens = static_cast<int32_t>(tokens);
    s.x = ptr<const uint8_t>(*x);
    s.x_stride = static_cast<uint64_t>(x->stride(0)) * x->element_size();
    if (x_scale != nullptr) {
      s.x_scale = ptr<const uint8_t>(*x_scale);
      s.x_scale_stride_elem = x_scale->stride(1);
      s.x_scale_stride_token = x_scale->stride(0);
    }
    s.indices = ptr<const uint32_t>(*indices);
    s.indices_stride = static_cast<uint64_t>(indices->stride(0));
    s.weights = ptr<const float>(*weights);
    s.weights_stride = static_cast<uint64_t>(weights->stride(0));
    s.bound_m = bound;
    s.quantize = quantize;
    if (args[11] != Py_None) {
      const at::Tensor* logits = tensor(args[11]);
      if (logits == nullptr || logits->dim() != 2 || logits->size(0) != tokens || logits->size(1) < p.num_experts ||
          p.num_experts > p.local_experts * p.world || logits->stride(1) != 1 ||
          (logits->scalar_type() != at::kFloat && logits->scalar_type() != at::kBFloat16)) {
        Py_RETURN_NONE;
      }
      s.logits = logits->const_data_ptr();
      s.logits_stride = logits->stride(0);
      s.logits_bf16 = logits->scalar_type() == at::kBFloat16;
      if (args[12] != Py_None) {
        const at::Tensor* bias = tensor(args[12]);
        if (bias == nullptr || bias->scalar_type() != at::kFloat || !bias->is_contiguous() || bias->numel() < p.num_experts) {
          Py_RETURN_NONE;
        }
        s.logits_bias = ptr<const float>(*bias);
      }
    }
    pplx::DispatchRecvArgs r{};
    r.out_num_tokens = ptr<int32_t>(*num);
    r.out_x = ptr<uint8_t>(*out_x);
    r.out_x_stride = static_cast<uint64_t>(out_x->stride(0)) * out_x->element_size();
    if (out_scale != nullptr) {
      r.out_x_scale = ptr<uint8_t>(*out_scale);
      r.out_x_scale_stride_elem = out_scale->stride(1);
      r.out_x_scale_stride_token = out_scale->stride(0);
    }
    r.out_rows = static_cast<uint32_t>(out_x->size(0));
    if (!g_api->a2a_dispatch(p.context, send ? &s : nullptr, recv ? &r : nullptr, c10::cuda::getCurrentCUDAStream().stream())) {
      return nullptr;
    }
    Py_RETURN_TRUE;
  });
}

// a2a_combine(plan, out_tokens, indices, weights, expert_y | None, bound_m | None, do_send, do_recv, accumulate)
PyObject* a2a_combine(PyObject*, PyObject* const* args, Py_ssize_t nargs) {
  return guarded([&]() -> PyObject* {
    if (nargs != 9) Py_RETURN_NONE;
    const A2APlan* plan = plan_of(args[0]);
    if (plan == nullptr) return nullptr;
    const A2APlan& p = *plan;
    const at::Tensor *out = tensor(args[1]), *indices = tensor(args[2]), *weights = tensor(args[3]);
    const bool send = PyObject_IsTrue(args[6]) == 1, recv = PyObject_IsTrue(args[7]) == 1;
    if (out == nullptr || indices == nullptr || indices->dim() != 2 || (!send && !recv)) Py_RETURN_NONE;
    const int64_t tokens = indices->size(0);
    if (!routing_ok(p, indices, weights, tokens) || !is_matrix(*out, tokens, p.hidden, p.out_type)) Py_RETURN_NONE;
    at::ScalarType y_type = p.out_type;
    pplx::CombineSendArgs s{};
    if (args[4] == Py_None) {
      if (send) Py_RETURN_NONE;
    } else {
      const at::Tensor* y = tensor(args[4]);
      if (y == nullptr || y->dim() != 2 || y->size(1) != p.hidden || y->stride(1) != 1) Py_RETURN_NONE;
      y_type = y->scalar_type();
      if (y_type != at::kHalf && y_type != at::kBFloat16 && y_type != at::kFloat) Py_RETURN_NONE;
      if (y->element_size() != static_cast<int64_t>(c10::elementSize(p.out_type))) Py_RETURN_NONE;
      s.expert_y = ptr<const uint8_t>(*y);
      s.expert_y_stride = static_cast<uint64_t>(y->stride(0)) * y->element_size();
    }
    pplx::CombineRecvArgs r{};
    if (!bound_ok(args[5], &r.bound_m)) Py_RETURN_NONE;
    r.num_tokens = static_cast<int32_t>(tokens);
    r.out_tokens = ptr<uint8_t>(*out);
    r.out_tokens_stride = static_cast<uint64_t>(out->stride(0));
    r.indices = ptr<const uint32_t>(*indices);
    r.indices_stride = static_cast<uint64_t>(indices->stride(0));
    r.weights = ptr<const float>(*weights);
    r.weights_stride = static_cast<uint64_t>(weights->stride(0));
    r.accumulate = PyObject_IsTrue(args[8]) == 1;
    // torch's scalar type codes are the kernels' (A2ADtype)
    if (!g_api->a2a_combine(p.context, send ? &s : nullptr, recv ? &r : nullptr, static_cast<int>(y_type),
                            c10::cuda::getCurrentCUDAStream().stream())) {
      return nullptr;
    }
    Py_RETURN_TRUE;
  });
}

// ---------------------------------------------------------------------------
// grouped GEMM
// ---------------------------------------------------------------------------

// The tuple AllToAllContext.combine_send_external() returns for a rank, with the optional bulk flag.
bool scatter_of(PyObject* t, pplx::ops::CombineScatter* sc) {
  if (!PyTuple_Check(t) || (PyTuple_GET_SIZE(t) != 9 && PyTuple_GET_SIZE(t) != 10)) return false;
  auto num = [&](Py_ssize_t i) { return PyLong_AsUnsignedLongLong(PyTuple_GET_ITEM(t, i)); };
  PyObject *recv = PyTuple_GET_ITEM(t, 2), *flags = PyTuple_GET_ITEM(t, 4);
  sc->row_src = reinterpret_cast<const uint32_t*>(num(0));
  sc->row_tk = reinterpret_cast<const uint32_t*>(num(1));
  sc->slot_stride = num(3);
  sc->world = static_cast<int>(num(5));
  sc->signal_value = static_cast<uint32_t>(num(6));
  sc->done_counter = reinterpret_cast<uint32_t*>(num(7));
  sc->status = reinterpret_cast<const uint32_t*>(num(8));
  if (PyTuple_GET_SIZE(t) == 10) sc->bulk = static_cast<int>(num(9));
  if (sc->world < 1 || sc->world > pplx::ops::CombineScatter::kMaxPeers || !PyList_Check(recv) || !PyList_Check(flags) ||
      PyList_GET_SIZE(recv) != sc->world || PyList_GET_SIZE(flags) != sc->world) {
    return false;
  }
  for (int i = 0; i < sc->world; ++i) {
    sc->peer_recv[i] = reinterpret_cast<uint8_t*>(PyLong_AsUnsignedLongLong(PyList_GET_ITEM(recv, i)));
    sc->peer_flag[i] = reinterpret_cast<uint32_t*>(PyLong_AsUnsignedLongLong(PyList_GET_ITEM(flags, i)));
  }
  return !PyErr_Occurred();
}

// grouped_fp8_gemm(a, a_scale, b, b_scale, expert_num_tokens, out | None, out_scale | None, mode, expert_padding,
//                  error_flag | None, num_ctas, wait_cycles | None, debug_skip, trace | None, scatter | None,
//                  tile_rows, scale_format) -> True | None
PyObject* grouped_fp8_gemm(PyObject*, PyObject* const* args, Py_ssize_t nargs) {
  return guarded([&]() -> PyObject* {
    if (nargs != 17) Py_RETURN_NONE;
    const at::Tensor *a = tensor(args[0]), *a_scale = tensor(args[1]), *b = tensor(args[2]), *b_scale = tensor(args[3]);
    const at::Tensor* counts = tensor(args[4]);
    if (a == nullptr || a_scale == nullptr || b == nullptr || b_scale == nullptr || counts == nullptr) Py_RETURN_NONE;
    int v[17] = {};
    for (int i : {7, 8, 10, 12, 15, 16}) v[i] = static_cast<int>(PyLong_AsLong(args[i]));
    if (PyErr_Occurred()) return nullptr;
    constexpr at::ScalarType kFp8 = at::kFloat8_e4m3fn;
    if (a->dim() != 2 || b->dim() != 3 || a->scalar_type() != kFp8 || b->scalar_type() != kFp8 || a->stride(1) != 1 ||
        !b->is_contiguous() || !b_scale->is_contiguous()) {
      Py_RETURN_NONE;
    }
    const int64_t rows = a->size(0), k = a->size(1), e = b->size(0), n = b->size(1);
    if (b->size(2) != k || a_scale->dim() != 2 || a_scale->size(0) != rows || a_scale->size(1) != k / 128 ||
        a_scale->scalar_type() != at::kFloat || b_scale->dim() != 3 || b_scale->size(0) != e || b_scale->size(1) != n / 128 ||
        b_scale->size(2) != k / 128 || b_scale->scalar_type() != at::kFloat || counts->scalar_type() != at::kInt ||
        counts->dim() != 1 || counts->size(0) != e) {
      Py_RETURN_NONE;
    }
    pplx::ops::GroupedGemmParams p;
    const int mode = v[7];
    const at::Tensor* out = args[5] == Py_None ? nullptr : tensor(args[5]);
    if (mode == pplx::ops::kBf16Scatter) {
      if (args[5] != Py_None || args[14] == Py_None) Py_RETURN_NONE;
    } else if (mode == pplx::ops::kSwiGLUQuant) {
      const at::Tensor* out_scale = args[6] == Py_None ? nullptr : tensor(args[6]);
      if (out == nullptr || !is_matrix(*out, rows, n / 2, kFp8) || out_scale == nullptr ||
          !is_matrix(*out_scale, rows, n / 256, at::kFloat)) {
        Py_RETURN_NONE;
      }
      p.out_scale = ptr<float>(*out_scale);
      p.out_scale_stride_row = out_scale->stride(0);
    } else if (out == nullptr || !is_matrix(*out, rows, n, at::kBFloat16)) {
      Py_RETURN_NONE;
    }
    if (args[14] != Py_None && !scatter_of(args[14], &p.scatter)) {
      if (!PyErr_Occurred()) PyErr_SetString(PyExc_ValueError, "not a scatter descriptor of combine_send_external()");
      return nullptr;
    }
    at::Tensor own_flag;
    const at::Tensor* flag = args[9] == Py_None ? nullptr : tensor(args[9]);
    if (flag == nullptr) {
      if (args[9] != Py_None) Py_RETURN_NONE;
      own_flag = at::zeros({1}, a->options().dtype(at::kInt));
      flag = &own_flag;
    }
    const at::Tensor* wait_cycles = args[11] == Py_None ? nullptr : tensor(args[11]);
    const at::Tensor* trace = args[13] == Py_None ? nullptr : tensor(args[13]);
    p.a = a->const_data_ptr();
    p.a_stride = a->stride(0);
    p.a_scale = ptr<const float>(*a_scale);
    p.a_scale_stride_row = a_scale->stride(0);
    p.a_scale_stride_k = a_scale->stride(1);
    p.b = b->const_data_ptr();
    p.b_scale = ptr<const float>(*b_scale);
    p.expert_num_tokens = ptr<const int32_t>(*counts);
    p.out = out == nullptr ? ptr<void>(*a) : ptr<void>(*out);
    p.out_stride = out == nullptr ? 16 : out->stride(0) * out->element_size();
    p.error_flag = ptr<uint32_t>(*flag);
    p.num_experts = static_cast<int>(e);
    p.N = static_cast<int>(n);
    p.K = static_cast<int>(k);
    p.expert_padding = v[8];
    p.max_rows = static_cast<int>(rows);
    p.mode = mode;
    p.num_ctas = v[10];
    p.wait_cycles = wait_cycles == nullptr ? nullptr : ptr<unsigned long long>(*wait_cycles);
    p.debug_skip = v[12];
    p.trace = trace == nullptr ? nullptr : ptr<long long>(*trace);
    p.tile_rows = v[15];
    p.scale_format = v[16];
    if (!g_api->grouped_fp8_gemm(p, c10::cuda::getCurrentCUDAStream().stream())) return nullptr;
    Py_RETURN_TRUE;
  });
}

#define FAST(name) {#name, reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(name)), METH_FASTCALL, nullptr}
PyMethodDef kMethods[] = {
    FAST(topk_route), FAST(a2a_plan), FAST(a2a_dispatch), FAST(a2a_combine), FAST(grouped_fp8_gemm),
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
