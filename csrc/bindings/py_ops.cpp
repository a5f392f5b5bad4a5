// Bindings of the expert-side compute ops (no counterpart in the reference, which ships no
// expert computation at all).
#include <pybind11/pybind11.h>
#include <pybind11/stl.h>

#include "../core/error.h"
#include "../ops/grouped_gemm.h"
#include "../ops/multimem.h"
#include "../ops/router.h"
#include "native_api.h"
#include "py_util.h"

namespace py = pybind11;
using namespace pplx;
using namespace pplx::ops;

pplx_py::NativeApi* pplx_py::native_api() {
  static NativeApi api = [] {
    NativeApi a{};
    a.topk_route = [](const TopkRouteParams& p, cudaStream_t stream) {
      return call_guarded([&] { topk_route(p, stream); });
    };
    a.grouped_fp8_gemm = [](const GroupedGemmParams& p, cudaStream_t stream) {
      return call_guarded([&] {
        if (p.scale_format == kScalesFp32 && (p.wait_cycles != nullptr || p.trace != nullptr || p.debug_skip != 0)) {
          grouped_fp8_gemm_profiled(p, stream);
        } else {
          grouped_fp8_gemm(p, stream);
        }
      });
    };
    a.a2a_dispatch = api_a2a_dispatch;
    a.a2a_combine = api_a2a_combine;
    return a;
  }();
  return &api;
}

void bind_ops(py::module_& m) {
  m.def(
      "multimem_red_add_u32",
      [](uint64_t mc_ptr, uint32_t value, uint64_t stream) {
        multimem_red_add_u32(reinterpret_cast<uint32_t*>(mc_ptr), value, reinterpret_cast<cudaStream_t>(stream));
      },
      py::arg("mc_ptr"), py::arg("value"), py::arg("stream"),
      "Adds value to the 32-bit word at a multicast-mapped address on every bound GPU (one multimem.red).");
}
