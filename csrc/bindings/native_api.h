// The calls that csrc/torch_ops makes into this extension. That module links libtorch, so that it can
// read tensors and allocate results without going through Python; this one does not, so that the
// tokenizer, the transfer engine and their tests run where torch is not installed. The table travels
// as a capsule (`pplx_garden._native._api`). Every entry needs the GIL, sets a Python exception and
// returns false when the call throws.
#pragma once

#include <cuda_runtime.h>

#include "../a2a/a2a_types.h"
#include "../ops/grouped_gemm.h"
#include "../ops/router.h"

namespace pplx_py {

struct NativeApi {
  bool (*topk_route)(const pplx::ops::TopkRouteParams& params, cudaStream_t stream);
  bool (*grouped_fp8_gemm)(const pplx::ops::GroupedGemmParams& params, cudaStream_t stream);
  // `context`: AllToAllContext._handle(), alive as long as that object. A null phase is not run.
  bool (*a2a_dispatch)(void* context, const pplx::DispatchSendArgs* send, const pplx::DispatchRecvArgs* recv,
                       cudaStream_t stream);
  bool (*a2a_combine)(void* context, const pplx::CombineSendArgs* send, const pplx::CombineRecvArgs* recv, int y_dtype,
                      cudaStream_t stream);
};

// py_a2a.cpp
bool api_a2a_dispatch(void* context, const pplx::DispatchSendArgs* send, const pplx::DispatchRecvArgs* recv,
                      cudaStream_t stream);
bool api_a2a_combine(void* context, const pplx::CombineSendArgs* send, const pplx::CombineRecvArgs* recv, int y_dtype,
                     cudaStream_t stream);

NativeApi* native_api();   // py_ops.cpp

constexpr const char* kNativeApiName = "pplx_garden._native._api";

}  // namespace pplx_py
