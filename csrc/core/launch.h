// Launch of a kernel that begins with ptx.cuh's grid_wait().
#pragma once

#include <cuda_runtime.h>

namespace pplx {

// The kernel may be brought onto the SMs while its predecessor on the stream is still running (once that
// has called grid_allow_next() in every block, or block by block as it ends), so that its launch and
// whatever it does before grid_wait() overlap the predecessor's end. It must read and write global
// memory only after grid_wait(), in every block: the wait is what orders it after the predecessor, and
// a kernel that ended without it would let the one after it start before the one before it had ended.
// And it must read by ordinary loads: what the predecessor writes changes while this kernel is already
// resident, so it is not the read-only memory that __ldg, ld.global.nc and ptx.cuh's ld_input_v4 ask
// for (nor does the wait hold an __ldg back: the compiler may move it up).
// It pays where a step is a chain of short kernels: dispatch + combine of 128 tokens x 7168 bf16 16.4 ->
// 13.5 us a pass, routing of 128 tokens 5.6 -> 4.6 us, a Qwen3-like layer of 2048 tokens (five kernels)
// 135 -> 130 us.
inline cudaError_t launch_overlapped(const void* kernel, dim3 grid, dim3 block, void** args, size_t smem, cudaStream_t stream) {
  cudaLaunchAttribute attr{};
  attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr.val.programmaticStreamSerializationAllowed = 1;
  cudaLaunchConfig_t config{};
  config.gridDim = grid;
  config.blockDim = block;
  config.dynamicSmemBytes = smem;
  config.stream = stream;
  config.attrs = &attr;
  config.numAttrs = 1;
  return cudaLaunchKernelExC(&config, kernel, args);
}

}  // namespace pplx
