// Shared host-side plumbing lives with the public headers: include/cuvs/core/b200_common.hpp.
#pragma once
#include <cuvs/core/b200_common.hpp>

#include <utility>

namespace cuvs_b200 {

// Launch of a kernel that begins with chain_begin(): its blocks may be placed while the last blocks of the kernel before
// it on the stream still run (programmatic dependent launch), so that the launch itself costs little between two
// dependent kernels: one query of 32 probes (six kernels) 65.9 -> 55.5 us, 100 queries (nine) 123 -> 116 us.
template <typename... Params, typename... Args>
void launch_chained(void (*kernel)(Params...), dim3 grid, dim3 block, size_t smem, cudaStream_t stream, Args&&... args)
{
  cudaLaunchAttribute attr{};
  attr.id                                         = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr.val.programmaticStreamSerializationAllowed = 1;
  cudaLaunchConfig_t config{};
  config.gridDim          = grid;
  config.blockDim         = block;
  config.dynamicSmemBytes = smem;
  config.stream           = stream;
  config.attrs            = &attr;
  config.numAttrs         = 1;
  CUDA_TRY(cudaLaunchKernelEx(&config, kernel, std::forward<Args>(args)...));
}

#ifdef __CUDACC__
// First statement of such a kernel, in every thread: waits until the kernels before this one have completed and their
// writes are visible, and only then lets the next one's blocks in -- so whatever was launched two kernels earlier is
// complete when a block starts.
__device__ __forceinline__ void chain_begin()
{
  asm volatile("griddepcontrol.wait;" ::: "memory");
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
}
#endif

}  // namespace cuvs_b200
