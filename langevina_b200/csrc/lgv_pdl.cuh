// lgv_pdl.cuh -- programmatic dependent launch of the sub-step kernels.
//
// The sub-steps of a step are short kernels that each depend on the one
// before.  Launched with programmatic stream serialization, a kernel's blocks
// are placed as soon as every block of the previous kernel has started
// (pdl_launch) and there is room, and do what needs no field -- coordinates,
// noise -- before pdl_wait, which returns when the previous kernel is complete
// and its writes are visible.
//
// Rules the kernels keep: every thread that touches device memory calls
// pdl_wait first, and no kernel of a chain ends without a block having waited,
// so that completion of a kernel implies completion of all before it.  What an
// earlier kernel writes is never read through a const __restrict__ pointer: the
// compiler may move such a load above the wait.
// Anything else on the stream (copies, events, kernels launched plainly) is
// ordered as usual.
#pragma once

#include <cuda_runtime.h>

#include <utility>

namespace lgv {

__device__ __forceinline__ void pdl_launch() { asm volatile("griddepcontrol.launch_dependents;\n" ::: "memory"); }
__device__ __forceinline__ void pdl_wait() { asm volatile("griddepcontrol.wait;\n" ::: "memory"); }

template <typename... P, typename... A>
inline cudaError_t launch_pdl(void (*kern)(P...), dim3 grid, dim3 block, size_t smem, cudaStream_t st, A &&...args) {
  cudaLaunchConfig_t c{};
  c.gridDim = grid;
  c.blockDim = block;
  c.dynamicSmemBytes = smem;
  c.stream = st;
  cudaLaunchAttribute at{};
  at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at.val.programmaticStreamSerializationAllowed = 1;
  c.attrs = &at;
  c.numAttrs = 1;
  return cudaLaunchKernelEx(&c, kern, P(std::forward<A>(args))...);
}

}  // namespace lgv
