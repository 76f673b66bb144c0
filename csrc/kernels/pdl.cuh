// Programmatic dependent launch: a kernel may be placed on the SMs while its predecessor in the stream still runs, and waits
// there for the predecessor's results. What it hides is the launch latency and the set-up of the next kernel (about 1.5 us
// per launch in a captured chain of small kernels).
//
// Only kernels that read their inputs through TMA and ordinary loads are launched this way (`launch`: GEMM, attention);
// kernels with `const __restrict__` inputs may be given non-coherent loads, which must not run beside the writer. Those are
// launched normally and only trigger their successor early. All threads of a kernel launched through `launch` execute
// pdl_wait() before they touch global memory, so a kernel that has completed has also seen its own predecessor complete:
// the chain orders everything as a plain stream does. Without pdl_trigger() the next kernel starts when this one ends.
#pragma once
#include <cuda_runtime.h>

namespace opk {

__device__ __forceinline__ void pdl_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void pdl_trigger() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }

template <class... P, class... A>
cudaError_t launch(void (*kernel)(P...), dim3 grid, dim3 block, size_t smem, cudaStream_t stream, A&&... args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = block;
  cfg.dynamicSmemBytes = smem;
  cfg.stream = stream;
  cudaLaunchAttribute at;
  at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at.val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = &at;
  cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg, kernel, static_cast<A&&>(args)...);
}

}  // namespace opk
