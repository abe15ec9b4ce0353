// Dependent launches: a kernel launched with launch_after may start while the
// kernel before it on the stream is still finishing (programmatic stream
// serialization); it must call wait_before before it touches anything that
// the earlier kernel wrote, and may read constant data (link lists, weights)
// before that. A time step of a small domain is a chain of kernels of a few
// microseconds, and the launch of each next one is then hidden behind its
// predecessor. The wait returns once every earlier kernel of the stream has
// finished and its writes are visible, so every block calls it before any
// early return: a grid none of whose blocks waited could itself finish before
// its predecessor.
#pragma once
#include <utility>
#include <cuda_runtime.h>

namespace aslb {

// wait_before, then let_next: the next kernel may launch once this one's blocks
// have all waited. In this order what a kernel reads before its own wait was
// written before its predecessor began (a list built just before a time loop
// is visible to the loop's first condition launch, too).
__device__ __forceinline__ void let_next() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
__device__ __forceinline__ void wait_before() { asm volatile("griddepcontrol.wait;" ::: "memory"); }

template <class... P, class... A>
inline cudaError_t launch_after(void (*kern)(P...), dim3 grid, dim3 block, size_t smem, cudaStream_t st, A&&... args) {
  cudaLaunchAttribute at{};
  at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at.val.programmaticStreamSerializationAllowed = 1;
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = grid;
  cfg.blockDim = block;
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cfg.attrs = &at;
  cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg, kern, P(std::forward<A>(args))...);
}

}  // namespace aslb
