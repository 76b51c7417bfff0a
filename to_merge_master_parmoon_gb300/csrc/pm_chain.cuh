// pm_chain.cuh — launches that overlap their predecessor (programmatic
// dependent launch): the kernel may start while the previous kernel of the
// stream still runs and waits for it on the device before it reads its
// results.
//
// A kernel launched this way may be resident while its predecessor writes the
// vectors that it reads after the wait.  Such vectors are no read-only data of
// the launch: they are read by ordinary loads (no __ldg, no const __restrict__
// pointer, which become non-coherent loads) or from L2 (__ldcg).
#ifndef PM_CHAIN_CUH
#define PM_CHAIN_CUH

#include <cuda_runtime.h>

namespace pm {

// the previous kernel of the stream has finished and its writes are visible
__device__ __forceinline__ void wait_previous() {
  asm volatile("griddepcontrol.wait;" ::: "memory");
}
// the next kernel of the stream may start (it waits before it reads results)
__device__ __forceinline__ void start_next() {
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
}

// every block of the kernel has to call wait_previous(); overlap = false: an
// ordinary launch of the same kernel, after its predecessor
template <typename... Args>
int launch_overlapped(bool overlap, void (*kernel)(Args...), dim3 grid, int block, size_t smem,
                      cudaStream_t s, const Args &...args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = dim3((unsigned)block);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = s;
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = at;
  cfg.numAttrs = overlap ? 1 : 0;
  return cudaLaunchKernelEx(&cfg, kernel, args...) == cudaSuccess ? 1 : -1;
}
template <typename... Args>
int launch_chained(void (*kernel)(Args...), dim3 grid, int block, size_t smem, cudaStream_t s,
                   const Args &...args) {
  return launch_overlapped(true, kernel, grid, block, smem, s, args...);
}

}  // namespace pm

#endif
