// Programmatic dependent launch for the kernels of a training step.
//
// A kernel whose first instruction is `pdl_prolog()` may be launched with programmatic stream serialization: its
// blocks become resident as soon as every block of the kernel before it on the stream has started (that kernel's own
// prolog releases them), and they wait inside `griddepcontrol.wait` until that kernel has completed and its writes
// are visible. What is saved is the launch latency and ramp-up between dependent kernels, ~1-3 us per boundary inside
// a captured graph; nothing changes in what a kernel may read or write. Launched without the attribute the two
// instructions do nothing.
#pragma once
#include <cuda_runtime.h>
#include <utility>

namespace rb {

// 1 when the kernels of a step (not only the tensor-core kernel) are to be launched with the attribute: planner
// option `pdl` = 2 (RB_GEMM_PDL); defined in gemm_tc.cu.
int pdl_enabled();

__device__ __forceinline__ void pdl_prolog() {
  asm volatile("griddepcontrol.wait;" ::: "memory");
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
}

// `l1_first`: a kernel started early otherwise inherits the split of on-chip memory that the tensor-core kernel before it
// asked for, 28 KB of L1 an SM, which holds too few of a long stream's loads at once. Asking for the L1 side first has the
// split changed, and costs the early start on an SM where the other kernel is still resident. So it is for kernels that run
// long out of HBM; the short kernels of the normalisations, beside weight-gradients, lose by it (figures below).
template <class... KArgs, class... Args>
inline cudaError_t launch_step(bool l1_first, void (*kernel)(KArgs...), dim3 grid, dim3 block, size_t smem,
                               cudaStream_t stream, Args&&... args) {
  cudaLaunchConfig_t cfg;
  cfg.gridDim = grid;
  cfg.blockDim = block;
  cfg.dynamicSmemBytes = smem;
  cfg.stream = stream;
  cudaLaunchAttribute at[2];
  unsigned n = 0;
  if (pdl_enabled() != 0) {
    at[n].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[n++].val.programmaticStreamSerializationAllowed = 1;
  }
  if (l1_first) {
    at[n].id = cudaLaunchAttributePreferredSharedMemoryCarveout;
    at[n++].val.sharedMemCarveout = cudaSharedmemCarveoutMaxL1;
  }
  cfg.attrs = at;
  cfg.numAttrs = n;
  return cudaLaunchKernelEx(&cfg, kernel, std::forward<Args>(args)...);
}

template <class... KArgs, class... Args>
inline cudaError_t launch_pdl(void (*kernel)(KArgs...), dim3 grid, dim3 block, size_t smem, cudaStream_t stream,
                              Args&&... args) {
  return launch_step(false, kernel, grid, block, smem, stream, std::forward<Args>(args)...);
}

// Measured (us): the parameter sweep of AlexNet 284 -> 238, its step 1475 -> 1435. Asked for by every kernel without dynamic
// shared memory, the step of the 20-layer CIFAR network grows from 970 to 1030 and that of the Go network from 1420 to 1535:
// their normalisations wait for SMs to be empty. The poolings and the LRN gain 8 of AlexNet's 1435 and lose 5 of NIN's 720 at
// inference: not for them.
template <class... KArgs, class... Args>
inline cudaError_t launch_streaming(void (*kernel)(KArgs...), dim3 grid, dim3 block, size_t smem, cudaStream_t stream,
                                    Args&&... args) {
  return launch_step(true, kernel, grid, block, smem, stream, std::forward<Args>(args)...);
}

}  // namespace rb
