// Launches without a gap between dependent kernels. A step is a chain of short kernels (10 to 20 us
// each for a small system), and an ordinary launch starts about 2 us after the end of the one
// before it: the flush of its writes and the launch itself are in sequence. launch_pdl lets the
// blocks be scheduled once every block of the predecessor has exited, and pdl_enter, the first thing
// such a kernel does before global memory is touched, waits for the predecessor's writes. A
// kernel launched with launch_pdl calls pdl_enter in every thread; everything before its predecessor
// is then complete as well, since the predecessor waited in the same way or was launched
// without overlap.
//
// The predecessor gives no earlier signal (griddepcontrol.launch_dependents). With one at its start the
// blocks of the next kernel are placed while the SMs are partly taken, and a grid of one
// or two blocks per SM ends up with three on some: measured 8.95 ms for five FP64 steps of 256
// walkers in 120 orbitals, 7.71 with the signal left to the blocks' exits and 8.00 with ordinary
// launches; 2.44 / 2.24 / 2.48 ms for a pair of 512 walkers in 60 orbitals, mixed precision.
#pragma once
#include <cuda_runtime.h>

namespace afq {

__device__ __forceinline__ void pdl_enter() { asm volatile("griddepcontrol.wait;" ::: "memory"); }

template <class... P, class... A>
inline cudaError_t launch_pdl(void (*kernel)(P...), dim3 grid, dim3 block, size_t smem, cudaStream_t st, A&&... args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = block;
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg, kernel, static_cast<P>(args)...);
}

// A kernel's limit of dynamic shared memory, raised to smem where it is lower. The limit belongs to the function, for
// all threads of the process: one that set it to its own launch's need could lower it between another thread's
// setting and launch, which then fails. It is only ever raised.
cudaError_t raise_smem_limit(const void* kernel, size_t smem);

}  // namespace afq
