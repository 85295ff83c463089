// pdl.cuh -- programmatic dependent launch: a kernel of a chain starts while the
// one before it ends, makes its set-up (barriers, TMEM, indexes of the plan)
// and waits for that kernel's results before it reads them.
//
// Used where the kernel before has few CTAs left when it triggers and the
// waiting CTAs keep no SM from other work: the two GEMMs of the mixed product
// behind the table and operator kernels (FT N = 1000 57.4 -> 55.6 us, F N = 200
// 44.3 -> 39.5).  Chaining the operator kernel as well cost up to 7% (FTS N =
// 4096 236 -> 253: the second GEMM then holds its SMs from the first on), and so
// did the FP64 product's kernels (FTS N = 120 86 -> 98-108).
//
// Every kernel of a chain calls chain_wait in at least one CTA, so that its end
// implies the end of all kernels before it; a kernel launched without the
// attribute does not wait.  What a kernel of the chain wrote is read with plain
// loads: read-only ones (__ldg) may be moved ahead of the wait.
#pragma once

#include <cuda_runtime.h>

namespace lsg {

// the kernels before this one are complete and their writes visible
__device__ __forceinline__ void
chain_wait ()
{
  asm volatile ("griddepcontrol.wait;" ::: "memory");
}

// the next kernel of the chain may start once every CTA is here
__device__ __forceinline__ void
chain_next ()
{
  asm volatile ("griddepcontrol.launch_dependents;" ::: "memory");
}

template <class... P, class... A>
inline cudaError_t
launch_chained (void (*kernel) (P...), dim3 grid, dim3 block, size_t smem, cudaStream_t st,
                const A &...args)
{
  cudaLaunchAttribute at {};
  at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at.val.programmaticStreamSerializationAllowed = 1;
  cudaLaunchConfig_t c {};
  c.gridDim = grid;
  c.blockDim = block;
  c.dynamicSmemBytes = smem;
  c.stream = st;
  c.attrs = &at;
  c.numAttrs = 1;
  return cudaLaunchKernelEx (&c, kernel, P (args)...);
}

}  // namespace lsg
