/*
 * cf_launch.cuh -- launches that overlap the end of the kernel before them (programmatic dependent
 * launch).
 *
 * A step is two to four kernels of 5 to 200 us, each waiting for the one before it.  Launched by
 * launch_pdl, a kernel's blocks are brought up as the last blocks of the kernel before it exit, and
 * wait in pdl_begin until that one has completed and its writes are visible.  (Allowing the successor
 * earlier, by griddepcontrol.launch_dependents at a kernel's start, makes waiting blocks resident beside
 * working ones and is slower: canal 1.4k triangles 21.7 us per step without overlap, 24.6 allowed at the
 * start, 21.5 at the exit; batched descent iteration 3.34, 3.11, 2.80 ms.)
 */
#ifndef CF_LAUNCH_CUH
#define CF_LAUNCH_CUH

#include <cuda_runtime.h>

namespace cf {
namespace {

/* A thread of a kernel launched by launch_pdl calls this before it touches memory that a kernel, or a copy
 * made by a call, may have written; what it may read earlier are the tables (member constants among them)
 * that the host copied when the context or the adjoint was made.  Some thread of such a kernel calls it in
 * any case, since its dependents take its end for the end of all kernels before it.  A kernel launched
 * plainly needs nothing, whichever way its neighbours are launched: it begins when all before it have
 * ended, and a dependent of it waits here for its end. */
__device__ __forceinline__ void pdl_begin() {
  asm volatile("griddepcontrol.wait;" ::: "memory");
}

template <class... P, class... A>
void launch_pdl(void (*kernel)(P...), int grid, int block, cudaStream_t st, const A&... args) {
  cudaLaunchAttribute at;
  at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at.val.programmaticStreamSerializationAllowed = 1;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)grid);
  cfg.blockDim = dim3((unsigned)block);
  cfg.stream = st;
  cfg.attrs = &at;
  cfg.numAttrs = 1;
  cudaLaunchKernelEx(&cfg, kernel, P(args)...);
}

}  // namespace
}  // namespace cf

#endif
