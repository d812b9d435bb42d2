// Programmatic dependent launch, used by the codec kernels.
//
// A kernel launched the ordinary way behind another on this device starts on
// the next tick of a 2.05 us clock: chains of a kernel that spins for 3, 4, 5,
// 6 us run at 6.2, 6.2, 8.2, 8.2 us per launch.  Launched with programmatic
// serialisation, and waiting in the kernel for what the stream holds before it,
// the same chains run at 3.7, 4.7, 5.7, 6.7 us, and the launch call itself is
// 0.5 us cheaper on the host.  Calls on tensors up to some MiB last 3 ... 20 us,
// so this is worth a tenth to a third of them.
//
// The contract: a kernel calls pdl_wait() before it touches global memory that
// is not a constant of the library, and every CTA calls it.  What the stream
// held before is then finished and visible, whatever it was.
//
// The exception: sparse_pack_kernel, sparse_pack_sum_kernel and sparse_onepass_kernel read
// the call's input before they wait.  That is sound because a kernel of the same call in front of them
// (the counting one; the one that clears the cursor) triggers only behind its own wait,
// so that whatever produced the input has finished before either can start, also where
// another kernel stands in between that triggers early (the scan).  A launch of one of
// them without such a kernel in front would race with the producer.
//
// pdl_trigger() lets the next kernel of the stream be brought in once all CTAs of
// this one have started, for chains inside one call whose next kernel has
// something to do meanwhile.  Kernels that fill the device do not trigger: the
// next grid's CTAs would be packed onto the SMs that happen to be free (a 128-CTA
// codec kernel behind another took 10.0 us a launch that way and 7 without).
#pragma once
#include <cuda_runtime.h>

#include <cstddef>
#include <utility>

namespace csw {

__device__ __forceinline__ void pdl_trigger() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
__device__ __forceinline__ void pdl_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
// the same, for a pointer that is read through the read-only path: its loads depend on the
// wait and cannot be moved in front of it, which a memory clobber alone does not promise for them
template <class T>
__device__ __forceinline__ void pdl_wait(T* __restrict__& p) {
  asm volatile("griddepcontrol.wait;" : "+l"(p)::"memory");
}

// An error that a call returns is its caller's to report: left pending in the runtime as well,
// the next cudaGetLastError of the process (torch's after a launch of its own, say) would meet it.
inline cudaError_t taken(cudaError_t e) {
  if (e != cudaSuccess) cudaGetLastError();
  return e;
}

template <class... P, class... A>
inline cudaError_t pdl_launch(void (*kernel)(P...), unsigned grid, unsigned block, size_t smem, cudaStream_t stream,
                              A&&... args) {
  cudaLaunchAttribute attr{};
  attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr.val.programmaticStreamSerializationAllowed = 1;
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3(grid);
  cfg.blockDim = dim3(block);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = stream;
  cfg.attrs = &attr;
  cfg.numAttrs = 1;
  return taken(cudaLaunchKernelEx(&cfg, kernel, P(std::forward<A>(args))...));
}

}  // namespace csw
