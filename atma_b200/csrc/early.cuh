// Launches that may begin before the kernel in front of them has ended (programmatic dependent launch), for chains of kernels
// of a few microseconds: a CTA of the next kernel takes its place on an SM, and asks for the weights it is going to stream,
// while the one in front is still running.
//
// A kernel launched this way begins with early_start(): it lets its own successor take place and then waits until the kernel
// in front has ended and its writes are visible.  Every thread of every CTA calls it before it reads or writes anything of
// device memory, so that the end of a kernel still means the end of all kernels in front of it; the one thing allowed before
// it is a request to bring memory into L2, which is coherent and so may be early for whatever is written there later.
// Inputs are not declared __restrict__: read-only loads could be moved in front of the wait.
//
// Only steps of a few rows are launched so: their products are this library's too.  Between a library's kernels, which neither
// release early nor start early, it gives nothing (64 rows of Zemivik: 573 us a step without, 576 with).
#pragma once

#include <cuda_runtime.h>
#include <cstdint>

namespace atma {

__device__ __forceinline__ void early_start() {
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  asm volatile("griddepcontrol.wait;" ::: "memory");
}

__device__ __forceinline__ void prefetch_l2(const void* p) { asm volatile("prefetch.global.L2 [%0];" ::"l"(p)); }     // the line of p

constexpr int kEarlyRows = 16;              // rows of a step that decode_linear serves

template <typename... P, typename... A>
void launch_early(int64_t rows_of_step, void (*kernel)(P...), dim3 grid, dim3 block, size_t smem, cudaStream_t st, A... args) {
  cudaLaunchAttribute early;
  early.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  early.val.programmaticStreamSerializationAllowed = 1;
  cudaLaunchConfig_t c = {};
  c.gridDim = grid; c.blockDim = block; c.dynamicSmemBytes = smem; c.stream = st;
  c.attrs = &early; c.numAttrs = rows_of_step <= kEarlyRows ? 1 : 0;
  cudaLaunchKernelEx(&c, kernel, static_cast<P>(args)...);       // an error is the caller's to read (launch_status)
}

}  // namespace atma
