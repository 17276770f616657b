// Launches of kernels that follow one another on a stream as programmatic
// dependents: such a kernel begins with grid_wait, which returns when the whole
// grid before it has finished and its writes are visible.  The order is the
// stream's; what overlaps is the launch (and whatever the kernel does before
// the wait, on data that no earlier kernel of the stream writes) with the
// previous kernel's end.  After the wait, data of earlier kernels is read
// through pointers without __restrict__: a load from a const __restrict__
// pointer may be hoisted above the wait or take the read-only path.
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

namespace mgcfd {

__device__ __forceinline__ void grid_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }

// Lets the next kernel start its blocks before this one's exit.
__device__ __forceinline__ void grid_trigger() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }

// Launches a kernel that begins with grid_wait as the programmatic dependent
// of the kernel before it in the stream (`chained`), else in plain stream order.
template <class... P, class... A>
void launch_shared(size_t shared_bytes, void (*kernel)(P...), int64_t blocks, int threads, cudaStream_t stream,
                   bool chained, A... args) {
  cudaLaunchConfig_t c = {};
  c.dynamicSmemBytes = shared_bytes;
  cudaLaunchAttribute at;
  c.gridDim = dim3((unsigned)blocks);
  c.blockDim = dim3((unsigned)threads);
  c.stream = stream;
  at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at.val.programmaticStreamSerializationAllowed = 1;
  c.attrs = &at;
  c.numAttrs = chained ? 1 : 0;
  cudaLaunchKernelEx(&c, kernel, P(args)...);  // errors: the callers' cudaGetLastError
}

template <class... P, class... A>
void launch(void (*kernel)(P...), int64_t blocks, int threads, cudaStream_t stream, bool chained, A... args) {
  launch_shared(0, kernel, blocks, threads, stream, chained, args...);
}

static __global__ void k_nothing() {}

// To be called once memory has been given back on a stream that lives on
// (cudaFreeAsync): an empty launch in plain order.  Until the stream has had a
// launch in plain order, that memory costs every later cudaMallocAsync of the
// process about 1 us for each such stream (measured: 20 us a call with 16
// streams, 4 with this launch; the set-up of a 17^3 mesh 6.1 ms with 32 streams,
// 0.9 with it).  Programmatic dependents do not count.
inline void after_free(cudaStream_t stream) { k_nothing<<<1, 1, 0, stream>>>(); }

}  // namespace mgcfd
