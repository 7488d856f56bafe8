// Launches that may start while the kernel before them on the stream still runs (programmatic
// dependent launch). Such a kernel waits for its predecessor where it first needs that one's work; what
// a kernel lets its successor read before then must be complete when it lets it start. Without the
// launch attribute the device calls are nothing.
#pragma once
#include <cuda_runtime.h>

// The successor's blocks may be scheduled from now on (once every block of this kernel got here).
__device__ __forceinline__ void letNextStart() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
// The predecessor has ended and its writes are visible. Every thread that may be a block's last calls
// it before the block ends, so that a kernel's end is its predecessors' end too.
__device__ __forceinline__ void waitForPrevious() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
// A kernel that needs its predecessor from the start: only its launch overlaps. The successor starts
// when everything before this kernel is complete.
__device__ __forceinline__ void enterChain() {
  waitForPrevious();
  letNextStart();
}

template <class Kernel, class... Args>
static void launchChained(bool overlap, Kernel kernel, int grid, int threads, size_t smem, cudaStream_t st, Args... args) {
  cudaLaunchConfig_t c = {};
  c.gridDim = dim3((unsigned)grid);
  c.blockDim = dim3((unsigned)threads);
  c.dynamicSmemBytes = smem;
  c.stream = st;
  cudaLaunchAttribute a = {};
  a.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  a.val.programmaticStreamSerializationAllowed = 1;
  c.attrs = &a;
  c.numAttrs = overlap ? 1 : 0;
  cudaLaunchKernelEx(&c, kernel, args...);
}
