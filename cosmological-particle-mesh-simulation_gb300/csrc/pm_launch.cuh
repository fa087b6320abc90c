// Programmatic launches.  A kernel launched with launch_chained may be set up -- and its blocks
// started on SMs that the kernel before it in the stream has already left -- before that kernel
// has finished.  Every such kernel calls chain_begin() before it touches global memory: it waits
// until the kernel before it is complete and its writes are visible, then lets the kernel
// after it be set up in turn.  Since each kernel waits for the one before, a complete kernel
// means that all before it are complete, as in plain stream order.
#pragma once
#include <cuda_runtime.h>

namespace pm {

__device__ __forceinline__ void chain_begin() {
  asm volatile("griddepcontrol.wait;" ::: "memory");
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
}

// A stream, and whether the launches on it are programmatic.  What a chain saves are the launch
// gaps and the ramp of each kernel (a 192^3 Poisson solve 104 -> 90 us, a 32^3 / 64^3 step 75 -> 60);
// what it can cost is occupancy: a block that starts early takes the SM as the kernel before left
// it, with that kernel's split between L1 and shared memory.  So callers chain grids of up to
// 256 cells a side (on 512 the step went from 2168 to 2205 us), and never a kernel that lives on L1
// behind one with large shared memory (the kick behind the transforms: 67 -> 107 us on 256).
struct Launch {
  cudaStream_t st;
  bool chain;
  Launch(cudaStream_t s, bool c = false) : st(s), chain(c) {}
  operator cudaStream_t() const { return st; }
};

template <class... P, class... A>
cudaError_t launch_chained(void (*kernel)(P...), int grid, int block, size_t smem, Launch l, A&&... args) {
  cudaLaunchConfig_t c = {};
  c.gridDim = dim3((unsigned)grid);
  c.blockDim = dim3((unsigned)block);
  c.dynamicSmemBytes = smem;
  c.stream = l.st;
  cudaLaunchAttribute a = {};
  a.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  a.val.programmaticStreamSerializationAllowed = 1;
  c.attrs = &a;
  c.numAttrs = l.chain ? 1 : 0;
  return cudaLaunchKernelEx(&c, kernel, static_cast<P>(args)...);
}

}  // namespace pm
