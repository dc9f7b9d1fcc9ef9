// launch.cuh - dependent kernel launches.  The kernels of a time step follow
// each other on one stream, each reading what the one before wrote.  Launched
// with the programmatic-serialisation attribute, a kernel is set up and its CTAs
// take their places as soon as every CTA of the one before has started and
// called dep_launch(); it calls dep_wait() before it first touches anything a
// kernel of the step writes, which returns when the kernel before has finished
// and its writes are visible.  What stands before dep_wait() (barriers, tables,
// trace taps, model constants) runs while the kernel before drains; on a 601 x
// 300 line shot, whose kernels take 3-8 us, set-up and drain were a third of the
// step.  Every thread of every such kernel calls dep_wait(), so that one
// kernel's end implies the end of all before it; a launch without the attribute
// waits for the whole stream as usual.
#pragma once
#include <cuda_runtime.h>

namespace rtm {

__device__ __forceinline__ void dep_launch() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
__device__ __forceinline__ void dep_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }

// k<<<grid, block, smem, st>>>(args...) with the attribute
template <typename... P, typename... A>
void launch_dep(void (*k)(P...), dim3 grid, dim3 block, size_t smem, cudaStream_t st, const A &...args) {
  cudaLaunchConfig_t c{};
  c.gridDim = grid, c.blockDim = block, c.dynamicSmemBytes = smem, c.stream = st;
  cudaLaunchAttribute at{};
  at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at.val.programmaticStreamSerializationAllowed = 1;
  c.attrs = &at, c.numAttrs = 1;
  cudaLaunchKernelEx(&c, k, static_cast<P>(args)...);  // an error stays for the caller's check
}

}  // namespace rtm
