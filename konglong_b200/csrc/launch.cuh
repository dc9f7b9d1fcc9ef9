// launch.cuh - dependent kernel launches.  The kernels of a time step follow
// each other on one stream, each reading what the one before wrote.  Launched
// with the programmatic-serialisation attribute, a kernel is set up and its CTAs
// take their places as soon as every CTA of the one before has started and
// called dep_launch(); it calls dep_wait() before it first touches anything a
// kernel of the step writes, which returns when the kernel before has finished
// and its writes are visible.  What stands before dep_wait() (barriers, tables,
// trace taps, model constants) runs while the kernel before drains; on a 601 x
// 300 line shot, whose kernels take 3-8 us, set-up and drain were a third of the
// step.
//
// Such a kernel is resident while the one before still writes, so what a step
// writes (wavefields, gradient parts, slab scales, receiver planes, PML and Q
// memory) is read behind dep_wait() by ordinary loads, ld_l2() or asynchronous
// copies.  The read-only path (__ldg) asks for data that nobody writes during the
// kernel's lifetime; a load through a __restrict__ pointer may become one or move
// above the wait, which such a pointer does not alias; and an intrinsic like
// __ldcg may move.  __ldg and __restrict__ stay with model volumes and tables.
//
// Every thread of every such kernel calls dep_wait(), so that one
// kernel's end implies the end of all before it; a launch without the attribute
// waits for the whole stream as usual.
#pragma once
#include <cuda_runtime.h>

namespace rtm {

__device__ __forceinline__ void dep_launch() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
__device__ __forceinline__ void dep_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
// a coherent load through L2 that stays where it stands, behind the wait
__device__ __forceinline__ float4 ld_l2(const float4 *p) {
  float4 v;
  asm volatile("ld.global.cg.v4.f32 {%0, %1, %2, %3}, [%4];"
               : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w)
               : "l"(__cvta_generic_to_global(p))
               : "memory");
  return v;
}

// Two launches of one pass over disjoint tiles (PML tiles, then interior tiles),
// the second free to run beside the first: the PML tiles come in one or two
// uneven waves (813 tiles on 592 places: the SMs stood idle for a quarter of the
// launch), and the interior tiles fill what they leave.  The first launch lets
// the second in only after its own dep_wait(), so whatever both read is written
// by then; block 0 says so in `flag` (release / acquire, a number of its own for
// each pair), and a second launch that does not find its number waits as usual.  The
// second launch calls dep_wait() as its last act instead of its first: its end
// then implies the end of the first, and the kernel after it need wait for
// nothing more.  For its loads the acquire stands in for dep_wait().  No launch waits for one behind it: the second is let in when
// every CTA of the first has its place.
enum { PAIR_NONE = 0, PAIR_FIRST = 1, PAIR_SECOND = 2 };
struct LaunchPair {
  int role;
  unsigned *flag;
  unsigned number;
};
// in place of dep_launch(); __syncthreads(); dep_wait(): called by every thread,
// after what the CTA prepares; `lead` is one thread, the one that issues copies
__device__ __forceinline__ void pair_begin(const LaunchPair &p, bool lead) {
  if (p.role == PAIR_FIRST) {
    __syncthreads();
    dep_wait();
    if (lead) {
      if (blockIdx.x == 0) asm volatile("st.release.gpu.global.u32 [%0], %1;" ::"l"(p.flag), "r"(p.number) : "memory");
      dep_launch();
    }
    return;
  }
  dep_launch();
  int seen = 1;
  if (p.role == PAIR_SECOND && lead) {
    unsigned v;
    asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p.flag) : "memory");
    asm volatile("fence.proxy.async.global;" ::: "memory");
    seen = v == p.number;
  }
  seen = __syncthreads_and(seen);
  if (p.role == PAIR_NONE || !seen) dep_wait();
}
__device__ __forceinline__ void pair_end(const LaunchPair &p) {
  if (p.role == PAIR_SECOND) dep_wait();
}

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
