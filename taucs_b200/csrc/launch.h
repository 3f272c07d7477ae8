// Kernel launches whose start overlaps the end of the kernel before
// (programmatic dependent launch).  Most launches of a factorization or solve
// are a level of a tree: short, and dependent on the one before.  With a plain
// launch the next kernel's CTAs are set up and read their descriptors only after
// the last CTA of the one before has left; here they are resident by then and
// wait on the SM (griddepcontrol.wait, which also makes every write of the
// kernels before visible).
//
// What every kernel launched this way keeps to:
// * grid_wait() before it reads or writes anything that another kernel of the
//   stream writes or reads, in every CTA that has work (a grid none of whose
//   CTAs waited could finish before its predecessors);
// * grid_trigger(), which lets the next kernel's CTAs start, only after its own
//   grid_wait(): so whatever the kernel before the previous one wrote may be read
//   ahead of the wait (A's values, the plan, in a solve L and the inverses);
// * what the kernel before may still be writing when this one starts (update
//   matrices and panels, work vectors, iterates, residuals) is read by plain or
//   L2 loads (__ldcg) only: not by __ldg, and not through a const __restrict__
//   pointer, which the compiler turns into the same read-only loads.  Those are
//   for data that nobody writes while the kernel lives, and may be moved;
// * the trigger late, when its CTAs are about to write their results: CTAs that
//   arrive while the grid still works are stacked on the SMs that happen to have
//   room, and stay there.  With triggers at the start a factorization of a
//   40x41x39 grid went from 6.56 to 7.00 ms and a solve with 64^3's factor from
//   2.07 to 2.41.
// CTAs that leave count as triggered.
// Whole steps without and with it: 139x142 mixed 1.75 and 1.65 ms, 29x24x26 mixed
// 2.22 and 2.13, 100x100 FP64 1.15 and 1.11; solves with 64^3's factor the same.
#pragma once

#include <cuda_runtime.h>

namespace tb {

#ifdef __CUDACC__
__device__ __forceinline__ void grid_trigger() { asm volatile("griddepcontrol.launch_dependents;"); }
__device__ __forceinline__ void grid_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void grid_wait_then_trigger() {
  grid_wait();
  grid_trigger();
}
#endif

// (a parameter's own type, so that arguments convert to it)
template <typename P>
struct AsParam { using type = P; };

template <typename... P>
inline cudaError_t launch(void (*k)(P...), dim3 grid, dim3 block, size_t smem, cudaStream_t st,
                          typename AsParam<P>::type... a) {
  cudaLaunchAttribute at = {};
  at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at.val.programmaticStreamSerializationAllowed = 1;
  cudaLaunchConfig_t c = {};
  c.gridDim = grid;
  c.blockDim = block;
  c.dynamicSmemBytes = smem;
  c.stream = st;
  c.attrs = &at;
  c.numAttrs = 1;
  return cudaLaunchKernelEx(&c, k, a...);
}

}  // namespace tb
