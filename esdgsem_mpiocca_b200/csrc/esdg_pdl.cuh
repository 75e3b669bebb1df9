// Programmatic dependent launch of the step's kernels.
#pragma once

namespace esdg {

// The step's kernels are launched while the kernel before them still runs
// (Engine::launch).  Every one of them waits here, before its first access to
// anything a step writes, until that kernel has completed and its writes are
// visible; what it reads before is constant during a step (connectivity,
// geometry, operators).  The release lets the next kernel's blocks take their
// places; the persistent kernels give it with their last tile, the one-shot
// ones at once (it takes effect when their last block has started).
__device__ __forceinline__ void pdl_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void pdl_release() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }

}  // namespace esdg
