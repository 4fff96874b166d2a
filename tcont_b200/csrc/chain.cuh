// chain.cuh -- device side of launch_chained (kernels.hpp).
#pragma once

namespace tcontb {

// Every block calls both, once: chain_wait returns when all kernels in front of this one in the stream have finished and
// their writes are visible, chain_release lets the next kernel's blocks be scheduled as soon as an SM has room for them.
// (All blocks must wait: a kernel that ended without waiting would count as finished before the one in front of it.)
__device__ __forceinline__ void chain_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void chain_release() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }

}  // namespace tcontb
