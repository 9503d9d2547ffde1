// pdl.cuh -- device side of programmatic dependent launches.
//
// A kernel launched with cudaLaunchAttributeProgrammaticStreamSerialization may
// start while the launch before it still runs, from the moment all of that
// one's blocks have called pdl_release() or ended; pdl_wait() returns when it
// has completed and its writes are visible. A kernel that waits before it
// touches memory, and itself completes only after that, keeps the order of the
// whole chain.
#pragma once

#include <stdint.h>

namespace tpt {

__device__ __forceinline__ void pdl_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void pdl_release() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }

// A load of memory that the launch before may have written. The read-only
// path (__ldg) is not for it: that is defined for data which nobody writes
// while the kernel runs, and the compiler may move such a load ahead of
// pdl_wait(). An ordinary load stays behind the wait's memory clobber; the
// assumption keeps it a load from global memory where the pointer itself comes
// from a structure in memory. Measured on B200 against __ldg: equal within the
// runs' spread everywhere but for 2048x2048 air, 240.7 and 244.7 us per tick
// (in calls back to back; the kernels alone take the same).
template <typename T> __device__ __forceinline__ T load_after_wait(const T *p) {
    __builtin_assume(__isGlobal(p));
    return *p;
}

}  // namespace tpt
