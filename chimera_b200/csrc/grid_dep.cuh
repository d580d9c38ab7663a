// grid_dep.cuh -- waiting for, and making way for, the neighbouring kernels of a
// stream.
#pragma once
#include <cuda_runtime.h>

namespace chimera {

// Programmatic dependent launch: the host lets a kernel start while the one
// before it in the stream still runs.  grid_wait() holds until that one has
// completed, its writes visible; everything a kernel reads comes after it.
// grid_release(), once every CTA of a grid has called it or ended, lets the next
// kernel's CTAs take up free places and wait there.  Both do nothing in an
// ordinary launch.
__device__ __forceinline__ void grid_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void grid_release() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }

}  // namespace chimera
