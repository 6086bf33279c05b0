#pragma once

namespace b2 {

// Programmatic dependent launch: a kernel launched with the attribute may start before the kernel ahead of it in
// the stream has finished; it must not touch anything that kernel writes until pdl_wait() returns. Both are
// no-ops in a kernel launched the ordinary way.
__device__ __forceinline__ void pdl_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void pdl_launch_dependents() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }

}  // namespace b2
