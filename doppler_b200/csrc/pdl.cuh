// Programmatic dependent launch (griddepcontrol) helpers.
//
// pdl_launch(): lets the next kernel in the stream start being scheduled now.
// pdl_wait():   blocks until the previous kernel in the stream has completed and its
//               writes are visible.  Both are no-ops for a kernel launched without the
//               programmatic-serialization attribute.
// Rule used throughout: before pdl_wait() a kernel touches only data that no earlier kernel of the SAME STEP writes: the packed
// weights, and (decode attention) positions, lengths and cache rows, which earlier steps wrote.  After it, it reads
// activations and writes.  pdl_launch() comes first, or behind pdl_wait() where dependents that are resident early cost more
// than they save.
// The second half of that data needs the previous STEP to be complete when any kernel of this one starts.  Every step is a
// graph launch of its own, which sees to it; and the kernels that begin a step (gather_f16_kernel, stream_embed_kernel)
// launch their dependents behind their wait, so that it holds as well for steps that share a graph or run without one.
#pragma once
__device__ __forceinline__ void pdl_launch() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
__device__ __forceinline__ void pdl_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
