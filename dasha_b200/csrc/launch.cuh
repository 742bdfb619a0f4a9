// Programmatic dependent launch: a kernel starts when the last CTA of the stream's kernel before has left, so that its
// launch, its index arithmetic and its mbarriers overlap that kernel's completion (the flush of its writes, the
// launch latency): some 2 us of every launch.
#pragma once

#include <cuda_runtime.h>

#include <utility>

namespace dasha {

// Holds a CTA until every kernel before in the stream has completed and its writes are visible.  Nothing that a
// kernel of the stream writes may be read, and nothing stored, before; every kernel started by launch_overlapped
// calls it, so it covers all kernels before.  In an ordinary launch it does nothing.
__device__ __forceinline__ void wait_for_stream() { asm volatile("griddepcontrol.wait;" ::: "memory"); }

// Starts a kernel that calls wait_for_stream.  Measured per step or call: 64x32x64 FP64 0.619 -> 0.461 ms, 100x44x77
// FP32 0.776 -> 0.602, 128x128x128 FP32 1.92 -> 1.75, 256x128x256 FP32 6.35 -> 6.18; a gradient on 44x24x50
// 12.1 -> 8.5 ms; a bounded 41x25x33 step 1.04 -> 0.89 ms; dasha_current_noalloc 82 -> 69 us.  Started earlier still
// (griddepcontrol.launch_dependents at the kernels' start) the waiting CTAs take room from the running
// ones: 0.556, 0.649, 1.86, 6.60 ms.
template <class... P, class... A>
inline void launch_overlapped(cudaStream_t st, bool overlap, void (*fn)(P...), dim3 grid, int threads, size_t smem, A&&... a) {
    cudaLaunchAttribute at{};
    at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at.val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t c{};
    c.gridDim = grid;
    c.blockDim = dim3((unsigned)threads);
    c.dynamicSmemBytes = smem;
    c.stream = st;
    c.attrs = &at;
    c.numAttrs = overlap ? 1 : 0;
    cudaLaunchKernelEx(&c, fn, std::forward<A>(a)...);
}

}  // namespace dasha
