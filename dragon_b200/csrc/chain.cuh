// Launches of the kernels of a step one behind the other in a stream with
// programmatic dependent launch: a kernel's CTAs are placed as soon as the one
// before it has started its last, and wait there (chained) until it has
// finished and its writes are visible. Without it each of a step's two to eight
// kernel boundaries costs the launch latency and an idle GPU: a 1D step of
// 512 cells 13.7 -> 9.7 us, Orszag-Tang 384^2 (eight kernels) 0.150 -> 0.138 ms.
#pragma once

#include <cuda_runtime.h>

#include <utility>

namespace dgpu {

// First statement of every thread of a kernel that chain() launches. No thread
// may leave before it: the kernel after this one takes this one's end for the
// end of all before it.
//
// What the kernel before it may write is read with plain loads, after this
// statement, which no load is moved above. The read-only path (ld.global.nc:
// __ldg, or a kernel parameter that is const and __restrict__) is for memory
// that nobody writes from the reading kernel's launch on, and such a load may
// be moved up. tests/test_chained_loads.py looks for both.
__device__ __forceinline__ void chained() {
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    asm volatile("griddepcontrol.wait;" ::: "memory");
}
// The same for a kernel whose follower is better placed at its end: the fused
// mixed MHD step holds one CTA pair per SM for its whole run, and placed around
// a running ghost fill it took 1.2 % longer (Orszag-Tang 1024^2).
__device__ __forceinline__ void chained_last() { asm volatile("griddepcontrol.wait;" ::: "memory"); }

// kernel<<<grid, block, smem, st>>>(args...) with the chaining attribute; the
// caller reads the outcome from cudaGetLastError().
template <class... P, class... A>
inline void chain(void (*kernel)(P...), dim3 grid, dim3 block, size_t smem, cudaStream_t st, A&&... args) {
    cudaLaunchConfig_t c{};
    c.gridDim = grid;
    c.blockDim = block;
    c.dynamicSmemBytes = smem;
    c.stream = st;
    cudaLaunchAttribute a{};
    a.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    a.val.programmaticStreamSerializationAllowed = 1;
    c.attrs = &a;
    c.numAttrs = 1;
    cudaLaunchKernelEx(&c, kernel, static_cast<P>(std::forward<A>(args))...);
}

}  // namespace dgpu
