// Launches of the kernels of a step one behind the other in a stream with
// programmatic dependent launch: a kernel's CTAs are placed as soon as the one
// before it has started its last, and wait there (chained) until it has
// finished and its writes are visible. Without it each of a step's two to eight
// kernel boundaries costs the launch latency and an idle GPU: @@CHAIN@@
#pragma once

#include <cuda_runtime.h>

#include <utility>

namespace dgpu {

// First statement of every thread of a kernel that chain() launches. No thread
// may leave before it: the kernel after this one takes this one's end for the
// end of all before it.
__device__ __forceinline__ void chained() {
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    asm volatile("griddepcontrol.wait;" ::: "memory");
}

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
