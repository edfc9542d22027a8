// Kernels of one commit launched as a chain (programmatic dependent launch).
//
// A chained kernel's CTAs are placed as soon as its predecessor's have exited,
// without waiting for that grid to be retired, and chain_wait() returns once
// the predecessor has completed and its writes are visible.  Every kernel
// launched with launch_chained calls chain_wait() before it touches the
// message, the codeword or the tree, so a kernel completes after its
// predecessor and the order is that of plain launches.  In a kernel launched
// the plain way chain_wait() returns at once.
//
// A commit is 4 to 9 launches: 2^17 words of 32 lanes 97 -> 79 us, 2^20 of
// 1024 lanes 262 -> 249 us.  The predecessors do not trigger the launch early
// (griddepcontrol.launch_dependents): the waiting CTAs of a leaf kernel then
// crowd onto the SMs that free first, and the latter commit takes 309 us.
#pragma once
#include <cuda_runtime.h>

#include <utility>

namespace bz {

__device__ __forceinline__ void chain_wait() {
    asm volatile("griddepcontrol.wait;" ::: "memory");
}

template <typename... P, typename... A>
inline void launch_chained(void (*kernel)(P...), dim3 grid, unsigned threads, size_t smem,
                           cudaStream_t st, A &&...args) {
    cudaLaunchAttribute at{};
    at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at.val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = grid;
    cfg.blockDim = dim3(threads);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cfg.attrs = &at;
    cfg.numAttrs = 1;
    cudaLaunchKernelEx(&cfg, kernel, std::forward<A>(args)...);
}

}  // namespace bz
