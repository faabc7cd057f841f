// Programmatic dependent launch of the step's kernels. A kernel launched this
// way is set up while its predecessor in the stream still runs, and its
// blocks wait in pdl_wait() until that one has completed and its writes are
// visible; every kernel so launched calls pdl_wait() before it touches memory
// that an earlier launch writes, and the order of the stream's work is kept
// (after a copy, a memset or an event the launch is an ordinary one).
//
// Back-to-back ordinary launches on a GB300 complete on a grid of about
// 2.06 us: a step of a 16^3 lattice took 4.16 us (two of them), of a 64^3
// lattice 10.34 us (five). Without the grid they take 2.43 and 8.66 us.
// Releasing the next kernel early (griddepcontrol.launch_dependents at the
// start) measured slower, 2.7-3.0 and 8.8-9.3 us: its waiting blocks take
// slots from the running ones.
#pragma once

#include <cuda_runtime.h>

namespace fcfd {

template <class V>
__device__ __forceinline__ void after_wait(V& v) {
    if constexpr (sizeof(V) == 8) asm volatile("" : "+l"(v)::"memory");
    else asm volatile("" : "+r"(v)::"memory");
}

/// The wait. Volatile loads and those through pointers that may alias stay
/// behind it by its memory clobber. A load that is to the compiler a function
/// of its address alone does not: through a const restrict pointer, __ldg, or
/// an assembler statement that is not volatile. A kernel that reads what
/// earlier launches wrote in such a way hands the indices or pointers over from
/// which the addresses are formed; they come back as values that the compiler
/// cannot have had before.
template <class... V>
__device__ __forceinline__ void pdl_wait(V&... v) {
    asm volatile("griddepcontrol.wait;" ::: "memory");
    (after_wait(v), ...);
}

template <class... P, class... A>
cudaError_t launch_pdl(void (*kernel)(P...), dim3 grid, dim3 block, cudaStream_t st, A... args) {
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = grid;
    cfg.blockDim = block;
    cfg.stream = st;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, kernel, static_cast<P>(args)...);
}

} // namespace fcfd
