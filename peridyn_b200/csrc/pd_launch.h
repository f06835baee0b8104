// pd_launch.h -- programmatic dependent launch of the stepping kernels.
#pragma once

#include <cuda_runtime.h>

#include <cstdlib>
#include <cstring>

namespace pd {

// Programmatic dependent launch.  The stepping kernels are launched with
// programmatic stream serialization (launch_dep): a kernel's blocks may be
// dispatched while the previous kernel on the stream finishes, and wait
// here, before they read anything a previous kernel writes, until it has
// completed and its writes are visible.  Having passed the wait, a block lets the next
// kernel be dispatched in turn, so at most two grids of the chain are in
// flight and the older one never waits.  Without the launch attribute
// both instructions return at once.
__device__ __forceinline__ void pdl_enter() {
    asm volatile("griddepcontrol.wait;" ::: "memory");
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
}

// Launch of a stepping kernel with programmatic stream serialization (the
// kernel enters through pdl_enter); PD_NO_PDL=1 gives ordinary launches.
template <class... P>
inline void launch_dep_smem(void (*kern)(P...), unsigned grid, unsigned block, size_t smem, cudaStream_t st,
                            P... args) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(grid);
    cfg.blockDim = dim3(block);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[0].val.programmaticStreamSerializationAllowed = 1;
    const char *off = std::getenv("PD_NO_PDL");
    cfg.attrs = at;
    cfg.numAttrs = (off && std::strcmp(off, "1") == 0) ? 0 : 1;
    cudaLaunchKernelEx(&cfg, kern, args...);
}

template <class... P>
inline void launch_dep(void (*kern)(P...), unsigned grid, unsigned block, cudaStream_t st, P... args) {
    launch_dep_smem(kern, grid, block, 0, st, args...);
}

}  // namespace pd
