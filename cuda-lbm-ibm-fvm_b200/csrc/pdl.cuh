// pdl.cuh -- programmatic dependent launch, for chains of short kernels.
#pragma once
#include <cuda_runtime.h>

#include <utility>

namespace vof {

// Programmatic dependent launch.  Every kernel of the convergent solve is launched with
// cudaLaunchAttributeProgrammaticStreamSerialization (pdl_launch) and begins
// with pdl_enter(): it waits for the grid before it to complete (and its
// writes to be visible) before its first global memory access, then lets the
// next grid launch.  The launch and prologue of a kernel so overlap the end of
// the one before, which removes most of the gap between the short kernels of
// the coarse levels.  Launched without the attribute, the wait returns at once.
__device__ __forceinline__ void pdl_enter() {
    asm volatile("griddepcontrol.wait;" ::: "memory");
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
}

// The same for kernels that read through __restrict__ pointers or __ldg: such a
// load may be moved before the wait, whose memory clobber does not bind it.
// The pointers are opaque after the wait, and known to be global (as opaque
// generic ones they cost the V-cycle 2 to 3 %: 16^3 MIXED 663 -> 683 us a step;
// so 668, and the reverse pass of 64^3 x 40 steps takes 6.84 ms for 7.04).
// The solve's kernels, the step's small-grid ones, the layout copies and the
// adjoint's short kernels begin so (24 x 20 x 16, one step a call: 640 -> 485
// us for six); the large grids' kernels do not: registers for the opaque
// pointers cost them 1 %.
template <typename... P>
__device__ __forceinline__ void pdl_enter(P&... p) {
    asm volatile("griddepcontrol.wait;" ::: "memory");
    (([&] {
         size_t a = __cvta_generic_to_global(p);
         asm volatile("" : "+l"(a));
         p = static_cast<P>(__cvta_global_to_generic(a));
     }()),
     ...);
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
}

template <typename... KArgs, typename... Args>
static cudaError_t pdl_launch(void (*kernel)(KArgs...), dim3 grid, dim3 block, size_t smem, cudaStream_t s,
                              Args&&... args) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = grid;
    cfg.blockDim = block;
    cfg.dynamicSmemBytes = smem;
    cfg.stream = s;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, kernel, std::forward<Args>(args)...);
}

}  // namespace vof
