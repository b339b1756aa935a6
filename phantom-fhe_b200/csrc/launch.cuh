// launch.cuh - how every kernel of the library is launched.
#pragma once
#include <cuda_runtime.h>

#include <utility>

// Every kernel of the library is launched with the programmatic-serialisation attribute and begins with pdl_enter()
// (modarith.cuh): the next kernel's launch and block scheduling overlap the end of the previous one, and its CTAs wait until
// that kernel has completed and its writes are visible. At small sizes a key switch is a chain of kernels of 2 to 5 us, where
// launch latency is a third of the time (one transform pair of 8 limbs at N = 2^14: 30.7 -> 22.1 us; a rotation at
// N = 2^13: 74 -> 54). No kernel signals before it ends (griddepcontrol.launch_dependents): CTAs that are scheduled early
// take SM slots from the running grid and bunch up on the SMs that empty first (signalled on entry, eight hoisted rotations
// at N = 2^15 take 708 us; before the exchange of the transforms 597; never 599; without the attribute 670).
// `cluster`: CTAs per thread-block cluster along x.
template <class... P, class... A>
static void launch_cl(unsigned cluster, void (*kernel)(P...), dim3 grid, dim3 block, size_t smem, cudaStream_t s, A &&...args) {
    cudaLaunchAttribute at[2] = {};
    at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[0].val.programmaticStreamSerializationAllowed = 1;
    at[1].id = cudaLaunchAttributeClusterDimension;
    at[1].val.clusterDim.x = cluster, at[1].val.clusterDim.y = 1, at[1].val.clusterDim.z = 1;
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = grid, cfg.blockDim = block, cfg.dynamicSmemBytes = smem, cfg.stream = s, cfg.attrs = at, cfg.numAttrs = cluster > 1 ? 2 : 1;
    (void)cudaLaunchKernelEx(&cfg, kernel, P(std::forward<A>(args))...);  // the caller reads the error
}
template <class... P, class... A>
static void launch_k(void (*kernel)(P...), dim3 grid, dim3 block, size_t smem, cudaStream_t s, A &&...args) {
    launch_cl(1, kernel, grid, block, smem, s, std::forward<A>(args)...);
}
