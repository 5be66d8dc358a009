/*
 * Launches that overlap the end of the kernel before them (programmatic
 * dependent launch).
 */
#ifndef SMATRAN_LAUNCH_AFTER_CUH
#define SMATRAN_LAUNCH_AFTER_CUH

#include <cuda_runtime.h>

namespace smat {

/* Kernels of a step (of the FDTD loop, or of a sweep of the layer transfer)
 * follow one another as programmatic dependents (launch_after): one is set up
 * while the one before ends and waits for its results in prior_done, which every
 * thread that touches fields, the ring or the step counter calls first (most of
 * a microsecond a launch: 14.1 -> 12.8 us for a step of two FP32 sweeps at 48^3
 * cells, 21.0 -> 20.0 at 100^3, 71.9 -> 71.4 at 160 x 160 x 120).  What the kernel
 * before writes is read through coherent loads (no const __restrict__: such loads
 * may count on data that stands still for the whole kernel).  After
 * next_may_start in every block the next kernel may run up to its own prior_done
 * beside this one: index arithmetic and loads of what no launch of a run changes
 * (coefficients, addresses, orders, records). */
__device__ __forceinline__ void prior_done() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void next_may_start() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
template <class... P, class... A>
inline cudaError_t launch_after_in(unsigned cluster, void (*fn)(P...), dim3 grid, dim3 block, size_t smem, cudaStream_t st, A... args)
{
    cudaLaunchAttribute at[2];
    at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[0].val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = grid;
    cfg.blockDim = block;
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    if (cluster) { /* CTAs of a cluster */
        at[1].id = cudaLaunchAttributeClusterDimension;
        at[1].val.clusterDim.x = cluster;
        at[1].val.clusterDim.y = at[1].val.clusterDim.z = 1;
        cfg.numAttrs = 2;
    }
    return cudaLaunchKernelEx(&cfg, fn, static_cast<P>(args)...);
}

template <class... P, class... A>
inline cudaError_t launch_after(void (*fn)(P...), dim3 grid, dim3 block, size_t smem, cudaStream_t st, A... args)
{
    return launch_after_in(0, fn, grid, block, smem, st, args...);
}

} // namespace smat

#endif
