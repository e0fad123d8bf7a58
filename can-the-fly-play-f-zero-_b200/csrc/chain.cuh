// Chains of short kernels, each the next one's only predecessor in a stream, as programmatic dependent launches.
#pragma once
#include <cuda_runtime.h>

namespace fb {

// A kernel lets its successor be set up while it runs (at its start) and itself waits, before it
// touches any global memory, until its predecessor has completed and its writes are visible. Every
// block executes both before its first return, so completion stays transitive along the stream,
// and a block waits only for blocks that are already resident (with their TMEM): a successor starts
// when all of its predecessor's blocks have come this far. Behind an ordinary launch or copy, and
// before one, the order is the stream's as ever.
//
// What any earlier work of the stream may have written is read with plain loads: a kernel of the chain is
// resident while its predecessors still write, so such data is not read-only for its lifetime, as __ldg
// demands (the compiler may move an __ldg above the wait, and the read-only path may hold old contents).
// __ldg is for what is written before the chain begins, as the connectome.
__device__ __forceinline__ void pdl_chain()
{
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    asm volatile("griddepcontrol.wait;" ::: "memory");
}

// The two halves apart, for a kernel whose successor is better set up late: a successor's blocks settle on the SMs
// that have room when they are let go, all of them on a few where this kernel fills the others.
__device__ __forceinline__ void pdl_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void pdl_launch() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }

// The same for a kernel whose successor reads, before its own wait, what was in memory before this kernel
// began: the successor starts when all that has completed.
__device__ __forceinline__ void pdl_chain_behind()
{
    asm volatile("griddepcontrol.wait;" ::: "memory");
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
}

// A launch of such a chain, as clusters of 1 x cy x cz blocks
template <typename... P, typename... A>
cudaError_t launch_chain(void (*kernel)(P...), dim3 grid, dim3 block, size_t smem, cudaStream_t st, unsigned cy, unsigned cz, A... args)
{
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = grid;
    cfg.blockDim = block;
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cudaLaunchAttribute at[2];
    at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[0].val.programmaticStreamSerializationAllowed = 1;
    at[1].id = cudaLaunchAttributeClusterDimension;
    at[1].val.clusterDim.x = 1;
    at[1].val.clusterDim.y = cy;
    at[1].val.clusterDim.z = cz;
    cfg.attrs = at;
    cfg.numAttrs = cy * cz > 1 ? 2 : 1;
    return cudaLaunchKernelEx(&cfg, kernel, P(args)...);
}

}  // namespace fb
