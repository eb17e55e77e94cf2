// chain.cuh -- kernels of one stream whose launches overlap (programmatic dependent launch).
// This part has no counterpart in the reference.
//
// A kernel launched with launchChained may start while the kernel before it in the stream
// still runs, once every CTA of that one has called letNextStart.  It sets up what needs no
// memory (barriers, tensor memory, indices) and calls afterPrevious before it reads or writes
// any; that returns when the kernel before it has completed, which for its part completed only
// after the one before.  Every thread calls afterPrevious; a kernel that is launched this way
// never leaves it out.
// The kernels of one network pass are chained this way: their launch and set-up, 1 to 2 us
// each, lie behind the tail of the one before.  One patch of 64^3 (14 kernels) 187 -> 169 us,
// a training step of 8 (52 kernels) 2091 -> 2058 us, 200 x 264 x 232 voxels 2010 -> 1983 us.
#pragma once

#include <utility>

#include <cuda_runtime.h>

namespace dxmcg {
namespace chain {
    __device__ __forceinline__ void afterPrevious() { asm volatile("griddepcontrol.wait;\n" ::: "memory"); }
    __device__ __forceinline__ void letNextStart() { asm volatile("griddepcontrol.launch_dependents;\n" ::: "memory"); }

    template <class... P, class... A>
    cudaError_t launchChained(void (*kernel)(P...), dim3 grid, dim3 block, size_t smem, cudaStream_t s, A&&... args)
    {
        cudaLaunchAttribute attr {};
        attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
        attr.val.programmaticStreamSerializationAllowed = 1;
        cudaLaunchConfig_t cfg {};
        cfg.gridDim = grid;
        cfg.blockDim = block;
        cfg.dynamicSmemBytes = smem;
        cfg.stream = s;
        cfg.attrs = &attr;
        cfg.numAttrs = 1;
        return cudaLaunchKernelEx(&cfg, kernel, static_cast<P>(std::forward<A>(args))...);
    }
} // namespace chain
} // namespace dxmcg
