// launch.cuh -- programmatic dependent launches: a kernel launched with launch_pdl may be
// scheduled while the kernel before it on the stream still runs, and waits in pdl_wait()
// until that one has completed and its writes are visible.  What is saved is the launch
// latency between two short kernels.
#pragma once

#include <cstdint>
#include <cuda_runtime.h>

namespace sloth {

// Waits for the kernels this one depends on (returns at once after an ordinary launch).
// Every kernel launched with launch_pdl calls it before its first access to global memory,
// so that "the kernel before" always covers everything before that one too.
//
// Read-only loads (__ldg, const __restrict__) are for what nobody writes while the kernel
// lives, and it lives from before the wait: a mesh, and what kernels before the one just
// before it wrote (that one waited for them before it let this one start).  What the kernel
// just before writes -- keys and tile generations for the resolve, transformed vertices for
// setup, sample ranges for the large counts, entries for the raster -- is read by plain loads.
// The zero it returns is added to the indices of the loads that follow: read-only loads are
// not ordered by the memory clobber, and this makes their addresses depend on the wait.
__device__ __forceinline__ uint32_t pdl_wait()
{
    uint32_t zero;
    asm volatile("griddepcontrol.wait;\nmov.u32 %0, 0;" : "=r"(zero)::"memory");
    return zero;
}

// pdl_wait, and then lets this kernel's dependents be scheduled (once every block has come
// here or left).  Not before the wait: a chain of kernels would all become resident behind
// the first, and take the SMs from work on other streams (the newline fold of the uneven
// batch, launched so, ran after the fill instead of beside the scan: 1612 us a pass became 1716).
__device__ __forceinline__ uint32_t pdl_begin()
{
    const uint32_t zero = pdl_wait();
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    return zero;
}

// Lets this kernel's dependents be scheduled before it has waited itself: what they may not
// overtake, it waits for before it ends (pdl_wait).
__device__ __forceinline__ void pdl_trigger() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }

// An ordinary launch with the same arguments: what the kernels of a captured graph use, where
// the edges between dependents cost what they save (uneven batch 1583 us a pass with them,
// 1561 without; 24 views of 160x48 38.4 and 36.0).  Two are dependent there all the same: the
// setup of 32 triangles a block, behind the reset (24 views 29.3 us, plain 29.5), and the scan,
// whose launcher contexts share (1557 us either way).
template <class... K, class... A>
cudaError_t launch(void (*kernel)(K...), dim3 grid, dim3 block, size_t smem, cudaStream_t s, A... args)
{
    kernel<<<grid, block, smem, s>>>(static_cast<K>(args)...);
    return cudaGetLastError();
}

template <class... K, class... A>
cudaError_t launch_pdl(void (*kernel)(K...), dim3 grid, dim3 block, size_t smem, cudaStream_t s, A... args)
{
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = grid;
    cfg.blockDim = block;
    cfg.dynamicSmemBytes = smem;
    cfg.stream = s;
    cudaLaunchAttribute at{};
    at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at.val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = &at;
    cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, kernel, static_cast<K>(args)...);
}

}  // namespace sloth
