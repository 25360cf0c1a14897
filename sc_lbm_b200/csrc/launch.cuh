// launch.cuh -- kernels launched as programmatic dependents of the one before.
//
// A kernel launched this way may start while the kernel before it in the
// stream drains, which hides its launch latency.  Before dependent_wait it reads
// only what no kernel in the stream writes (a batch's tile list and argument
// blocks, which a copy waited for brought there), and writes nothing outside its
// CTA; dependent_launch follows the wait, so at most two kernels of a chain are
// under way and the one before them has ended: with two buffers in turn, nothing
// that a kernel writes is still being read.  Data of the kernel before is read
// with ordinary loads (the read-only path may hold lines from before the wait).
#pragma once
#include <cuda_runtime.h>

#include <utility>

namespace sclbm {

// everything the previous kernel of the stream wrote is visible after this
__device__ __forceinline__ void dependent_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
// the next kernel of the stream may take its places from here on
__device__ __forceinline__ void dependent_launch()
{
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
}

// launches kern as a programmatic dependent of the previous kernel in s
template <typename... P, typename... A>
inline cudaError_t launch_dependent(void (*kern)(P...), dim3 grid, dim3 block, size_t smem, cudaStream_t s,
                                    A &&...args)
{
    cudaLaunchAttribute at{};
    at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at.val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t c{};
    c.gridDim = grid;
    c.blockDim = block;
    c.dynamicSmemBytes = smem;
    c.stream = s;
    c.attrs = &at;
    c.numAttrs = 1;
    return cudaLaunchKernelEx(&c, kern, std::forward<A>(args)...);
}

} // namespace sclbm
