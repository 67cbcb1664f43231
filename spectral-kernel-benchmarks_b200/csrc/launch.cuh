// Stream-ordered launches whose start overlaps the end of the kernel before.
//
// A plan's stages are short kernels in one stream (a 128^2 flux is five of 8 to
// 27 us).  Launched with programmatic stream serialization, a kernel's launch
// and its prologue run while its predecessor ends; grid_wait() returns once the
// predecessor has completed and its writes are visible.  Everything before
// grid_wait() touches only the plan's constant tables, shared memory and
// registers.  Every such kernel calls grid_wait() in all its threads, so
// completion is transitive along the stream.  Launched after any other work (a
// copy, another library's kernel) the order is the ordinary one.
//
// Measured: 128^2 flux 80.6 -> 68.4 us, FP32 spectral pipeline at 128^2 (seven
// kernels) 70.7 -> 55.7, pruned FP32 256^2 round trip 70.1 -> 60.3.  No kernel
// releases its successor early (griddepcontrol.launch_dependents): waiting CTAs
// take shared memory, and so L1, from the running ones; with early release a
// 256^2 flux of 4 members ran 2 to 8 % longer, and nothing gained over 1 %.

#pragma once

#include <cuda_runtime.h>

namespace skb {

__device__ __forceinline__ void grid_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }

template <typename... P, typename... A>
cudaError_t launch_chained(void (*kernel)(P...), dim3 grid, unsigned threads, size_t bytes, cudaStream_t stream,
                           A&&... args) {
    cudaLaunchAttribute attribute{};
    attribute.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attribute.val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t config{};
    config.gridDim = grid;
    config.blockDim = dim3(threads);
    config.dynamicSmemBytes = bytes;
    config.stream = stream;
    config.attrs = &attribute;
    config.numAttrs = 1;
    // A refused launch is reported here, once: the code left standing would be the
    // next cudaGetLastError()'s, in a later launch or in the caller's own code.
    const cudaError_t err = cudaLaunchKernelEx(&config, kernel, static_cast<P>(args)...);
    if (err != cudaSuccess) cudaGetLastError();
    return err;
}

}  // namespace skb
