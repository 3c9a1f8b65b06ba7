// launch.cuh -- launches that follow one another in a stream.
//
// A step is one to six kernels of a few microseconds to a few hundred, each on the
// results of the one before.  launch_next lets the device set a grid up while the
// kernel before it drains (programmatic stream serialization); the kernel calls
// after_previous first, which returns once that one has completed and its writes are
// visible, so nothing is read or written early.  The kernels give no early signal:
// no block of the next grid takes room from them.  About 2 us a launch: FP64 lid 32^3
// 7.2 -> 5.7 us a step, FP32 lid 97^3 26.9 -> 24.6, heated 81^3 21.7 -> 19.0.
// Such a kernel does not read through __ldg or const __restrict__: read-only loads are
// for memory that nothing writes during the kernel's lifetime, and that begins before
// the wait.
#pragma once
#include <cuda_runtime.h>

namespace mglc {

// first statement of every kernel launched so
__device__ __forceinline__ void after_previous() { cudaGridDependencySynchronize(); }

template <typename... P, typename... A>
inline cudaError_t launch_next(void (*kernel)(P...), dim3 grid, dim3 block, size_t smem,
                               cudaStream_t s, A... args) {
    cudaLaunchAttribute a[1];
    a[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    a[0].val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t c{};
    c.gridDim = grid;
    c.blockDim = block;
    c.dynamicSmemBytes = smem;
    c.stream = s;
    c.attrs = a;
    c.numAttrs = 1;
    return cudaLaunchKernelEx(&c, kernel, static_cast<P>(args)...);
}

}  // namespace mglc
